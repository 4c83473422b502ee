// particle3d.cuh -- particle stage of a 3-D single-layer cloud by groups of
// rows; included by step.cu inside its namespace.
//
// One block of kNT threads per group of up to four rows (interior rows and
// wall rows in separate groups), staged in shared memory by bulk copies;
// thread t holds the nodes t, t + kNT, ... of every row of the group.
//   1. FP64 sums over the rows, one reduction for the group;
//   2. the rows' scalars, one row per lane of warp 0, and the axis factors
//      spread over the block;
//   3. diffuse walls, or the collision, written straight to the
//      distribution, and the macros by linearity (k_particle_stream).
// The group shares the chain of barriers, divisions and exponentials that a
// row needs between its two passes, which is what a warp or a block per row
// waits for; the rest is about seven FP64-pipe operations a value, with their
// conversions and indices (issue slots 76 % busy, the FP64 pipe 28 %), beside
// the HBM traffic of the row in and out.
// All arithmetic is FP64, as in the general kernel.
// Measured, particle stage: cavity3d Nx 24 Nv 16 FP32 688 us by the general
// kernel (a warp per row, its copy read and written in every pass), 240 us
// here (HBM 68); FP64 Nx 40 Nv 10 470 us streamed, 425 here.
#pragma once

constexpr int kGroupRows = 4;

// Rows per block: four or two where four blocks an SM have room for them
// (or two blocks, for rows up to 50 KB), one up to the limit.
static int groupRows(const StepParams &p, size_t es)
{
    const size_t row = (size_t)p.ldf * es;
    if (4 * row <= 42u * 1024u) return 4;
    if (2 * row <= 100u * 1024u) return 2;
    return row <= 200u * 1024u ? 1 : 0;
}

template <typename T>
__global__ void __launch_bounds__(kNT, 4)
k_particle_group(ParticleArgs<T> a, StepParams p, int rows, int interior)
{
    constexpr int P = kGroupRows, kW = kNT / 32;
    __shared__ double velD[kMaxNv];
    __shared__ double tab[P][3][kMaxNv];
    __shared__ double red[kW][P * 8], tot[P][8];
    __shared__ double par[P][9];          // ux, uy, uz, 1/(2RT), lam A, scale, fix, M0, T
    __shared__ double wallS[P][7];
    __shared__ int part[P], mode[P];
    __shared__ T redMin[kW][P];
    __shared__ __align__(8) uint64_t bar;
    extern __shared__ __align__(128) unsigned char groupSmem[];
    T *buf = reinterpret_cast<T *>(groupSmem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int V = p.V, Nv = p.Nv, ldf = p.ldf;
    const double dvN = p.dvN;
    // groups of interior rows first, then groups of wall rows
    const int gi = (interior + rows - 1) / rows;
    const bool wallG = (int)blockIdx.x >= gi;
    const int t0 = wallG ? interior + ((int)blockIdx.x - gi) * rows : (int)blockIdx.x * rows;
    const int n = min(rows, (wallG ? p.N : interior) - t0);
    if (tid < n) part[tid] = a.rowOrder[t0 + tid];
    for (int q = tid; q < Nv; q += kNT) velD[q] = fma((double)q, p.dv, p.vmin);
    if (tid == 0)
    {
        mbarInit(&bar, 1);
        mbarInitFence();
    }
    __syncthreads();
    if (tid == 0)
    {
        const uint32_t bytes = (uint32_t)(ldf * sizeof(T));
        mbarExpectTx(&bar, bytes * n);
        for (int q = 0; q < n; ++q)
            bulkLoad(buf + (size_t)q * ldf, a.g + (size_t)part[q] * ldf, bytes, &bar);
    }
    const bool screenG = p.limiter == 2 && !wallG;
    double2 nad = make_double2(INFINITY, -INFINITY);
    if (tid < n && screenG) nad = reinterpret_cast<const double2 *>(a.nad)[part[tid]];
    if (wallG)
        for (int j = tid; j < 7 * n; j += kNT)
            wallS[j / 7][j % 7] = a.wall[7 * (size_t)part[j / 7] + j % 7];
    bool dead = false;
    mbarWait(&bar, 0, dead);
    if (__syncthreads_or(dead))
    {
        // The rows never arrived: report, give the copies a second bounded
        // wait, stop.
        if (tid == 0)
        {
            atomicOr(&a.sc->err, 4);
            bool d2 = false;
            mbarWait(&bar, 0, d2);
        }
        __syncthreads();
        return;
    }

    const int dI = kNT % Nv, dJ = (kNT / Nv) % Nv, dK = kNT / (Nv * Nv);
    const int iv0 = tid % Nv, jv0 = (tid / Nv) % Nv, kv0 = tid / (Nv * Nv);
    auto walk = [&](auto &&fn) {
        int iv = iv0, jv = jv0, kv = kv0;
        for (int k = tid; k < V; k += kNT)
        {
            fn(k, iv, jv, kv);
            iv += dI;
            jv += dJ;
            kv += dK;
            if (iv >= Nv) { iv -= Nv; ++jv; }
            if (jv >= Nv) { jv -= Nv; ++kv; }
        }
    };
    // A warp's sums of eight values of row q, and the block's totals.
    auto warpPart = [&](const double (&v)[8], int q) {
        const double w = warpSum8(v, lane);
        if ((lane & 3) == 0)
            red[warp][q * 8 + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)] = w;
    };
    auto totals = [&]() {
        __syncthreads();
        if (tid < n * 8)
        {
            double s = 0.0;
            for (int w = 0; w < kW; ++w) s += red[w][tid];
            tot[tid >> 3][tid & 7] = s;
        }
        __syncthreads();
    };
    // 1. all values, the negative ones, momentum, energy (one row after the
    // other: few live sums, so that four blocks share an SM)
#pragma unroll 1
    for (int q = 0; q < n; ++q)
    {
        double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        const T *row = buf + q * ldf;
        walk([&](int k, int iv, int jv, int kv) {
            const double vx = velD[iv], vy = velD[jv], vz = velD[kv];
            const T xt = row[k];
            const double x = (double)xt;
            v[0] += x;
            if (xt < T(0)) v[1] += x;
            v[2] = fma(vx, x, v[2]);
            v[3] = fma(vy, x, v[3]);
            v[4] = fma(vz, x, v[4]);
            v[5] = fma(fma(vx, vx, fma(vy, vy, vz * vz)), x, v[5]);
        });
        warpPart(v, q);
    }
    totals();
    bool anyFix = false;
    for (int q = 0; q < n; ++q) anyFix |= Positivity(tot[q][0] - tot[q][1], tot[q][1]).fix;
    if (anyFix && !wallG)
    {
        // Rare, the whole block alike: the moments of the kept part of every
        // row of the group ([6]: its mass), beside the sums of the raw row.
#pragma unroll 1
        for (int q = 0; q < n; ++q)
        {
            const Positivity pv(tot[q][0] - tot[q][1], tot[q][1]);
            double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            const T *row = buf + q * ldf;
            walk([&](int k, int iv, int jv, int kv) {
                const double vx = velD[iv], vy = velD[jv], vz = velD[kv];
                const double x = (double)row[k], h = pv.v1(x);
                v[0] += x;
                if (x < 0.0) v[1] += x;
                v[2] = fma(vx, h, v[2]);
                v[3] = fma(vy, h, v[3]);
                v[4] = fma(vz, h, v[4]);
                v[5] = fma(fma(vx, vx, fma(vy, vy, vz * vz)), h, v[5]);
                v[6] += h;
            });
            warpPart(v, q);
        }
        totals();
    }
    // 2. decisions and scalars, one row per lane
    if (tid < n)
    {
        const int q = tid, i = part[q];
        const double neg = tot[q][1], pos = tot[q][0] - neg, m = pos + neg;
        const Positivity pv(pos, neg);
        int flagged = 0;
        if (screenG)
        {
            if (!isfinite(tot[q][0]) || !isfinite(neg) || m <= 0.0) flagged = 1;
            else if (isfinite(nad.x) && isfinite(nad.y))
            {
                const double rn = m * dvN;
                const double slack = 0.1 * fmax(nad.y - nad.x, 1.0e-12) + 1.0e-9 +
                                     p.nadNoise * fmax(fabs(nad.x), fabs(nad.y));
                flagged = (rn < nad.x - slack || rn > nad.y + slack);
            }
        }
        a.flag[i] = flagged;
        if (pv.fix) atomicAdd(&a.sc->nfix, 1);
        if (flagged) a.flagList[atomicAdd(&a.sc->nflag, 1)] = i;
        else a.massPos[i] = m * dvN;
        mode[q] = flagged;
        par[q][5] = pv.s;
        par[q][6] = pv.fix ? 1.0 : 0.0;
        if (!wallG && !flagged)
        {
            const double M0 = (anyFix ? tot[q][6] : tot[q][0]) * dvN;
            if (!(M0 > 1.0e-30) || p.tauVar)
            {
                a.degList[atomicAdd(&a.sc->ndeg, 1)] = i;
                mode[q] = 1;
            }
            else
            {
                const double w = dvN / M0;
                const double ux = tot[q][2] * w, uy = tot[q][3] * w, uz = tot[q][4] * w;
                const double Tt =
                    fmax((tot[q][5] * w - (ux * ux + uy * uy + uz * uz)) * p.inv3R, 1.0e-6);
                const double twoRT = 2.0 * p.R * Tt, piT = kPi * twoRT;
                par[q][0] = ux; par[q][1] = uy; par[q][2] = uz;
                par[q][3] = 1.0 / twoRT;
                par[q][4] = p.lam * M0 / (piT * sqrt(piT));
                par[q][7] = M0; par[q][8] = Tt;
            }
        }
    }
    __syncthreads();

    if (wallG)
    {
        // Diffuse wall (BoundaryConditions/DiffuseWall.cpp:19-154), the forms
        // of finishWallStream.
        for (int j = tid; j < n * 3 * Nv; j += kNT)
        {
            const int q = j / (3 * Nv), r = j - q * 3 * Nv, d = r / Nv, x = r - d * Nv;
            const double RT2w = 2.0 * p.R * wallS[q][6], va = velD[x] - wallS[q][3 + d];
            const double e = exp(-va * va / RT2w);
            tab[q][d][x] = d == 0 ? e / (kPi * RT2w * sqrt(kPi * RT2w)) : e;
        }
        __syncthreads();
#pragma unroll 1
        for (int q = 0; q < n; ++q)
        {
            const bool fix = par[q][6] != 0.0;
            const double sc = par[q][5];
            double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            walk([&](int k, int iv, int jv, int kv) {
                const double cn = bcCn(3, velD[iv], velD[jv], velD[kv], wallS[q]);
                double h = (double)buf[q * ldf + k];
                if (fix) h = h < 0.0 ? 0.0 : h * sc;
                if (cn < 0.0) v[0] += cn * h * dvN;
                else if (cn > 0.0) v[1] += cn * (tab[q][0][iv] * tab[q][1][jv] * tab[q][2][kv]) * dvN;
            });
            warpPart(v, q);
        }
        totals();
        if (tid < n) par[tid][0] = (tot[tid][1] > 1.0e-30) ? (-tot[tid][0] / tot[tid][1]) : 1.0;
        __syncthreads();
#pragma unroll 1
        for (int q = 0; q < n; ++q)
        {
            const bool fix = par[q][6] != 0.0;
            const double sc = par[q][5], rhow = par[q][0];
            T *row = a.g + (size_t)part[q] * ldf;
            double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            walk([&](int k, int iv, int jv, int kv) {
                const double vx = velD[iv];
                const double cn = bcCn(3, vx, velD[jv], velD[kv], wallS[q]);
                double h = (double)buf[q * ldf + k];
                if (fix) h = h < 0.0 ? 0.0 : h * sc;
                if (cn > 0.0)
                {
                    const double Mw = rhow * (tab[q][0][iv] * tab[q][1][jv] * tab[q][2][kv]);
                    v[0] += vx * (Mw - h) * dvN;
                    h = Mw;
                }
                const T g1 = T(h);
                row[k] = g1;
                v[1] += (double)g1;
            });
            warpPart(v, q);
        }
        totals();
        if (tid < n)
        {
            const int i = part[tid];
            const double rhow = par[tid][0], Tw = wallS[tid][6];
            double *mac = a.macNew + 6 * (size_t)i;
            mac[0] = rhow; mac[1] = wallS[tid][3]; mac[2] = wallS[tid][4]; mac[3] = wallS[tid][5];
            mac[4] = Tw; mac[5] = rhow * p.R * Tw;
            a.dpx[i] = tot[tid][0];
            a.massEnd[i] = tot[tid][1] * dvN;
            a.minG[i] = 0.0;
        }
        return;
    }

    // 3. collision
    const double c1 = p.c1;
    for (int j = tid; j < n * 3 * Nv; j += kNT)
    {
        const int q = j / (3 * Nv), r = j - q * 3 * Nv, d = r / Nv, x = r - d * Nv;
        if (mode[q]) continue;
        const double va = velD[x] - par[q][d], e = exp(-va * va * par[q][3]);
        const double f = d == 0 ? par[q][4] * e : e;
        tab[q][d][x] = f;
    }
    __syncthreads();
    if (warp < n && !mode[warp])
    {
        // a row's macros by one warp: sums of velocity^0,1,2 times the axis
        // factors, one per lane
        const int q = warp;
        double Sl = 0.0;
        if (lane < 9)
        {
            const int d = lane / 3, mom = lane - 3 * d;
            for (int x = 0; x < Nv; ++x)
            {
                const double va = velD[x], e = tab[q][d][x];
                Sl += mom == 0 ? e : (mom == 1 ? va * e : va * va * e);
            }
        }
        double S[9];
#pragma unroll
        for (int j = 0; j < 9; ++j) S[j] = __shfl_sync(0xffffffffu, Sl, j);
        if (lane == 0)
        {
            const int i = part[q];
            const double N0 = c1 * (par[q][7] + dvN * S[0] * S[3] * S[6]);
            const double Nx = c1 * dvN * (tot[q][2] + S[1] * S[3] * S[6]);
            const double Ny = c1 * dvN * (tot[q][3] + S[0] * S[4] * S[6]);
            const double Nz = c1 * dvN * (tot[q][4] + S[0] * S[3] * S[7]);
            const double NE = c1 * dvN * (tot[q][5] + (S[2] * S[3] * S[6] + S[0] * S[5] * S[6] +
                                                       S[0] * S[3] * S[8]));
            double r2 = par[q][7], x2 = par[q][0], y2 = par[q][1], z2 = par[q][2], T2 = par[q][8];
            if (N0 > 1.0e-30)
            {
                const double iN0 = 1.0 / N0;
                r2 = N0; x2 = Nx * iN0; y2 = Ny * iN0; z2 = Nz * iN0;
                T2 = fmax((NE * iN0 - (x2 * x2 + y2 * y2 + z2 * z2)) * p.inv3R, 1.0e-6);
            }
            double *mac = a.macNew + 6 * (size_t)i;
            mac[0] = r2; mac[1] = x2; mac[2] = y2; mac[3] = z2; mac[4] = T2;
            mac[5] = r2 * p.R * T2;
            a.dpx[i] = 0.0;
            a.massEnd[i] = N0;
        }
    }
#pragma unroll 1
    for (int q = 0; q < n; ++q)
    {
        if (mode[q]) continue;
        const double am = c1 * par[q][5], lo = par[q][6] != 0.0 ? 0.0 : -INFINITY;
        const T *src = buf + q * ldf;
        T *row = a.g + (size_t)part[q] * ldf;
        T mn = T(INFINITY);
        walk([&](int k, int iv, int jv, int kv) {
            const double x = (double)src[k];
            const double lM = tab[q][0][iv] * (tab[q][1][jv] * tab[q][2][kv]);
            const T h = T(fma(am, x < lo ? lo : x, c1 * lM));
            row[k] = h;
            mn = mn < h ? mn : h;
        });
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            const T b = __shfl_xor_sync(0xffffffffu, mn, o);
            mn = mn < b ? mn : b;
        }
        if (lane == 0) redMin[warp][q] = mn;
    }
    __syncthreads();
    if (tid < n && !mode[tid])
    {
        T w = redMin[0][tid];
        for (int x = 1; x < kW; ++x) w = w < redMin[x][tid] ? w : redMin[x][tid];
        a.minG[part[tid]] = (double)w;
    }
}
