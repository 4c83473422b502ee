// coeffs_dev.cu -- the MLS transport coefficient tables built on the device,
// one thread per (stencil class, velocity node), equal bitwise to the host
// builder of coeffs.cpp (and so to the reference's MLS solve that the host
// builder restates, MLSTransport/MLSTransport.cpp:88-311 with the basis and
// weight of Core/MLSBasis.hpp:142-202 and the pivot-skip elimination of
// MLSTransport.cpp:20-62).
//
// The host builder is compiled without floating-point contraction, so this
// file is compiled with -fmad=false and follows the host's operations and
// loop orders one for one: foot point, per-slot weight and basis, the
// normal-equation matrix summed slot by slot, elimination with unit
// right-hand sides, and the coefficients w_s * (row 0 of the inverse . b_s).
#include <cuda_runtime.h>

#include <vector>

#include "coeffs.h"
#include "ctx.h"

namespace alebgk {

namespace {

struct ClassArgs
{
    int dim, Nv, V, S, ncls, mlsOrder;
    double dt, h, vmin, dv;
    int periodic[3];
    double L[3];
};

__device__ __forceinline__ double minImageD(double d, double L)
{
    return d - L * round(d / L);
}

__device__ __forceinline__ double weightSqD(double r2, double h)
{
    double q2 = r2 / (h * h);
    if (q2 >= 1.0) return 0.0;
    double w = 1.0 - q2;
    return w * w;
}

// Basis of size P (3, 6: 2-D linear, quadratic; 4, 10: 3-D) at the offset
// scaled by the support.
template <int P>
__device__ __forceinline__ void basisOf(double sx, double sy, double sz, double *b)
{
    b[0] = 1.0; b[1] = sx; b[2] = sy;
    if (P == 6)
    {
        b[3] = sx * sx; b[4] = sx * sy; b[5] = sy * sy;
    }
    if (P == 4 || P == 10) b[3] = sz;
    if (P == 10)
    {
        b[4] = sx * sx; b[5] = sy * sy; b[6] = sz * sz;
        b[7] = sx * sy; b[8] = sx * sz; b[9] = sy * sz;
    }
}

// One (class, node): the coefficients of its slots into cc, with the basis
// size fixed at compile time so that the normal matrix needs no indexed memory
// from its first term to the last back substitution (registers; of the
// quadratic 3-D one the compiler spills 372 bytes).  The elimination
// (partial pivots, |pivot| < 1e-30 skipped, as solveSkipGE) keeps its
// multipliers below the diagonal and its pivot rows in one word; the unit
// right-hand sides, of which only the first unknown is needed, then go
// through it one by one.  Same operations on the same values as the host's.
template <typename T, int P>
__device__ __forceinline__ void classNode(const ClassArgs &a, int c, int n, double xf, double yf,
                                          double zf, const double *__restrict__ sp,
                                          T *__restrict__ cc, int k, int *degen)
{
    constexpr bool d3 = P == 4 || P == 10;
    const int V = a.V;
    // weight and scaled offset of slot s; false outside the support
    auto slotAt = [&](int s, double &ws, double &sx, double &sy, double &sz) {
        double dx = sp[3 * s] - xf, dy = sp[3 * s + 1] - yf;
        double dz = d3 ? sp[3 * s + 2] - zf : 0.0;
        if (a.periodic[0]) dx = minImageD(dx, a.L[0]);
        if (a.periodic[1]) dy = minImageD(dy, a.L[1]);
        if (d3 && a.periodic[2]) dz = minImageD(dz, a.L[2]);
        const double r2 = dx * dx + dy * dy + dz * dz;
        ws = weightSqD(r2, a.h);
        if (ws < 1.0e-30) return false;
        sx = dx / a.h;
        sy = dy / a.h;
        sz = dz / a.h;
        return true;
    };
    double A[P][P];
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
        for (int j = 0; j < P; ++j) A[i][j] = 0.0;
    bool any = false;
#pragma unroll 1
    for (int s = 1; s < n; ++s)
    {
        double ws, sx, sy, sz, b[P];
        if (!slotAt(s, ws, sx, sy, sz)) continue;
        basisOf<P>(sx, sy, sz, b);
#pragma unroll
        for (int i = 0; i < P; ++i)
        {
            const double wb = ws * b[i];
#pragma unroll
            for (int j = 0; j < P; ++j) A[i][j] += wb * b[j];
        }
        any = true;
    }
    if (!any) { cc[k] = (T)1.0; return; }
    unsigned long long piv = 0;      // pivot row of column q in bits [4 q, 4 q + 4)
    unsigned good = 0;               // columns with a pivot
#pragma unroll
    for (int col = 0; col < P; ++col)
    {
        int pr = col;
        double mx = fabs(A[col][col]);
#pragma unroll
        for (int row = col + 1; row < P; ++row)
            if (fabs(A[row][col]) > mx)
            {
                mx = fabs(A[row][col]);
                pr = row;
            }
        piv |= (unsigned long long)pr << (4 * col);
#pragma unroll
        for (int row = col + 1; row < P; ++row)
        {
            const bool sw = pr == row;
#pragma unroll
            for (int j = col; j < P; ++j)
            {
                const double t = A[col][j];
                A[col][j] = sw ? A[row][j] : t;
                A[row][j] = sw ? t : A[row][j];
            }
        }
        const double d = A[col][col];
        if (!(fabs(d) < 1.0e-30))
        {
            good |= 1u << col;
#pragma unroll
            for (int row = col + 1; row < P; ++row)
            {
                const double f = A[row][col] / d;
#pragma unroll
                for (int j = col + 1; j < P; ++j) A[row][j] -= f * A[col][j];
                A[row][col] = f;     // the multiplier; nothing reads the column again
            }
        }
    }
    if (good != (1u << P) - 1) atomicAdd(degen + c, 1);
    double B0[P];
#pragma unroll
    for (int m = 0; m < P; ++m)
    {
        double x[P];
#pragma unroll
        for (int i = 0; i < P; ++i) x[i] = i == m ? 1.0 : 0.0;
#pragma unroll
        for (int col = 0; col < P; ++col)
        {
            const int pr = (int)(piv >> (4 * col)) & 15;
#pragma unroll
            for (int row = col + 1; row < P; ++row)
            {
                const bool sw = pr == row;
                const double t = x[col];
                x[col] = sw ? x[row] : t;
                x[row] = sw ? t : x[row];
            }
            if (good >> col & 1u)
#pragma unroll
                for (int row = col + 1; row < P; ++row) x[row] -= A[row][col] * x[col];
        }
#pragma unroll
        for (int i = P - 1; i >= 0; --i)
        {
            double s = x[i];
#pragma unroll
            for (int j = i + 1; j < P; ++j) s -= A[i][j] * x[j];
            x[i] = fabs(A[i][i]) > 1.0e-30 ? s / A[i][i] : 0.0;
        }
        B0[m] = x[0];
    }
    // FP32 tables: the largest coefficient takes the rounding of the node's
    // sum, as roundCoefFP32 does on the host (same order, same operations).
    double s64 = 0.0, s32 = 0.0, big = -1.0;
    int smax = 0;
#pragma unroll 1
    for (int s = 1; s < n; ++s)
    {
        double ws, sx, sy, sz, b[P];
        if (!slotAt(s, ws, sx, sy, sz)) continue;
        basisOf<P>(sx, sy, sz, b);
        double acc = 0.0;
#pragma unroll
        for (int m = 0; m < P; ++m) acc += B0[m] * b[m];
        const double w = ws * acc;
        cc[(size_t)s * V + k] = (T)w;
        if (sizeof(T) == 4)
        {
            s64 += w;
            s32 += (double)(T)w;
            if (fabs(w) > big) { big = fabs(w); smax = s; }
        }
    }
    if (sizeof(T) == 4 && big > 0.0)
    {
        const size_t q = (size_t)smax * V + k;
        cc[q] = (T)((double)cc[q] + (s64 - s32));
    }
}

// Per class: rep position (3), mesh velocity (3), wall state (7), then the
// positions of slots 1..nsl-1 (3 each) at [c][S][3].  A block is of one
// class (grid y and z), so its threads take one basis size.
// Bound: the chain of dependent FP64 operations of a node (about 280 a slot in
// the support and 4 000 for the elimination, uncontracted) at two warps a
// scheduler: the FP64 pipe is busy 39 % of the cycles.  Measured, cavity3d-cube Nx 40 Nv 10
// (1 099 classes x 1 000 nodes, FP32 tables): quadratic 14.2 ms with both
// matrices in local memory, read and written for every slot; 3.1 ms in
// registers (255, two blocks an SM).  Linear 1.92 -> 1.87 ms.
template <typename T>
__global__ void __launch_bounds__(128, 2)
k_class_tables(ClassArgs a, int order0, const int *__restrict__ boundary,
               const int *__restrict__ nsl, const double *__restrict__ rep,
               const double *__restrict__ slotPos, T *__restrict__ table, int *__restrict__ degen)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = blockIdx.z * gridDim.y + blockIdx.y;
    if (k >= a.V || c >= a.ncls) return;
    const int ndim = a.dim, Nv = a.Nv, V = a.V;
    const bool bnd = boundary[c] != 0;
    const int order = bnd ? 1 : order0;
    const double *rp = rep + 13 * (size_t)c;
    const double *wl = rp + 6;
    T *cc = table + (size_t)c * a.S * V;
    const int iv = k % Nv, jv = (k / Nv) % Nv, kv = (ndim == 3) ? k / (Nv * Nv) : 0;
    const double vx = fma((double)iv, a.dv, a.vmin);
    const double vy = fma((double)jv, a.dv, a.vmin);
    const double vz = fma((double)kv, a.dv, a.vmin);
    if (bnd)
    {
        const double ca = vx - wl[3], cb = vy - wl[4];
        const double cn = (ndim == 3) ? fma(vz - wl[5], wl[2], fma(ca, wl[0], cb * wl[1]))
                                      : fma(ca, wl[0], cb * wl[1]);
        if (cn >= 0.0) { cc[k] = (T)1.0; return; }
    }
    const double xf = rp[0] - (vx - rp[3]) * a.dt;
    const double yf = rp[1] - (vy - rp[4]) * a.dt;
    const double zf = rp[2] - (vz - rp[5]) * a.dt;
    const int n = nsl[c];
    const double *sp = slotPos + (size_t)c * a.S * 3;
    if (ndim == 3)
    {
        if (order >= 2) classNode<T, 10>(a, c, n, xf, yf, zf, sp, cc, k, degen);
        else classNode<T, 4>(a, c, n, xf, yf, zf, sp, cc, k, degen);
    }
    else if (order >= 2) classNode<T, 6>(a, c, n, xf, yf, zf, sp, cc, k, degen);
    else classNode<T, 3>(a, c, n, xf, yf, zf, sp, cc, k, degen);
}

}  // namespace

cudaError_t buildTablesDevice(const CoeffInput &in, const CoeffTables &cls, int order,
                              void *table, bool f64, std::vector<int> &degenerate,
                              cudaStream_t st)
{
    const int ncls = cls.ncls, S = cls.S, V = cls.V;
    std::vector<int> bnd(ncls), nsl(ncls);
    std::vector<double> rep(13 * (size_t)ncls), pos((size_t)ncls * S * 3, 0.0);
    for (int c = 0; c < ncls; ++c)
    {
        const int r = cls.rep[c];
        bnd[c] = in.boundary[r];
        const bool packed = cls.slots.empty();
        nsl[c] = packed ? cls.repNslot[c] : cls.nslot[r];
        double *o = &rep[13 * (size_t)c];
        for (int q = 0; q < 3; ++q) { o[q] = in.xyz[3 * (size_t)r + q]; o[3 + q] = in.meshv[3 * (size_t)r + q]; }
        for (int q = 0; q < 7; ++q) o[6 + q] = in.wall[7 * (size_t)r + q];
        const int *sl = packed ? &cls.repSlots[(size_t)c * S] : &cls.slots[(size_t)r * S];
        for (int s = 1; s < nsl[c]; ++s)
            for (int q = 0; q < 3; ++q) pos[((size_t)c * S + s) * 3 + q] = in.xyz[3 * (size_t)sl[s] + q];
    }
    ClassArgs a{};
    a.dim = in.dim; a.Nv = in.Nv; a.V = V; a.S = S; a.ncls = ncls; a.mlsOrder = order;
    a.dt = in.dt; a.h = in.h; a.vmin = in.vmin; a.dv = in.dv;
    for (int q = 0; q < 3; ++q) { a.periodic[q] = in.periodic[q] ? 1 : 0; a.L[q] = in.L[q]; }
    int *dBnd = nullptr, *dNsl = nullptr, *dDeg = nullptr;
    double *dRep = nullptr, *dPos = nullptr;
    auto freeAll = [&]() {
        for (void *p : {(void *)dBnd, (void *)dNsl, (void *)dDeg, (void *)dRep, (void *)dPos})
            if (p) cudaFree(p);
    };
    cudaError_t e = cudaMalloc(&dBnd, 4 * (size_t)ncls);
    if (e == cudaSuccess) e = cudaMalloc(&dNsl, 4 * (size_t)ncls);
    if (e == cudaSuccess) e = cudaMalloc(&dDeg, 4 * (size_t)ncls);
    if (e == cudaSuccess) e = cudaMalloc(&dRep, 8 * rep.size());
    if (e == cudaSuccess) e = cudaMalloc(&dPos, 8 * pos.size());
    if (e == cudaSuccess) e = cudaMemcpyAsync(dBnd, bnd.data(), 4 * (size_t)ncls, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dNsl, nsl.data(), 4 * (size_t)ncls, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(dDeg, 0, 4 * (size_t)ncls, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dRep, rep.data(), 8 * rep.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dPos, pos.data(), 8 * pos.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(table, 0, (size_t)ncls * S * V * (f64 ? 8 : 4), st);
    if (e == cudaSuccess)
    {
        const dim3 grid = yzGrid((V + 127) / 128, ncls);
        if (f64)
            k_class_tables<double><<<grid, 128, 0, st>>>(a, order, dBnd, dNsl, dRep, dPos,
                                                         static_cast<double *>(table), dDeg);
        else
            k_class_tables<float><<<grid, 128, 0, st>>>(a, order, dBnd, dNsl, dRep, dPos,
                                                        static_cast<float *>(table), dDeg);
        e = cudaGetLastError();
    }
    degenerate.assign(ncls, 0);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(degenerate.data(), dDeg, 4 * (size_t)ncls, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    freeAll();
    return e;
}

}  // namespace alebgk
