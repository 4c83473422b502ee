// tiles.cu -- coefficient-gather transport of a 3-D cloud that is a lattice
// for the most part (a cavity with bodies in it): the particles inside it go
// in tiles of 4 x 2 lattice neighbours, those of the layers along its walls in
// strips of four, the rest through the plain gather.
//
// A tile is eight particles of one full stencil class (80 neighbours at the
// lattice offsets |o|^2 <= 6) whose neighbours, by their own slot lists, lie
// in rows of consecutive particle indices: row (dz, y), y = -2..3, holds the
// x = -2..5 around the tile.  The plan checks every slot of every member on
// the device, so holes, surfaces and cut rows need no rules: a tile that does
// not hold leaves its particles to the strips and the gather.  A strip is four
// particles along x of one class whose slots are whole rows of the template
// (a wall layer's: some rows are missing, none in part), checked the same way.
//
// Transport: one warp per tile (or strip) and chunk of velocities.  Each
// neighbour value is loaded once for the tile and each coefficient once per
// row pair, 180 + 160 loads for the 640 FMAs of eight particles, 144 + 80 for
// a strip's 320 (the gather loads a value and a coefficient for every FMA and
// is bound by L1 throughput), beside slot 0: the particle's own value, whose
// coefficient is 1 for a node whose foot point has no neighbour in the support
// (a step of more than the support's reach) and 0 for every other.  Every
// particle sums its slots in slot order, as the gather does.
// Measured, cavity3d-cube Nx 40 Nv 10 FP32: transport 1.53 ms by the gather
// alone; 0.756 ms with tiles (0.307 for 70 % of the particles, 0.456 for the
// gather of the rest).  The strips take the step there from 985 to 909 us, the
// pairs of nodes in the gather of the rest to 877.  Tiles and rest run at 69 and
// 75 % of L1's throughput.  (Which clouds take them: takeTiles in step.cu.)
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "coeffs.h"
#include "ctx.h"
#include "vel.cuh"

namespace alebgk {

namespace {

// A tile: class, its two first members, then the index of x = 0 of each row
// (dz + 2) * 6 + y + 2 (rows outside every member's stencil unused).
constexpr int kTileInts = 33;

// A strip: class, its first member, then for each row (dz + 2) * 5 + dy + 2
// the index of x = 0 (-1: no such row) and the slot of its first offset.
constexpr int kStripInts = 52;

__host__ __device__ constexpr int off3(int dx, int dy, int dz)
{
    int n = 0;
    for (int z = -2; z <= 2; ++z)
        for (int y = -2; y <= 2; ++y)
            for (int x = -2; x <= 2; ++x)
            {
                if (x * x + y * y + z * z > 6) continue;
                if (x == dx && y == dy && z == dz) return n;
                ++n;
            }
    return -1;
}
// Slot of an offset in a full class: the self first, then template order.
__host__ __device__ constexpr int slot3(int dx, int dy, int dz)
{
    const int o = off3(dx, dy, dz), self = off3(0, 0, 0);
    return o < 0 ? -1 : (o == self ? 0 : (o < self ? o + 1 : o));
}
static_assert(slot3(1, 1, 2) == 80 && slot3(-1, -1, -2) == 1, "80 neighbours");

struct Tmpl3
{
    signed char d[81][3];     // offset of each slot
    signed char slot[125];    // slot of (dz + 2) * 25 + (dy + 2) * 5 + dx + 2
};

Tmpl3 makeTmpl3()
{
    Tmpl3 t{};
    for (int z = -2; z <= 2; ++z)
        for (int y = -2; y <= 2; ++y)
            for (int x = -2; x <= 2; ++x)
            {
                const int s = slot3(x, y, z);
                t.slot[(z + 2) * 25 + (y + 2) * 5 + x + 2] = (signed char)s;
                if (s >= 0) { t.d[s][0] = (signed char)x; t.d[s][1] = (signed char)y; t.d[s][2] = (signed char)z; }
            }
    return t;
}

// The lattice's columns: spacing, and a particle of a full class as the origin
// (any other particle may lie off the lattice, a wall point between two columns).
struct TileGrid
{
    double x0, y0, hx, hy;
    __device__ long long col(const double *pos, int i) const
    {
        return llround((pos[3 * (size_t)i] - x0) / hx);
    }
    __device__ long long row(const double *pos, int i) const
    {
        return llround((pos[3 * (size_t)i + 1] - y0) / hy);
    }
};

__device__ __forceinline__ int rowSlot(const Tmpl3 &t, int dy, int dz)
{
    if (dy < -2 || dy > 2) return -1;
    return t.slot[(dz + 2) * 25 + (dy + 2) * 5 + 2];
}

// Index of x = 0 of row (dz, y) of the tile with first members i and j.
__device__ __forceinline__ int tileRow(const Tmpl3 &t, const int *slots, int S, int i, int j, int y,
                                       int dz)
{
    const int s = rowSlot(t, y, dz);
    if (s >= 0) return slots[(size_t)i * S + s];
    const int q = rowSlot(t, y - 1, dz);
    return q >= 0 ? slots[(size_t)j * S + q] : -1;
}

// One warp per particle: whether a tile starts there; marks its members.
// Tiles start on every fourth column and every second row, and each member's own
// column and row must be the start's plus its place in the tile.  So no two
// tiles share a particle, whatever the cloud, and N / 8 places are enough: as a
// member of a first row a particle has one start, i = itself - (column mod 4);
// as one of a second row (odd rows) likewise one j, and j's slots name one i.
__global__ void k_tile_mark(Tmpl3 t, TileGrid g, int N, int S, const double *__restrict__ pos,
                            const int *__restrict__ cls, const int *__restrict__ slots,
                            const int *__restrict__ full, int *__restrict__ flag,
                            int *__restrict__ covered)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= N) return;
    const int c = cls[i];
    bool ok = full[c] != 0 && i + 3 < N;
    int j = 0;
    const long long ix = ok ? g.col(pos, i) : 0, iy = ok ? g.row(pos, i) : 0;
    ok = ok && (ix & 3) == 0 && (iy & 1) == 0;
    if (ok)
    {
        j = slots[(size_t)i * S + t.slot[2 * 25 + 3 * 5 + 2]];      // (0, 1, 0)
        ok = j + 3 < N;
        for (int m = 0; m < 4 && ok; ++m) ok = cls[i + m] == c && cls[j + m] == c;
    }
    if (ok && lane < 8)
    {
        const int mem = lane >> 2 ? j + (lane & 3) : i + (lane & 3);
        ok = g.col(pos, mem) == ix + (lane & 3) && g.row(pos, mem) == iy + (lane >> 2);
    }
    if (ok)
        for (int q = lane; q < 8 * 80; q += 32)
        {
            const int m = q / 80, s = 1 + q % 80, b = m >> 2, x = m & 3;
            const int mem = b ? j + x : i + x;
            const int y = t.d[s][1] + b, dz = t.d[s][2];
            const int base = y == 0 && dz == 0 ? i : (y == 1 && dz == 0 ? j
                                                                        : tileRow(t, slots, S, i, j, y, dz));
            ok = ok && slots[(size_t)mem * S + s] == base + x + t.d[s][0];
        }
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) flag[i] = ok;
    if (ok && lane < 8) covered[lane >> 2 ? j + (lane & 3) : i + (lane & 3)] = 1;
}

// The same for strips, of the particles that no tile covers (a tile's have 1 in
// covered; strips write 2 for their own members, which no other strip has, by
// their columns).  first[c] is -1 for a class without the strips' form, else
// the class's row of rowFirst: per template row the slot of its first offset,
// -1 where the row is missing.
__global__ void k_strip_mark(Tmpl3 t, TileGrid g, int N, int S, const double *__restrict__ pos,
                             const int *__restrict__ cls, const int *__restrict__ nslot,
                             const int *__restrict__ slots, const int *__restrict__ first,
                             const signed char *__restrict__ rowFirst, int *__restrict__ strip,
                             int *__restrict__ covered)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= N) return;
    const int c = cls[i];
    bool ok = first[c] >= 0 && i + 3 < N && covered[i] != 1 && nslot[i] > 1;
    const long long ix = ok ? g.col(pos, i) : 0;
    ok = ok && (ix & 3) == 0;
    for (int m = 1; m < 4 && ok; ++m)
        ok = cls[i + m] == c && covered[i + m] != 1 && g.col(pos, i + m) == ix + m;
    if (ok)
    {
        const signed char *rs = rowFirst + 25 * first[c];
        const int ns = nslot[i];
        for (int q = lane; q < 4 * 25; q += 32)
        {
            const int m = q / 25, r = q % 25, s0 = rs[r];
            if (s0 < 0) continue;
            const int dy = r % 5 - 2, dz = r / 5 - 2;
            const int w = dy * dy + dz * dz <= 2 ? 2 : 1;     // offsets -w..w
            // (the first offset of the row is x = -w)
            const int base = slots[(size_t)i * S + s0] + w;
            int s = s0;
            for (int dx = -w; dx <= w; ++dx)
            {
                if (r == 12 && dx == 0) continue;             // the self
                ok = ok && s < ns && slots[(size_t)(i + m) * S + s] == base + m + dx;
                ++s;
            }
        }
    }
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) strip[i] = ok;
    if (ok && lane < 4) covered[i + lane] = 2;
}

// One block: places of the tiles, of the strips and of the particles outside
// both, in particle order, and their counts.
__global__ void __launch_bounds__(1024)
k_tile_scan(int N, int *flag, int *strip, int *covered, int *count)
{
    __shared__ int sh[3][1024];
    const int t = threadIdx.x, per = (N + 1023) / 1024;
    const int a = min(t * per, N), b = min(a + per, N);
    int n[3] = {0, 0, 0};
    for (int i = a; i < b; ++i)
    {
        n[0] += flag[i];
        n[1] += strip[i];
        n[2] += !covered[i];
    }
    for (int q = 0; q < 3; ++q) sh[q][t] = n[q];
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1)
    {
        int x[3];
        for (int q = 0; q < 3; ++q) x[q] = t >= o ? sh[q][t - o] : 0;
        __syncthreads();
        for (int q = 0; q < 3; ++q) sh[q][t] += x[q];
        __syncthreads();
    }
    for (int q = 0; q < 3; ++q) n[q] = sh[q][t] - n[q];
    for (int i = a; i < b; ++i)
    {
        flag[i] = flag[i] ? n[0]++ : -1;
        strip[i] = strip[i] ? n[1]++ : -1;
        covered[i] = covered[i] ? -1 : n[2]++;
    }
    if (t == 1023)
        for (int q = 0; q < 3; ++q) count[q] = sh[q][1023];
}

__global__ void k_tile_write(Tmpl3 t, int N, int S, const int *__restrict__ cls,
                             const int *__restrict__ slots, const int *__restrict__ flag,
                             const int *__restrict__ strip, const int *__restrict__ covered,
                             const int *__restrict__ first,
                             const signed char *__restrict__ rowFirst, int *__restrict__ tiles,
                             int *__restrict__ strips, int *__restrict__ rest)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= N) return;
    if (lane == 0 && covered[i] >= 0) rest[covered[i]] = i;
    if (strip[i] >= 0)
    {
        int *o = strips + (size_t)strip[i] * kStripInts;
        const int s0 = lane < 25 ? rowFirst[25 * first[cls[i]] + lane] : -1;
        if (lane < 25)
        {
            const int dy = lane % 5 - 2, dz = lane / 5 - 2, w = dy * dy + dz * dz <= 2 ? 2 : 1;
            o[2 + 2 * lane] = s0 >= 0 ? slots[(size_t)i * S + s0] + w : -1;
            o[3 + 2 * lane] = s0;
        }
        if (lane == 0)
        {
            o[0] = cls[i];
            o[1] = i;
        }
    }
    if (flag[i] < 0) return;
    int *o = tiles + (size_t)flag[i] * kTileInts;
    const int j = slots[(size_t)i * S + t.slot[2 * 25 + 3 * 5 + 2]];
    if (lane < 30)
    {
        const int dz = lane / 6 - 2, y = lane % 6 - 2;
        o[3 + lane] = dz == 0 && y == 0 ? i : (dz == 0 && y == 1 ? j : tileRow(t, slots, S, i, j, y, dz));
    }
    if (lane == 0)
    {
        o[0] = cls[i];
        o[1] = i;
        o[2] = j;
    }
}

template <int... I, typename F>
__device__ __forceinline__ void unroll3Impl(std::integer_sequence<int, I...>, F &&f)
{
    (f(std::integral_constant<int, I>{}), ...);
}
template <int M, typename F>
__device__ __forceinline__ void unroll3(F &&f)
{
    unroll3Impl(std::make_integer_sequence<int, M>{}, f);
}

// Grid (velocity chunks, blocks of eight tiles in y and z).
template <typename T, int VPL>
__global__ void __launch_bounds__(256, 2)
k_transport_tiles(const T *__restrict__ f, T *__restrict__ g, const T *__restrict__ coef,
                  const int *__restrict__ tiles, const int *__restrict__ count, int S, int V, int ldf,
                  const StepScalars *__restrict__ sc)
{
    typedef Vel<T, VPL> L;
    typedef typename L::V VT;
    const int tile = (blockIdx.z * gridDim.y + blockIdx.y) * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (tile >= __ldg(count)) return;
    const int k = (blockIdx.x * 32 + lane) * VPL;
    if (k >= V) return;
    const int *tl = tiles + (size_t)tile * kTileInts;
    const T *cc = coef + (size_t)__ldg(tl) * S * V + k;
    const T *fk = f + k;
    auto coefAt = [&](int s) { return __ldg(reinterpret_cast<const VT *>(cc + (size_t)s * V)); };
    // the particles' own values first (slot 0)
    VT acc[2][4];
    const VT c0 = coefAt(0);
#pragma unroll
    for (int b = 0; b < 2; ++b)
    {
        const T *own = fk + (size_t)__ldg(tl + 1 + b) * ldf;
#pragma unroll
        for (int x = 0; x < 4; ++x)
            acc[b][x] = L::fma(c0, __ldg(reinterpret_cast<const VT *>(own + (size_t)x * ldf)),
                               L::zero());
    }
    unroll3<30>([&](auto R) {
        constexpr int r = decltype(R)::value, dz = r / 6 - 2, y = r % 6 - 2;
        // member row 0 meets this row at offset dy = y, member row 1 at y - 1
        constexpr bool m0 = slot3(0, y, dz) >= 0, m1 = slot3(0, y - 1, dz) >= 0;
        if constexpr (m0 || m1)
        {
            const T *row = fk + (size_t)__ldg(tl + 3 + r) * ldf;
            VT v[8];
            unroll3<8>([&](auto X) {
                constexpr int x = decltype(X)::value - 2, z = decltype(R)::value / 6 - 2;
                constexpr int w = decltype(R)::value % 6 - 2;
                if constexpr ((x > -2 && x < 5) || slot3(2, w, z) >= 0 || slot3(2, w - 1, z) >= 0)
                    v[x + 2] = __ldg(reinterpret_cast<const VT *>(row + (long long)x * ldf));
            });
            unroll3<10>([&](auto D) {
                constexpr int bb = decltype(D)::value / 5, dx = decltype(D)::value % 5 - 2;
                constexpr int s = slot3(dx, decltype(R)::value % 6 - 2 - bb,
                                        decltype(R)::value / 6 - 2);
                if constexpr (s > 0)
                {
                    const VT c = coefAt(s);
                    unroll3<4>([&](auto M) {
                        constexpr int m = decltype(M)::value;
                        constexpr int bm = decltype(D)::value / 5, at = m + decltype(D)::value % 5;
                        acc[bm][m] = L::fma(c, v[at], acc[bm][m]);
                    });
                }
            });
        }
    });
    const T scale = T(sc->scale);
#pragma unroll
    for (int b = 0; b < 2; ++b)
    {
        T *o = g + (size_t)__ldg(tl + 1 + b) * ldf + k;
#pragma unroll
        for (int x = 0; x < 4; ++x)
            *reinterpret_cast<VT *>(o + (size_t)x * ldf) = L::mul(acc[b][x], scale);
    }
}

// Grid (velocity chunks, blocks of eight strips in y and z).
template <typename T, int VPL>
__global__ void __launch_bounds__(256, 3)
k_transport_strips(const T *__restrict__ f, T *__restrict__ g, const T *__restrict__ coef,
                   const int *__restrict__ strips, const int *__restrict__ count, int S, int V,
                   int ldf, const StepScalars *__restrict__ sc)
{
    typedef Vel<T, VPL> L;
    typedef typename L::V VT;
    const int strip = (blockIdx.z * gridDim.y + blockIdx.y) * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (strip >= __ldg(count)) return;
    const int k = (blockIdx.x * 32 + lane) * VPL;
    if (k >= V) return;
    const int *st = strips + (size_t)strip * kStripInts;
    const T *cc = coef + (size_t)__ldg(st) * S * V + k;
    const int i = __ldg(st + 1);
    const T *fk = f + k;
    // the particles' own values first (slot 0)
    VT acc[4];
    {
        const VT c0 = __ldg(reinterpret_cast<const VT *>(cc));
        const T *own = fk + (size_t)i * ldf;
#pragma unroll
        for (int m = 0; m < 4; ++m)
            acc[m] = L::fma(c0, __ldg(reinterpret_cast<const VT *>(own + (size_t)m * ldf)), L::zero());
    }
    unroll3<25>([&](auto Q) {
        constexpr int q = decltype(Q)::value, dy = q % 5 - 2, dz = q / 5 - 2;
        if constexpr (dy * dy + dz * dz <= 6 && slot3(0, dy, dz) >= 0)
        {
            const int base = __ldg(st + 2 + 2 * q);
            if (base >= 0)
            {
                const T *cs = cc + (size_t)__ldg(st + 3 + 2 * q) * V;
                const T *row = fk + (size_t)base * ldf;
                VT v[8];
                unroll3<8>([&](auto X) {
                    constexpr int x = decltype(X)::value - 2, qq = decltype(Q)::value;
                    if constexpr ((x > -2 && x < 5) || slot3(2, qq % 5 - 2, qq / 5 - 2) >= 0)
                        v[x + 2] = __ldg(reinterpret_cast<const VT *>(row + (long long)x * ldf));
                });
                unroll3<5>([&](auto D) {
                    constexpr int dx = decltype(D)::value - 2, qq = decltype(Q)::value;
                    constexpr int s = slot3(dx, qq % 5 - 2, qq / 5 - 2);
                    if constexpr (s > 0)
                    {
                        // the offset's place in its row (the self has none)
                        constexpr int w = slot3(2, qq % 5 - 2, qq / 5 - 2) >= 0 ? 2 : 1;
                        constexpr int at = dx + w - (qq == 12 && dx > 0 ? 1 : 0);
                        const VT c = __ldg(reinterpret_cast<const VT *>(cs + (size_t)at * V));
                        unroll3<4>([&](auto M) {
                            constexpr int m = decltype(M)::value;
                            acc[m] = L::fma(c, v[m + decltype(D)::value], acc[m]);
                        });
                    }
                });
            }
        }
    });
    const T scale = T(sc->scale);
    T *o = g + (size_t)i * ldf + k;
#pragma unroll
    for (int m = 0; m < 4; ++m)
        *reinterpret_cast<VT *>(o + (size_t)m * ldf) = L::mul(acc[m], scale);
}

}  // namespace

// The classes on the lattice, by their representatives (the spacing comes from
// a particle of 80 neighbours): full ones, whose slots are the whole template
// in order, and ones whose slots are whole rows of it in order, with the slot
// of each row's first offset.  False where there is no full class.
static bool latticeClasses(const CoeffInput &in, const CoeffTables &tb, const Tmpl3 &t,
                           std::vector<int> &full, std::vector<int> &first,
                           std::vector<signed char> &rowFirst, TileGrid &g)
{
    full.assign(tb.ncls, 0);
    first.assign(tb.ncls, -1);
    rowFirst.clear();
    if (tb.S < 81) return false;
    const bool packed = tb.slots.empty();
    auto slotsOf = [&](int c, int &ns) -> const int * {
        const int r = tb.rep[c];
        ns = packed ? tb.repNslot[c] : tb.nslot[r];
        return packed ? &tb.repSlots[(size_t)c * tb.S] : &tb.slots[(size_t)r * tb.S];
    };
    double h[3] = {0, 0, 0};
    auto onLattice = [&](const double *p, const double *q, int a, int d) {
        return std::fabs((q[a] - p[a]) / h[a] - d) < 1e-6;
    };
    bool any = false;
    for (int c = 0; c < tb.ncls; ++c)
    {
        int ns;
        const int *sl = slotsOf(c, ns);
        if (ns != 81 || in.boundary[tb.rep[c]]) continue;
        const double *p = in.xyz + 3 * (size_t)tb.rep[c];
        if (!any)
        {
            h[0] = in.xyz[3 * (size_t)sl[slot3(1, 0, 0)]] - p[0];
            h[1] = in.xyz[3 * (size_t)sl[slot3(0, 1, 0)] + 1] - p[1];
            h[2] = in.xyz[3 * (size_t)sl[slot3(0, 0, 1)] + 2] - p[2];
        }
        bool ok = h[0] > 0 && h[1] > 0 && h[2] > 0;
        for (int s = 1; s < 81 && ok; ++s)
            for (int a = 0; a < 3 && ok; ++a)
                ok = onLattice(p, in.xyz + 3 * (size_t)sl[s], a, t.d[s][a]);
        if (ok && !any) g = TileGrid{p[0], p[1], h[0], h[1]};
        full[c] = ok;
        any = any || ok;
    }
    if (!any) return false;
    for (int c = 0; c < tb.ncls; ++c)
    {
        int ns;
        const int *sl = slotsOf(c, ns);
        const double *p = in.xyz + 3 * (size_t)tb.rep[c];
        signed char rs[25];
        std::fill(rs, rs + 25, (signed char)-1);
        bool ok = ns <= 81;
        int s = 1;
        for (int r = 0; r < 25 && ok; ++r)
        {
            const int dy = r % 5 - 2, dz = r / 5 - 2;
            if (slot3(0, dy, dz) < 0) continue;
            const int w = slot3(2, dy, dz) >= 0 ? 2 : 1;
            auto at = [&](int q, int dx) {
                const double *x = in.xyz + 3 * (size_t)sl[q];
                return onLattice(p, x, 0, dx) && onLattice(p, x, 1, dy) && onLattice(p, x, 2, dz);
            };
            if (s >= ns || !at(s, -w)) continue;      // the row is missing
            rs[r] = (signed char)s;
            for (int dx = -w; dx <= w && ok; ++dx)
            {
                if (r == 12 && dx == 0) continue;
                ok = s < ns && at(s, dx);
                ++s;
            }
        }
        if (!ok || s != ns) continue;                 // other slots, or part of a row
        first[c] = (int)(rowFirst.size() / 25);
        rowFirst.insert(rowFirst.end(), rs, rs + 25);
    }
    return true;
}

// Plans the tiles and strips of the uploaded cloud (classes and slot lists on
// the device); c->d.tileCount holds their numbers and that of the rest.
cudaError_t buildTiles(alebgk_ctx *c, const CoeffInput &in, const CoeffTables &tb)
{
    static const Tmpl3 t = makeTmpl3();
    DeviceBuffers &d = c->d;
    const int N = c->sp.N;
    std::vector<int> full, first;
    std::vector<signed char> rowFirst;
    TileGrid g{0, 0, 1, 1};
    latticeClasses(in, tb, t, full, first, rowFirst, g);
    const size_t n = std::max<size_t>(full.size(), 1);
    rowFirst.resize(std::max<size_t>(rowFirst.size(), 25), -1);
    int *dCls = nullptr;              // full, first, then rowFirst
    cudaError_t e = cudaMalloc(&dCls, 8 * n + rowFirst.size());
    signed char *dRow = reinterpret_cast<signed char *>(dCls + 2 * n);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dCls, full.data(), 4 * full.size(), cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dCls + n, first.data(), 4 * first.size(), cudaMemcpyHostToDevice,
                            c->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dRow, rowFirst.data(), rowFirst.size(), cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d.tileCovered, 0, 4 * (size_t)N, c->stream);
    if (e == cudaSuccess)
    {
        const int blocks = (int)(((long long)N * 32 + 255) / 256);
        k_tile_mark<<<blocks, 256, 0, c->stream>>>(t, g, N, tb.S, d.pos, d.cls, d.slots, dCls,
                                                   d.tileFlag, d.tileCovered);
        k_strip_mark<<<blocks, 256, 0, c->stream>>>(t, g, N, tb.S, d.pos, d.cls, d.nslot, d.slots,
                                                    dCls + n, dRow, d.stripFlag, d.tileCovered);
        k_tile_scan<<<1, 1024, 0, c->stream>>>(N, d.tileFlag, d.stripFlag, d.tileCovered,
                                               d.tileCount);
        k_tile_write<<<blocks, 256, 0, c->stream>>>(t, N, tb.S, d.cls, d.slots, d.tileFlag,
                                                    d.stripFlag, d.tileCovered, dCls + n, dRow,
                                                    d.tiles, d.strips, d.tileRest);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (dCls) cudaFree(dCls);
    return e;
}

size_t tileInts(int N) { return (size_t)(N / 8 + 1) * kTileInts; }
size_t stripInts(int N) { return (size_t)(N / 4 + 1) * kStripInts; }

template <typename T, int VPL>
static void launchTilesT(alebgk_ctx *c, const void *f, void *g, cudaStream_t st)
{
    const StepParams &p = c->sp;
    const DeviceBuffers &d = c->d;
    // as many blocks as there could be tiles and strips: the plan's counts
    // stay on the device, and a refresh of the geometry changes no launch
    const unsigned chunks = (p.V + 32 * VPL - 1) / (32 * VPL);
    k_transport_tiles<T, VPL><<<yzGrid(chunks, (p.N / 8 + 8) / 8), 256, 0, st>>>(
        static_cast<const T *>(f), static_cast<T *>(g), static_cast<const T *>(d.coef), d.tiles,
        d.tileCount, p.S, p.V, p.ldf, d.sc);
    k_transport_strips<T, VPL><<<yzGrid(chunks, (p.N / 4 + 8) / 8), 256, 0, st>>>(
        static_cast<const T *>(f), static_cast<T *>(g), static_cast<const T *>(d.coef), d.strips,
        d.tileCount + 1, p.S, p.V, p.ldf, d.sc);
}

cudaError_t launchTiles(alebgk_ctx *c, const void *f, void *g, cudaStream_t st)
{
    if (c->cfg.precision == 64) launchTilesT<double, 1>(c, f, g, st);
    else if (c->sp.V % 2 == 0) launchTilesT<float, 2>(c, f, g, st);
    else launchTilesT<float, 1>(c, f, g, st);
    return cudaGetLastError();
}

}  // namespace alebgk
