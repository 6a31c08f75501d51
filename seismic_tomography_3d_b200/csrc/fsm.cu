// Noble-Gesret-Belayouni fast sweeping on the device, bit-exact with the reference's
// Accurate_FSM (src/eikonal/accurate_FSM/accurate_FSM.cpp:159-650).
//
// The reference runs 8 source-anchored sweeps and 8 full sweeps, each a Gauss-Seidel pass
// in one octant order (k outer, j, i inner).  The local operator reads only the node itself
// and its upwind neighbours in that octant, which all lie on earlier diagonal planes
// (constant (i-i0)di + (j-j0)dj + (k-k0)dk), so updating one diagonal plane at a time, all
// nodes of a plane in parallel, performs exactly the same operations on exactly the same
// values as the sequential loop.  With FP32 arithmetic in the reference's order (this file
// is compiled with -fmad=false; division and square root are IEEE) the result is the
// reference's, bit for bit.  All shots of a batch sweep together in one cooperative launch;
// blocks form `ngroups` independent groups (shots g, g+ngroups, ...), each with its own
// bounded barrier between planes.  The default schedule (k_fsm_tiled, below) orders the
// same updates tile by tile instead of plane by plane.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "fsm.cuh"

namespace tomo {

namespace {

// octant signs (z, x, y) of the 8 sweeps, in the reference's order
__device__ __constant__ int kSgn[8][3] = {{1, 1, 1},  {-1, 1, 1},  {1, 1, -1},  {-1, 1, -1},
                                          {1, -1, 1}, {-1, -1, 1}, {1, -1, -1}, {-1, -1, -1}};

__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }  // std::min
__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }  // std::max

// Group barrier over the blocks of one group (bounded spin; false on any error).  Every
// thread of a block gets thread 0's reading of the error word, so a block never splits over
// an error raised by another block while it passes the barrier.
__device__ __forceinline__ bool group_barrier(unsigned *bar, unsigned nblocks, unsigned *err,
                                              unsigned long long spin_limit)
{
    __shared__ unsigned err_seen;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned gen = ld_volatile(bar + 1);
        __threadfence();
        const unsigned arrived = atomicAdd(bar, 1u);
        if (arrived == nblocks - 1) {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            unsigned long long spins = 0;
            while (ld_volatile(bar + 1) == gen) {
                if (++spins > spin_limit || ld_volatile(err) != 0u) {
                    atomicCAS(err, 0u, (unsigned)kDevBarrierTimeout);
                    break;
                }
                __nanosleep(32);
            }
        }
        __threadfence();
        err_seen = ld_volatile(err);
    }
    __syncthreads();
    return err_seen == 0u;
}

struct ShotGrid {
    const FsmShot *s;
    float *T;
    long long n;
    int nxx, nyy, nzz;
};

// Flattened read like the reference: past a column edge lands in the next column; past the
// end of the shot's grid (undefined in the reference) reads 1e6.
__device__ __forceinline__ float tget(const ShotGrid &g, long long idx)
{
    return (idx >= 0 && idx < g.n) ? __ldcg(g.T + idx) : 1e6f;
}

// Slowness of halo-grid node (i, j, k): the window cropped and replicated by one node.
__device__ __forceinline__ const float *sptr(const FsmLaunch &p, const ShotGrid &g, int i, int j, int k)
{
    const int z = min(max(i - 1, 0), p.nz - 1);
    const int x = g.s->wx0 + min(max(j - 1, 0), g.s->wnx - 1);
    const int y = g.s->wy0 + min(max(k - 1, 0), g.s->wny - 1);
    return p.slow + z + (long long)x * p.nz + (long long)y * p.nx * p.nz;
}

__device__ __forceinline__ float sget(const FsmLaunch &p, const ShotGrid &g, int i, int j, int k)
{
    return __ldg(sptr(p, g, i, j, k));
}

// Traveltimes and slowness of one shot's halo grid as the sweep reads them, from global
// memory with the reference's flattened indexing (the plane schedule).
struct GlobalAcc {
    const FsmLaunch &p;
    const ShotGrid &g;
    __device__ __forceinline__ float t(int i, int j, int k) const
    {
        return tget(g, i + j * (long long)g.nzz + k * ((long long)g.nxx * g.nzz));
    }
    __device__ __forceinline__ float self(int i, int j, int k) const
    {
        return __ldcg(g.T + i + j * (long long)g.nzz + k * ((long long)g.nxx * g.nzz));
    }
    __device__ __forceinline__ float s(int i, int j, int k) const { return sget(p, g, i, j, k); }
};

// Inputs of one node update: the node's own value, its upwind traveltimes, and the
// slowness minima the operator uses -- m1..m3 (the 1D candidates), r1..r3 (the 2D
// candidates) and r0 (the 3D candidate).
struct NgbIn {
    float self, tv, te, tn, tev, ten, tnv, tnve;
    float m1, m2, m3, r1, r2, r3, r0;
};

// Accurate_FSM::inner_sweep (accurate_FSM.cpp:159-265) from the minima on: the same
// operations in the same order (this file is compiled with -fmad=false).
__device__ __forceinline__ float ngb_core(const FsmLaunch &p, const NgbIn &v)
{
    const float tv = v.tv, te = v.te, tn = v.tn, tev = v.tev, ten = v.ten, tnv = v.tnv, tnve = v.tnve;
    const float dz2i = p.dz2i, dx2i = p.dx2i, dy2i = p.dy2i;
    const float t1D1 = tv + p.dz * v.m1;
    const float t1D2 = te + p.dx * v.m2;
    const float t1D3 = tn + p.dy * v.m3;
    const float t1D = smin(t1D1, smin(t1D2, t1D3));

    float t2D1 = 1e6f, t2D2 = 1e6f, t2D3 = 1e6f, ta, tb, tc, Sref;
    Sref = v.r1;
    if ((tv < te + p.dx * Sref) && (te < tv + p.dz * Sref)) {
        ta = tev + te - tv;
        tb = tev - te + tv;
        t2D1 = ((tb * dz2i + ta * dx2i) + sqrtf(4.0f * Sref * Sref * (dz2i + dx2i) - dz2i * dx2i * (ta - tb) * (ta - tb))) /
               (dz2i + dx2i);
    }
    Sref = v.r2;
    if ((tv < tn + p.dy * Sref) && (tn < tv + p.dz * Sref)) {
        ta = tv - tn + tnv;
        tb = tn - tv + tnv;
        t2D2 = ((ta * dz2i + tb * dy2i) + sqrtf(4.0f * Sref * Sref * (dz2i + dy2i) - dz2i * dy2i * (ta - tb) * (ta - tb))) /
               (dz2i + dy2i);
    }
    Sref = v.r3;
    if ((te < tn + p.dy * Sref) && (tn < te + p.dx * Sref)) {
        ta = te - tn + ten;
        tb = tn - te + ten;
        t2D3 = ((ta * dx2i + tb * dy2i) + sqrtf(4.0f * Sref * Sref * (dx2i + dy2i) - dx2i * dy2i * (ta - tb) * (ta - tb))) /
               (dx2i + dy2i);
    }
    const float t2D = smin(t2D1, smin(t2D2, t2D3));

    float t3D = 1e6f;
    Sref = v.r0;
    ta = te - 0.5f * tn + 0.5f * ten - 0.5f * tv + 0.5f * tev - tnv + tnve;
    tb = tv - 0.5f * tn + 0.5f * tnv - 0.5f * te + 0.5f * tev - ten + tnve;
    tc = tn - 0.5f * te + 0.5f * ten - 0.5f * tv + 0.5f * tnv - tev + tnve;
    if (smin(t1D, t2D) > smax(tv, smax(te, tn))) {
        const float t2 = 9.0f * Sref * Sref * p.dsum;
        const float t3 = p.dz2dx2 * (ta - tb) * (ta - tb) + p.dz2dy2 * (tb - tc) * (tb - tc) + p.dx2dy2 * (ta - tc) * (ta - tc);
        if (t2 >= t3) {
            const float t1 = tb * dz2i + ta * dx2i + tc * dy2i;
            t3D = (t1 + sqrtf(t2 - t3)) / p.dsum;
        }
    }
    return smin(v.self, smin(t1D, smin(t2D, t3D)));
}

// The update with the reference's own neighbour indices and minima, read through the
// accessor with the reference's flattened indexing (the plane schedule).
template <class Acc>
__device__ __forceinline__ float ngb_update(const FsmLaunch &p, const Acc &A, int nxx, int nyy, int nzz, int i, int j,
                                            int k, int sgntz, int sgntx, int sgnty)
{
    const int sgnvz = sgntz == 1, sgnvx = sgntx == 1, sgnvy = sgnty == 1;
    const int i1 = i - sgnvz, j1 = j - sgnvx, k1 = k - sgnvy;
    const int jm = max(j - 1, 1), jp = min(j, nxx - 1), km = max(k - 1, 1), kp = min(k, nyy - 1);
    const int im = max(i - 1, 1), ip = min(i, nzz - 1);
    NgbIn v;
    v.self = A.self(i, j, k);
    v.tv = A.t(i - sgntz, j, k);
    v.te = A.t(i, j - sgntx, k);
    v.tn = A.t(i, j, k - sgnty);
    v.tev = A.t(i - sgntz, j - sgntx, k);
    v.ten = A.t(i, j - sgntx, k - sgnty);
    v.tnv = A.t(i - sgntz, j, k - sgnty);
    v.tnve = A.t(i - sgntz, j - sgntx, k - sgnty);
    v.m1 = smin(A.s(i1, jm, km), smin(A.s(i1, jm, kp), smin(A.s(i1, jp, km), A.s(i1, jp, kp))));
    v.m2 = smin(A.s(im, j1, km), smin(A.s(ip, j1, km), smin(A.s(im, j1, kp), A.s(ip, j1, kp))));
    v.m3 = smin(A.s(im, jm, k1), smin(A.s(im, jp, k1), smin(A.s(ip, jm, k1), A.s(ip, jp, k1))));
    v.r1 = smin(A.s(i1, j1, km), A.s(i1, j1, kp));
    v.r2 = smin(A.s(i1, jm, k1), A.s(i1, jp, k1));
    v.r3 = smin(A.s(im, j1, k1), A.s(ip, j1, k1));
    v.r0 = A.s(i1, j1, k1);
    return ngb_core(p, v);
}

}  // namespace

__global__ void __launch_bounds__(256, 3) k_fsm_sweeps(FsmLaunch p)
{
    const int G = p.ngroups;
    const int grp = blockIdx.x % G;
    const unsigned gblocks = (gridDim.x - grp + G - 1) / G;
    const int gb = blockIdx.x / G;
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const long long gwarp = (long long)gb * wpb + (threadIdx.x >> 5);
    const long long nwarps = (long long)gblocks * wpb;
    const long long gthread = (long long)gb * blockDim.x + threadIdx.x;
    const long long nthreads = (long long)gblocks * blockDim.x;
    unsigned *bar = p.bar + 2 * grp;
    const int nzz = p.nz + 2;
    const int ns = (p.nshots - grp + G - 1) / G;  // shots of this group: grp + m*G

    // T = 1e6 on the shots' halo grids, then the 27 analytic seeds (accurate_FSM.cpp:591-630)
    for (int m = 0; m < ns; m++) {
        const FsmShot &s = p.shots[grp + m * G];
        const long long n = (long long)nzz * (s.wnx + 2) * (s.wny + 2);
        for (long long q = gthread; q < n; q += nthreads) __stcg(p.T + s.t_off + q, 1e6f);
    }
    if (!group_barrier(bar, gblocks, p.err, p.spin_limit)) return;
    for (long long q = gthread; q < (long long)ns * 27; q += nthreads) {
        const FsmShot &s = p.shots[grp + (int)(q / 27) * G];
        const int e = (int)(q % 27), oz = e % 3 - 1, ox = (e / 3) % 3 - 1, oy = e / 9 - 1;
        const int nxx = s.wnx + 2;
        const long long sid = s.sidz + (long long)s.sidx * nzz + (long long)s.sidy * nxx * nzz;
        ShotGrid g{&s, p.T + s.t_off, 0, nxx, s.wny + 2, nzz};
        const float S0 = sget(p, g, s.sidz, s.sidx, s.sidy);
        __stcg(p.T + s.t_off + sid + oz + (long long)ox * nzz + (long long)oy * nxx * nzz, S0 * s.seed_dist[e]);
    }
    if (!group_barrier(bar, gblocks, p.err, p.spin_limit)) return;

    for (int q = 0; q < 16; q++) {
        const int sgz = kSgn[q & 7][0], sgx = kSgn[q & 7][1], sgy = kSgn[q & 7][2];
        int W = 0;
        for (int m = 0; m < ns; m++) {
            const FsmShot &s = p.shots[grp + m * G];
            const FsmRange rz = fsm_sweep_range(q, sgz, nzz, s.sidz), rx = fsm_sweep_range(q, sgx, s.wnx + 2, s.sidx),
                           ry = fsm_sweep_range(q, sgy, s.wny + 2, s.sidy);
            W = max(W, rz.L + rx.L + ry.L - 2);
        }
        for (int w = 0; w < W; w++) {
            // one warp per (shot, c) row of the plane; lanes stride over a
            for (long long row = gwarp; row < (long long)ns * nzz; row += nwarps) {
                const int m = (int)(row / nzz), c = (int)(row % nzz);
                const FsmShot &s = p.shots[grp + m * G];
                const FsmRange rz = fsm_sweep_range(q, sgz, nzz, s.sidz), rx = fsm_sweep_range(q, sgx, s.wnx + 2, s.sidx),
                               ry = fsm_sweep_range(q, sgy, s.wny + 2, s.sidy);
                if (c >= rz.L) continue;
                const int t = w - c;
                const int a_lo = max(0, t - (ry.L - 1)), a_hi = min(rx.L - 1, t);
                if (a_lo > a_hi) continue;
                ShotGrid g{&s, p.T + s.t_off, (long long)nzz * (s.wnx + 2) * (s.wny + 2), s.wnx + 2, s.wny + 2, nzz};
                const int i = rz.i0 + rz.di * c;
                for (int a = a_lo + lane; a <= a_hi; a += 32) {
                    const int j = rx.i0 + rx.di * a, k = ry.i0 + ry.di * (t - a);
                    const float v = ngb_update(p, GlobalAcc{p, g}, g.nxx, g.nyy, g.nzz, i, j, k, sgz, sgx, sgy);
                    __stcg(g.T + i + (long long)j * nzz + (long long)k * g.nxx * nzz, v);
                }
            }
            if (!group_barrier(bar, gblocks, p.err, p.spin_limit)) return;
        }
    }

    // reduce_model (accurate_FSM.cpp:62-72) into the brick-major pool of the shot
    for (int m = 0; m < ns; m++) {
        const int sidx = grp + m * G;
        const FsmShot &s = p.shots[sidx];
        const ShotDesc &d = p.desc[sidx];
        const long long n = (long long)d.nbx * d.nby * d.nbz * kBrickNodes;
        const int nxx = s.wnx + 2;
        for (long long e = gthread; e < n; e += nthreads) {
            const long long b = e / kBrickNodes;
            const int node = (int)(e % kBrickNodes);
            const int bz = (int)(b % d.nbz);
            const long long tq = b / d.nbz;
            const int bx = (int)(tq % d.nbx), by = (int)(tq / d.nbx);
            const int z = bz * 4 + (node & 3), x = bx * 4 + ((node >> 2) & 3), y = by * 4 + (node >> 4);
            float v = kInf;
            if (z < p.nz && x < s.wnx && y < s.wny)
                v = __ldcg(p.T + s.t_off + (z + 1) + (long long)(x + 1) * nzz + (long long)(y + 1) * nxx * nzz);
            p.Tb[d.t_off + e] = v;
        }
    }
}

cudaError_t fsm_solve(const FsmLaunch &p, int *grid_out, cudaStream_t st)
{
    int dev = 0, nsm = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fsm_sweeps, 256, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int grid = nsm * per_sm;
    if (p.ngroups < 1 || p.ngroups > grid) return cudaErrorInvalidValue;
    if (grid_out) *grid_out = grid;
    FsmLaunch pp = p;
    void *args[] = {&pp};
    return cudaLaunchCooperativeKernel((const void *)k_fsm_sweeps, dim3(grid), dim3(256), args, 0, st);
}

// -------------------------------------------------------------------------------------
// Tiled schedule.  One sweep is a Gauss-Seidel pass whose node updates depend only on the
// upwind neighbours of the sweep's octant.  The sweep's node box (sweep order z, x, y) is
// cut into kFsmTZ x kFsmTX x kFsmTY tiles; a tile depends only on the (up to 7) tiles
// below it on some axes, so tiles are handed out in the order of their tile diagonal
// tc + ta + tb.  One warp, or a group of eight, relaxes one tile in shared memory, diagonal plane by
// diagonal plane (the nodes of a plane are independent), after waiting for its upwind tiles'
// flags; every tile it waits on was handed out before its own and every CTA is resident, so
// the waits end.  Each node sees exactly the values it sees in the sequential loop, and the
// update performs the same operations, so the result is the plane schedule's bit for bit --
// with no grid barrier between sweeps of a batch: a shot's tile of sweep q + 1 also waits
// until all of that shot's sweep-q tiles are finished (a per-shot count), since those read its
// nodes in sweep q's order; shots are independent, so one shot's next sweep overlaps another's
// drain.  The sweep-q tiles were all handed out before any sweep-(q + 1) tile, so this
// wait ends too.  Few tiles keep a grid barrier between sweeps (sweep_barrier).
// Every source must lie off
// the far faces of its window (halo index sid <= n - 3), so that no read leaves the grid
// (the reference's flattened reads would otherwise cross a column edge).
//
// What bounds a tile is its chain of 30 planes: an update is a chain of some hundred dependent
// FP32 operations, and one warp runs it 46 times in a row (planes of up to 64 nodes), with 16
// warps an SM, as many tiles as shared memory holds.  k_fsm_tiled<8, ...> splits the update over
// four warps: warps 0 to 2 each form one 1D and one 2D candidate
// of every node of the plane -- the pairs that read the same slowness cells -- and warp 3 the
// 3D one; after a barrier two of them take the minimum the reference takes, and store.  The
// chain shortens to one candidate and four times the warps share the same shared memory.
// Two such sets of four warps keep one half of a plane's nodes each, so that no warp passes a
// plane twice.  One shot of 101 x 101 x 51: 11.4 -> 4.8 ms.  That is for few shots, which wait on
// the wavefront; in a batch one warp a tile issues fewer instructions, and there the shorter
// arithmetic (lesser, by_sum, root) and the mirrored tile, whose plane loop has one form and no
// index arithmetic for all eight octants, count: 64 shots of 201 x 201 x 101, windows of 60-100 %,
// 48.6 -> 46.2 ms with the short division and no branches, 40.5 with the short root and the
// mirrored tile, 38.5 with the one-instruction minimum (36.9 for the whole call in a later run, and
// 37.7 with std::min's order kept for NaN candidates, std_min).
// -------------------------------------------------------------------------------------
namespace {

constexpr int kHZ = kFsmTZ + 1, kHX = kFsmTX + 1, kHY = kFsmTY + 1;  // a tile + one layer per axis
// Strides of the staged arrays (z, then x; words): padded from 17 x 9 so that the lanes of a
// diagonal-plane pass, which differ by (+-19 -+ 1) a + (+-190 -+ 1) b words, fall in
// distinct banks (a search over the plane order and the 8 sweep signs: 548 shared-memory
// wavefronts per tile instead of 1,280).
constexpr int kPZ = 19, kPX = 10;
constexpr int kHN = kPZ * kPX * kHY;
constexpr int kTileN = kFsmTZ * kFsmTX * kFsmTY;
constexpr int kNPlanes = kFsmTZ + kFsmTX + kFsmTY - 2;
constexpr int kMaxPlane = kFsmTX * kFsmTY;  // nodes of the largest diagonal plane
constexpr int kCands = 7;                   // 1D x 3, 2D x 3, 3D
static_assert(kFsmTZ <= 32 && kFsmTX <= 8 && kFsmTY <= 8, "plane table packs a word and (c, a, b) in 16 + 5 + 3 + 3 bits");
static_assert(kPZ >= kHZ && kPX >= kHX, "padded strides");
static_assert(kFsmTZ >= kFsmTX && kFsmTZ >= kFsmTY && kMaxPlane <= 64, "a plane is at most two warps of nodes");

// Arithmetic of the operator.  kFast: the short division and square root of common.cuh, the
// same IEEE results in 3 and 6 instructions, and the hardware's minimum, one instruction where
// std::min's order of comparison takes two.  The minimum differs for NaN only.  A 2D candidate
// is NaN where its discriminant is negative although its test holds (a diagonal neighbour that
// no sweep has reached yet, at 1e6), and what std::min then drops is kept track of (std_min).
// An infinite slowness or seed would make candidates infinite, which the short forms turn into
// NaN, and a very small slowness takes the root's argument out of its range (fsm_solve_tiled);
// those and NaN itself are flagged before the sweeps (FsmLaunch::plain), and the model takes the
// plain forms, as it does where the spacings do not suit the divisors.
template <bool kFast>
__device__ __forceinline__ float by_sum(float a, const Divisor &d)
{
    return kFast ? fdiv(a, d) : a / d.y;
}

template <bool kFast>
__device__ __forceinline__ float root(float a)
{
    return kFast ? fsqrt(a) : sqrtf(a);
}

template <bool kFast>
__device__ __forceinline__ float lesser(float a, float b)
{
    return kFast ? fminf(a, b) : smin(a, b);
}

// std::min(a, b) of candidates that may be NaN: NaN if a is, a if b is.
template <bool kFast>
__device__ __forceinline__ float std_min(float a, float b)
{
    if (!kFast) return smin(a, b);
    float m;  // two instructions; fminf drops b's NaN
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(fminf(b, __int_as_float(0x7f800000))));
    return m;
}

// The candidates of Accurate_FSM::inner_sweep (accurate_FSM.cpp:159-265) for the node at T, in
// the reference's operation order (this file is compiled with -fmad=false).  The tile lies in
// shared memory in the sweep's own direction on every axis (staging mirrors the axes it runs
// down), so the upwind neighbours are the ones before the node whatever the octant.  The
// slowness at halo indices -1, 0 and 1 of an axis is one value (the window is replicated), and
// the operator's max(i - 1, 1) and min(i, n - 1) read the values at i - 1 and i: every minimum
// comes from the node's 2 x 2 x 2 cell cube (halo indices i-1..i, j-1..j, k-1..k), mirrored
// with the tile, so that its cell 0 on an axis is the upwind one (the reference's i1, j1, k1).
// A minimum of slownesses is exact and independent of its order, so each has the reference's value;
// with NaN it is not, and the plain form (not kFast) takes the cells in the reference's order,
// lower index first on each axis (flip: bit 0 z, 1 x, 2 y, set where the tile is mirrored).
constexpr int kDZ = 1, kDX = kPZ, kDY = kPZ * kPX;  // one step along each axis

// Minimum over the 2 x 2 cells spanned by steps u and v from c, u outermost; over the two along u.
template <bool kFast>
__device__ __forceinline__ float cell_minimum(const float *c, int u, int v, bool flip_u, bool flip_v)
{
    if (kFast) return fminf(fminf(c[0], c[u]), fminf(c[v], c[u + v]));
    const int u0 = flip_u ? u : 0, u1 = u - u0, v0 = flip_v ? v : 0, v1 = v - v0;
    return smin(c[u0 + v0], smin(c[u0 + v1], smin(c[u1 + v0], c[u1 + v1])));
}

template <bool kFast>
__device__ __forceinline__ float pair_minimum(const float *c, int u, bool flip)
{
    return kFast ? fminf(c[0], c[u]) : (flip ? smin(c[u], c[0]) : smin(c[0], c[u]));
}

template <bool kFast>
__device__ __forceinline__ float candidate_2d(float a, float b, float da, float db, float S, float num, float diff,
                                              float wsum, float wprod, const Divisor &by)
{
    const float cand = by_sum<kFast>(num + root<kFast>(4.0f * S * S * wsum - wprod * diff * diff), by);
    return ((a < b + db * S) && (b < a + da * S)) ? cand : 1e6f;
}

// Candidates of warp C: C = 0 z with (z, x), 1 y with (z, y), 2 x with (x, y), 3 the 3D one.
// Every candidate is computed and kept only where the reference's test holds.  Skipping those no lane needs by a branch was
// faster with the plain divisions and roots (48.6 vs 52.3 ms per 64-shot batch); with the short
// division it costs more than it saves (48.5 vs 46.2 ms).
template <int C, bool kFast>
__device__ __forceinline__ void candidates(const FsmLaunch &p, const float *T, const float *c, int flip, float &one,
                                           float &more)
{
    const bool fz = flip & 1, fx = flip & 2, fy = flip & 4;
    if (C == 0) {
        const float tv = T[-kDZ], te = T[-kDX], tev = T[-kDZ - kDX];
        const float r = pair_minimum<kFast>(c, kDY, fy);
        one = tv + p.dz * cell_minimum<kFast>(c, kDX, kDY, fx, fy);
        const float ta = tev + te - tv, tb = tev - te + tv;
        more = candidate_2d<kFast>(tv, te, p.dz, p.dx, r, tb * p.dz2i + ta * p.dx2i, ta - tb, p.by_zx.y, p.dz2dx2,
                                       p.by_zx);
    } else if (C == 1) {
        const float tv = T[-kDZ], tn = T[-kDY], tnv = T[-kDZ - kDY];
        const float r = pair_minimum<kFast>(c, kDX, fx);
        one = tn + p.dy * cell_minimum<kFast>(c, kDZ, kDX, fz, fx);
        const float ta = tv - tn + tnv, tb = tn - tv + tnv;
        more = candidate_2d<kFast>(tv, tn, p.dz, p.dy, r, ta * p.dz2i + tb * p.dy2i, ta - tb, p.by_zy.y, p.dz2dy2,
                                       p.by_zy);
    } else if (C == 2) {
        const float te = T[-kDX], tn = T[-kDY], ten = T[-kDX - kDY];
        const float r = pair_minimum<kFast>(c, kDZ, fz);
        one = te + p.dx * cell_minimum<kFast>(c, kDY, kDZ, fy, fz);
        const float ta = te - tn + ten, tb = tn - te + ten;
        more = candidate_2d<kFast>(te, tn, p.dx, p.dy, r, ta * p.dx2i + tb * p.dy2i, ta - tb, p.by_xy.y, p.dx2dy2,
                                       p.by_xy);
    } else {
        const float tv = T[-kDZ], te = T[-kDX], tn = T[-kDY], tev = T[-kDZ - kDX], ten = T[-kDX - kDY],
                    tnv = T[-kDZ - kDY], tnve = T[-kDZ - kDX - kDY];
        const float S = c[0];
        const float ta = te - 0.5f * tn + 0.5f * ten - 0.5f * tv + 0.5f * tev - tnv + tnve;
        const float tb = tv - 0.5f * tn + 0.5f * tnv - 0.5f * te + 0.5f * tev - ten + tnve;
        const float tc = tn - 0.5f * te + 0.5f * ten - 0.5f * tv + 0.5f * tnv - tev + tnve;
        const float t2 = 9.0f * S * S * p.dsum;
        const float t3 =
            p.dz2dx2 * (ta - tb) * (ta - tb) + p.dz2dy2 * (tb - tc) * (tb - tc) + p.dx2dy2 * (ta - tc) * (ta - tc);
        const float t1 = tb * p.dz2i + ta * p.dx2i + tc * p.dy2i;
        const float cand = by_sum<kFast>(t1 + root<kFast>(t2 - t3), p.by_sum);
        one = 0.0f;
        more = t2 >= t3 ? cand : 1e6f;
    }
}

// Asynchronous 4-byte copy global -> shared (cp.async, through L1).  Only for the slowness,
// which nothing writes while a solve runs, so an L1 line can never be stale; the
// traveltimes, written by other SMs between tiles, are read through L2 (__ldcg).
__device__ __forceinline__ void cp_async4(float *dst, const float *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// Waits for this thread's cp.async copies; a barrier after it shows them to the others.
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Barrier of the kWarps warps of group g of the CTA (barrier 0 is __syncthreads).
template <int kWarps>
__device__ __forceinline__ void group_sync(int g)
{
    __syncwarp();
    if (kWarps > 1) asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(32 * kWarps) : "memory");
}

// A tile in shared memory.  Node (c, a, b) of the tile, along the sweep, is word kNode0 + c kDZ
// + a kDX + b kDY of Ts, after the upwind layer; its cell cube starts at the same word of Ss
// less kNode0.
constexpr int kNode0 = kDZ + kDX + kDY;

struct Tile {
    float *Ts;               // traveltimes
    const float *Ss;         // slowness
    float *cand;             // kCands x kMaxPlane candidates of the current plane
    const unsigned *plane;   // the tile's nodes by diagonal plane: word | c << 16 | a << 21 | b << 24
    const int *pstart;       // first entry of each plane
    int nc, na, nb;          // the sweep's nodes left on each axis from the tile's first node
    bool full;               // no node of the tile lies beyond them
    int flip;                // axes on which the tile is mirrored (candidates)
};

// Word of the m-th node in plane order; false: not a node of the sweep.
__device__ __forceinline__ bool tile_node(const Tile &t, int m, int &word)
{
    const unsigned e = t.plane[m];
    word = (int)(e & 0xffffu);
    return t.full || ((int)(e >> 16 & 31u) < t.nc && (int)(e >> 21 & 7u) < t.na && (int)(e >> 24) < t.nb);
}

// The reference's minimum of the candidates of the node at T (accurate_FSM.cpp:258-264).
template <bool kFast>
__device__ __forceinline__ float least(const float *T, float z1, float x1, float y1, float zx, float zy, float xy,
                                       float zxy)
{
    const float t1D = lesser<kFast>(z1, lesser<kFast>(x1, y1)), t2D = std_min<kFast>(zx, std_min<kFast>(zy, xy));
    const bool above = lesser<kFast>(t1D, t2D) > smax(T[-kDZ], smax(T[-kDX], T[-kDY]));
    return lesser<kFast>(T[0], lesser<kFast>(t1D, std_min<kFast>(t2D, above ? zxy : 1e6f)));
}

// One tile, diagonal plane by diagonal plane, by one warp: all candidates of a node in its lane.
template <bool kFast>
__device__ __forceinline__ void relax_alone(const FsmLaunch &p, const Tile &t, int lane)
{
    int first = 0;
    for (int w = 0; w < kNPlanes; w++) {
        const int end = t.pstart[w + 1];
        for (int m = first + lane; m < end; m += 32) {
            int word;
            if (tile_node(t, m, word)) {
                float *T = t.Ts + word;
                const float *c = t.Ss + word - kNode0;
                float z1, x1, y1, zx, zy, xy, zxy, none;
                candidates<0, kFast>(p, T, c, t.flip, z1, zx);
                candidates<1, kFast>(p, T, c, t.flip, y1, zy);
                candidates<2, kFast>(p, T, c, t.flip, x1, xy);
                candidates<3, kFast>(p, T, c, t.flip, none, zxy);
                T[0] = least<kFast>(T, z1, x1, y1, zx, zy, xy, zxy);
            }
        }
        first = end;
        __syncwarp();
    }
}

// The same by eight warps: warp C of half `half` forms candidates C of its nodes, 32 of a plane.
template <int C, bool kFast>
__device__ __forceinline__ void relax_warp(const FsmLaunch &p, const Tile &t, int lane, int half, int group)
{
    const int k = 32 * half + lane, kc = 32 * C + lane;
    int first = 0;
    for (int w = 0; w < kNPlanes; w++) {
        const int end = t.pstart[w + 1], n = end - first;
        int word;
        if (k < n && tile_node(t, first + k, word)) {
            float one, more;
            candidates<C, kFast>(p, t.Ts + word, t.Ss + word - kNode0, t.flip, one, more);
            if (C < 3) t.cand[C * kMaxPlane + k] = one;
            t.cand[(3 + C) * kMaxPlane + k] = more;
        }
        group_sync<8>(group);
        // the minimum: warps 0 and 1 of the first half, 32 nodes each
        if (C < 2 && half == 0 && kc < n && tile_node(t, first + kc, word)) {
            const float *c = t.cand + kc;
            float *T = t.Ts + word;
            T[0] = least<kFast>(T, c[0], c[2 * kMaxPlane], c[kMaxPlane], c[3 * kMaxPlane], c[4 * kMaxPlane], c[5 * kMaxPlane],
                         c[6 * kMaxPlane]);
        }
        first = end;
        group_sync<8>(group);
    }
}

template <int kWarps, bool kFast>
__device__ __forceinline__ void relax_tile(const FsmLaunch &p, const Tile &t, int lane, int warp, int group)
{
    if (kWarps == 1) {
        relax_alone<kFast>(p, t, lane);
        return;
    }
    const int half = warp >> 2;
    switch (warp & 3) {
    case 0: relax_warp<0, kFast>(p, t, lane, half, group); break;
    case 1: relax_warp<1, kFast>(p, t, lane, half, group); break;
    case 2: relax_warp<2, kFast>(p, t, lane, half, group); break;
    default: relax_warp<3, kFast>(p, t, lane, half, group); break;
    }
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(unsigned *p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ int cdiv(int a, int b) { return (a + b - 1) / b; }

// Lowest halo index of the tile's own nodes on one axis (l0: the tile's first local index).
__device__ __forceinline__ int tile_lo(const FsmRange &r, int l0, int T)
{
    return r.di > 0 ? r.i0 + l0 : r.i0 - (l0 + T - 1);
}

// A work item as the group's first warp leaves it to the others; shot < 0: the sweep is over.
struct TileItem {
    int shot, tc, ta, tb;
};

// The group's next tile of sweep q (one warp).
__device__ __forceinline__ TileItem next_tile(const FsmLaunch &p, int q, int lane)
{
    const int sgz = fsm_sign_z(q), sgx = fsm_sign_x(q), sgy = fsm_sign_y(q);
    const int nzz = p.nz + 2;
    const int *tab = p.tab + p.tab_base[q];
    const int S = p.nshots, nd = p.tab_nd[q];
    const int total = tab[nd * S];
    TileItem it{-1, 0, 0, 0};
    int item = 0;
    if (lane == 0) item = ld_volatile(p.err) != 0u ? total : (int)atomicAdd(p.cursors + q, 1u);
    item = __shfl_sync(kFull, item, 0);
    if (item >= total) return it;
    // (diagonal, shot): the last table entry <= item (tab[lo] <= item < tab[hi]).  A
    // warp-wide search (32 probes per step, 2-3 dependent loads instead of 12) measured
    // 3 % slower on the config-2 batch: these loads are broadcasts that hit L1.
    int lo = 0, hi = nd * S;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(tab + mid) <= item)
            lo = mid;
        else
            hi = mid;
    }
    const int d = lo / S, si = lo % S;
    int r = item - __ldg(tab + lo);
    const FsmShot &sh = p.shots[si];
    const int nxx = sh.wnx + 2, nyy = sh.wny + 2;
    const FsmRange rz = fsm_sweep_range(q, sgz, nzz, sh.sidz), rx = fsm_sweep_range(q, sgx, nxx, sh.sidx),
                   ry = fsm_sweep_range(q, sgy, nyy, sh.sidy);
    const int A = cdiv(rz.L, kFsmTZ), B = cdiv(rx.L, kFsmTX), C = cdiv(ry.L, kFsmTY);
    // the r-th tile (tc, ta, tb) of diagonal d, tb ascending, then ta
    int tc = 0, ta = 0, tb = max(0, d - (A - 1) - (B - 1));
    for (; tb <= min(C - 1, d); tb++) {
        const int e = d - tb, alo = max(0, e - (A - 1)), ahi = min(B - 1, e);
        if (r <= ahi - alo) {
            ta = alo + r;
            tc = e - ta;
            break;
        }
        r -= ahi - alo + 1;
    }
    return TileItem{si, tc, ta, tb};
}

// Waits (one warp) for the tiles that a tile of sweep q depends on: the upwind tiles of this
// sweep (lanes 0-6: one each) and, lane 7, the end of the shot's previous sweep, whose tiles
// read this tile's nodes in their own order (a per-shot count of finished tiles instead of a
// grid barrier, so that shots that finish a sweep early start the next one while others drain
// theirs).  False: a wait ran out, here or elsewhere.
__device__ __forceinline__ bool wait_upwind(const FsmLaunch &p, int q, int lane, const TileItem &it)
{
    const int tc = it.tc, ta = it.ta, tb = it.tb, si = it.shot;
    const FsmShot &sh = p.shots[si];
    const int nzz = p.nz + 2, nxx = sh.wnx + 2;
    const int fa = cdiv(nzz - 1, kFsmTZ), fb = cdiv(nxx - 1, kFsmTX);
    const unsigned *flags = p.flags + sh.flag_off;
    bool gave_up = false;
    if (lane == 7 && q > 0 && !p.sweep_barrier) {
        const unsigned need = __ldg(p.shot_tiles + (size_t)si * 16 + (q - 1));
        const unsigned *cnt = p.shot_done + (size_t)si * 16 + (q - 1);
        unsigned long long spins = 0;
        while (ld_acquire(cnt) < need) {
            if (++spins > p.spin_limit || ld_volatile(p.err) != 0u) {
                atomicCAS(p.err, 0u, (unsigned)kDevBarrierTimeout);
                gave_up = true;
                break;
            }
            __nanosleep(32);
        }
    }
    if (lane < 7) {
        const int dc = (lane + 1) & 1, da = ((lane + 1) >> 1) & 1, db = (lane + 1) >> 2;
        if (tc >= dc && ta >= da && tb >= db) {
            const unsigned *f = flags + (tc - dc) + fa * ((ta - da) + fb * (tb - db));
            unsigned long long spins = 0;
            while (ld_acquire(f) != (unsigned)(q + 1)) {
                if (++spins > p.spin_limit || ld_volatile(p.err) != 0u) {
                    atomicCAS(p.err, 0u, (unsigned)kDevBarrierTimeout);
                    gave_up = true;
                    break;
                }
                __nanosleep(32);
            }
        }
    }
    return !__any_sync(kFull, gave_up);
}

}  // namespace

// CTA of one tile group of kWarps warps and its neighbours: 8 groups of one warp, or 2 of 8.
constexpr int fsm_threads(int warps) { return warps == 1 ? 256 : 512; }
// Words of shared memory per group.
constexpr int fsm_words(int warps) { return 2 * kHN + (warps == 1 ? 0 : kCands * kMaxPlane); }

template <int kWarps, bool kFast>
__global__ void __launch_bounds__(fsm_threads(kWarps), kWarps == 1 ? 2 : 1) k_fsm_tiled(FsmLaunch p)
{
    constexpr int kGroup = 32 * kWarps, kGroups = fsm_threads(kWarps) / kGroup;
    // unroll depth of the staging loop: a warp alone has 43 nodes a lane to bring in (4 -> 52.1,
    // 5 -> 49.3, 6 -> 48.6, 7 -> 49.1 ms per 64-shot batch), a group of eight 6 a thread
    constexpr int kStageUnroll = kWarps == 1 ? 6 : 2;
    // Bring in what does not depend on the upwind tiles before waiting for them.  A single shot
    // waits at every tile (5.22 -> 4.81 ms); in a batch the flags are mostly set on arrival and
    // the second round of reads costs more than it hides (69 vs 62 ms when it was measured).
    constexpr bool kAhead = kWarps > 1;
    extern __shared__ float smem[];
    __shared__ TileItem items[kGroups];
    __shared__ bool gone[kGroups];  // kAhead: the wait for the upwind tiles gave up
    const int group = threadIdx.x / kGroup, gt = threadIdx.x % kGroup;
    const int lane = threadIdx.x & 31, warp = gt >> 5;
    float *Ts = smem + group * fsm_words(kWarps), *Ss = Ts + kHN;
    unsigned *plane = reinterpret_cast<unsigned *>(smem + kGroups * fsm_words(kWarps));
    int *pstart = reinterpret_cast<int *>(plane + kTileN);
    // the tile's nodes (c, a, b) ordered by diagonal plane c + a + b
    if (threadIdx.x < kNPlanes) {
        const int w = threadIdx.x;
        int m = 0;
        for (int v = 0; v < w; v++)
            m += (int)fsm_diag_count(v, kFsmTZ, kFsmTX, kFsmTY);
        pstart[w] = m;
        for (int b = 0; b < kFsmTY; b++)
            for (int a = 0; a < kFsmTX; a++) {
                const int c = w - a - b;
                if (c >= 0 && c < kFsmTZ)
                    plane[m++] = (unsigned)(kNode0 + c * kDZ + a * kDX + b * kDY) | c << 16 | a << 21 | b << 24;
            }
        if (w == kNPlanes - 1) pstart[kNPlanes] = m;
    }
    const long long gthread = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    const int nzz = p.nz + 2;

    // T = 1e6 on the shots' halo grids, then the 27 analytic seeds (accurate_FSM.cpp:591-630)
    for (int m = 0; m < p.nshots; m++) {
        const FsmShot &s = p.shots[m];
        const long long n = (long long)nzz * (s.wnx + 2) * (s.wny + 2);
        for (long long q = gthread; q < n; q += nthreads) __stcg(p.T + s.t_off + q, 1e6f);
    }
    if (kFast) {
        bool any = false;
        const long long n = (long long)p.nx * p.ny * p.nz;
        for (long long q = gthread; q < n; q += nthreads) {
            const float s = fabsf(__ldg(p.slow + q));
            any |= !(s == 0.0f || (s >= p.s_lo && s <= p.s_hi));
        }
        if (__any_sync(kFull, any) && lane == 0) atomicOr(p.plain, 1u);
    }
    if (!group_barrier(p.bar, gridDim.x, p.err, p.spin_limit)) return;
    for (long long q = gthread; q < (long long)p.nshots * 27; q += nthreads) {
        const FsmShot &s = p.shots[(int)(q / 27)];
        const int e = (int)(q % 27), oz = e % 3 - 1, ox = (e / 3) % 3 - 1, oy = e / 9 - 1;
        const int nxx = s.wnx + 2;
        const long long sid = s.sidz + (long long)s.sidx * nzz + (long long)s.sidy * nxx * nzz;
        ShotGrid g{&s, p.T + s.t_off, 0, nxx, s.wny + 2, nzz};
        const float S0 = sget(p, g, s.sidz, s.sidx, s.sidy);
        const float t = S0 * s.seed_dist[e];
        if (kFast && !isfinite(t)) atomicOr(p.plain, 1u);
        __stcg(p.T + s.t_off + sid + oz + (long long)ox * nzz + (long long)oy * nxx * nzz, t);
    }
    if (!group_barrier(p.bar, gridDim.x, p.err, p.spin_limit)) return;
    const bool plain = !kFast || ld_volatile(p.plain) != 0u;

    for (int q = 0; q < 16; q++) {
        const int sgz = fsm_sign_z(q), sgx = fsm_sign_x(q), sgy = fsm_sign_y(q);
        for (;;) {
            if (warp == 0) {
                TileItem it = next_tile(p, q, lane);
                if (!kAhead && it.shot >= 0 && !wait_upwind(p, q, lane, it)) it.shot = -1;
                if (lane == 0) items[group] = it;
            }
            group_sync<kWarps>(group);  // the item (and the upwind tiles' stores) for every warp
            const TileItem it = items[group];
            if (it.shot < 0) break;
            const FsmShot &sh = p.shots[it.shot];
            const int tc = it.tc, ta = it.ta, tb = it.tb, nxx = sh.wnx + 2, nyy = sh.wny + 2;
            const FsmRange rz = fsm_sweep_range(q, sgz, nzz, sh.sidz), rx = fsm_sweep_range(q, sgx, nxx, sh.sidx),
                           ry = fsm_sweep_range(q, sgy, nyy, sh.sidy);
            // stage the tile along the sweep (mirrored on the axes it runs down): traveltimes of
            // the upwind layer and the tile, halo indices from tz.. in memory; slowness of the
            // halo indices one below the tile's lowest to its highest, from gz - 1..
            const int gz = tile_lo(rz, tc * kFsmTZ, kFsmTZ), gx = tile_lo(rx, ta * kFsmTX, kFsmTX),
                      gy = tile_lo(ry, tb * kFsmTY, kFsmTY);
            const int tz = rz.di > 0 ? gz - 1 : gz, tx = rx.di > 0 ? gx - 1 : gx, ty = ry.di > 0 ? gy - 1 : gy;
            const int wz = rz.di * kDZ, wx = rx.di * kDX, wy = ry.di * kDY;  // words per step in memory
            const int w0 = (rz.di > 0 ? 0 : kHZ - 1) * kDZ + (rx.di > 0 ? 0 : kHX - 1) * kDX +
                           (ry.di > 0 ? 0 : kHY - 1) * kDY;
            float *T = p.T + sh.t_off;
            ShotGrid g{&sh, T, 0, nxx, nyy, nzz};
            // The slowness goes by cp.async, so all its copies are in flight at once and hold
            // no registers; the traveltime loop is unrolled so that its loads are in
            // flight before their shared-memory stores wait on them.  Staged node m = gt +
            // kGroup it is (ci, cj, ck), advanced by kGroup nodes per iteration without divisions.
            static_assert(kGroup / kHZ + 1 <= 2 * kHX, "at most two carries into ck per step");
            int ci = gt % kHZ, cj = (gt / kHZ) % kHX, ck = gt / (kHZ * kHX);
#pragma unroll kStageUnroll
            for (int m = gt; m < kHZ * kHX * kHY; m += kGroup) {
                const int i = tz + ci, j = tx + cj, k = ty + ck;
                const int word = w0 + wz * ci + wx * cj + wy * ck;
                cp_async4(Ss + word, sptr(p, g, gz - 1 + ci, gx - 1 + cj, gy - 1 + ck));
                if (!kAhead) Ts[word] = (i >= 0 && i < nzz && j >= 0 && j < nxx && k >= 0 && k < nyy)
                                            ? __ldcg(T + i + (long long)j * nzz + (long long)k * nxx * nzz)
                                            : 1e6f;
                ci += kGroup % kHZ;
                cj += kGroup / kHZ;
                if (ci >= kHZ) { ci -= kHZ; ++cj; }
                if (cj >= kHX) { cj -= kHX; ++ck; }
                if (kGroup / kHZ + 1 > kHX && cj >= kHX) { cj -= kHX; ++ck; }
            }
            const int i0 = rz.i0 + rz.di * tc * kFsmTZ, j0 = rx.i0 + rx.di * ta * kFsmTX,
                      k0 = ry.i0 + ry.di * tb * kFsmTY;
            const int nc = rz.L - tc * kFsmTZ, na = rx.L - ta * kFsmTX, nb = ry.L - tb * kFsmTY;
            if (kAhead) {
                // The slowness and the tile's own nodes, which no other tile of the sweep writes,
                // come in while the upwind tiles finish; then only their layer is left to read.
                auto node = [&](int c, int a, int b) {
                    return T + (i0 + rz.di * c) + (long long)(j0 + rx.di * a) * nzz + (long long)(k0 + ry.di * b) * nxx * nzz;
                };
#pragma unroll
                for (int m = gt; m < kTileN; m += kGroup) {
                    const int c = m % kFsmTZ, a = m / kFsmTZ % kFsmTX, b = m / (kFsmTZ * kFsmTX);
                    if (c < nc && a < na && b < nb) Ts[kNode0 + c * kDZ + a * kDX + b * kDY] = __ldcg(node(c, a, b));
                }
                if (warp == 0) {
                    const bool ready = wait_upwind(p, q, lane, it);
                    if (lane == 0) gone[group] = !ready;
                }
                group_sync<kWarps>(group);
                if (gone[group]) break;
                constexpr int kFaceY = kHZ * kHX, kFaceX = kHZ * kFsmTY, kFaceZ = kFsmTX * kFsmTY;
#pragma unroll
                for (int m = gt; m < kFaceY + kFaceX + kFaceZ; m += kGroup) {
                    int c, a, b;  // the layer before the tile, -1 on one axis at least
                    if (m < kFaceY) {
                        c = m % kHZ - 1, a = m / kHZ - 1, b = -1;
                    } else if (m < kFaceY + kFaceX) {
                        c = (m - kFaceY) % kHZ - 1, a = -1, b = (m - kFaceY) / kHZ;
                    } else {
                        c = -1, a = (m - kFaceY - kFaceX) % kFsmTX, b = (m - kFaceY - kFaceX) / kFsmTX;
                    }
                    const int i = i0 + rz.di * c, j = j0 + rx.di * a, k = k0 + ry.di * b;
                    Ts[kNode0 + c * kDZ + a * kDX + b * kDY] =
                        (i >= 0 && i < nzz && j >= 0 && j < nxx && k >= 0 && k < nyy) ? __ldcg(node(c, a, b)) : 1e6f;
                }
            }
            cp_async_wait_all();
            group_sync<kWarps>(group);
            Tile t;
            t.Ts = Ts;
            t.Ss = Ss;
            t.cand = Ss + kHN;
            t.plane = plane;
            t.pstart = pstart;
            t.nc = nc;
            t.na = na;
            t.nb = nb;
            t.flip = (rz.di < 0 ? 1 : 0) | (rx.di < 0 ? 2 : 0) | (ry.di < 0 ? 4 : 0);
            t.full = t.nc >= kFsmTZ && t.na >= kFsmTX && t.nb >= kFsmTY;
            if (kFast && !plain)
                relax_tile<kWarps, kFast>(p, t, lane, warp, group);
            else
                relax_tile<kWarps, false>(p, t, lane, warp, group);
            // the tile's nodes back to global memory, then its flag
            for (int m = gt; m < kTileN; m += kGroup) {
                const int c = m % kFsmTZ, a = (m / kFsmTZ) % kFsmTX, b = m / (kFsmTZ * kFsmTX);
                if (c < t.nc && a < t.na && b < t.nb)
                    __stcg(T + (i0 + rz.di * c) + (long long)(j0 + rx.di * a) * nzz +
                               (long long)(k0 + ry.di * b) * nxx * nzz,
                           Ts[kNode0 + c * kDZ + a * kDX + b * kDY]);
            }
            __threadfence();
            group_sync<kWarps>(group);
            if (gt == 0) {
                const int fa = cdiv(nzz - 1, kFsmTZ), fb = cdiv(nxx - 1, kFsmTX);
                st_release(p.flags + sh.flag_off + tc + fa * (ta + fb * tb), (unsigned)(q + 1));
                if (!p.sweep_barrier) atomicAdd(p.shot_done + (size_t)it.shot * 16 + q, 1u);
            }
        }
        group_sync<kWarps>(group);  // every warp has read "the sweep is over" before the next item
        // few tiles: little to overlap a sweep's drain with, a barrier is cheaper than the per-tile
        // counts, and the tile's own nodes are read before the wait for the upwind tiles
        if (p.sweep_barrier && q < 15 && !group_barrier(p.bar, gridDim.x, p.err, p.spin_limit)) return;
    }
    if (!group_barrier(p.bar, gridDim.x, p.err, p.spin_limit)) return;

    // reduce_model (accurate_FSM.cpp:62-72) into the brick-major pool of the shot
    for (int m = 0; m < p.nshots; m++) {
        const FsmShot &s = p.shots[m];
        const ShotDesc &d = p.desc[m];
        const long long n = (long long)d.nbx * d.nby * d.nbz * kBrickNodes;
        const int nxx = s.wnx + 2;
        for (long long e = gthread; e < n; e += nthreads) {
            const long long b = e / kBrickNodes;
            const int node = (int)(e % kBrickNodes);
            const int bz = (int)(b % d.nbz);
            const long long tq = b / d.nbz;
            const int bx = (int)(tq % d.nbx), by = (int)(tq / d.nbx);
            const int z = bz * 4 + (node & 3), x = bx * 4 + ((node >> 2) & 3), y = by * 4 + (node >> 4);
            float v = kInf;
            if (z < p.nz && x < s.wnx && y < s.wny)
                v = __ldcg(p.T + s.t_off + (z + 1) + (long long)(x + 1) * nzz + (long long)(y + 1) * nxx * nzz);
            p.Tb[d.t_off + e] = v;
        }
    }
}

cudaError_t fsm_solve_tiled(const FsmLaunch &p, int *grid_out, cudaStream_t st)
{
    // Eight warps a tile, and a grid barrier between sweeps, where the tiles of a diagonal are few
    // enough that the groups wait on the wavefront; one warp a tile, and per-shot sweep counts,
    // where there are tiles enough to keep the SMs issuing (the split's barriers and repeated
    // loads cost more instructions than its lanes save).  ms per solve, eight | one, by the tiles
    // on the widest diagonal of all shots (shots x tiles of one; 101 x 101 x 51, 201 x 201 x 101 and
    // 260 x 260 x 120 nodes): 1 x 52 4.85 | 7.9 (2 shots 5.11 | 7.93), 8 x 52 6.37 | 8.04, 16 x 52 8.77 |
    // 8.53; 4 x 182 14.8 | 17.0, 8 x 182 25.2 | 19.7; 2 x 264 15.7 | 21.5, 4 x 264 24.5 | 23.8.
    const bool split = p.widest <= 800;
    bool fast = true;
    for (const float y : {p.by_zx.y, p.by_zy.y, p.by_xy.y, p.by_sum.y})
        fast = fast && y >= kDivMin && y <= kDivMax;
    const void *fn = split ? (fast ? (const void *)k_fsm_tiled<8, true> : (const void *)k_fsm_tiled<8, false>)
                           : (fast ? (const void *)k_fsm_tiled<1, true> : (const void *)k_fsm_tiled<1, false>);
    const int threads = fsm_threads(split ? 8 : 1), groups = threads / (split ? 256 : 32);
    const size_t smem = (size_t)groups * fsm_words(split ? 8 : 1) * sizeof(float) + kTileN * sizeof(unsigned) +
                        (kNPlanes + 1) * sizeof(int);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0, per_sm = 0;
    e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int grid = nsm * per_sm;
    if (grid_out) *grid_out = grid;
    FsmLaunch pp = p;
    pp.sweep_barrier = split ? 1 : 0;
    // Slownesses whose root arguments lie in fsqrt's range: the arguments are differences of
    // 4 s^2 w (w: a sum of two inverse squared spacings) or 9 s^2 dsum and what is at most that, so
    // they are 0 or at least 2^-25 of it, and below 2^126 as it is.  (Zero leaves no root but 0.)
    const double wmin = std::min(std::min(p.by_zx.y, p.by_zy.y), p.by_xy.y);
    pp.s_lo = (float)std::sqrt(0x1p-78 / wmin);
    pp.s_hi = (float)std::min(0x1p60, std::sqrt(0x1p121 / (double)p.by_sum.y));
    void *args[] = {&pp};
    return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(threads), args, smem, st);
}

}  // namespace tomo
