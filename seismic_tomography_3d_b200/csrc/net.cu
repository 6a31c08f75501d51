// Surrogate network kernels (sm_100a): the weight gradient of the 3x3x3 convolutions,
// resampling, head/loss, Adam, and the feature / target / data kernels.  The convolution
// forward (also used for dgrad, on flipped and transposed weights) runs on the tcgen05
// tensor cores (net_tc.cu).
//
// wgrad tiling.  Voxel tiles of 4 x 8 x 8 (256 voxels); the input halo of a 16-channel
// chunk (6 x 10 x 10 voxels, 32 B each) is staged in shared memory, and dW = dY^T X_shift
// is accumulated over the tiles with mma.sync.m16n8k16 (BF16 in, FP32 accumulate) and
// ldmatrix(.trans) operand loads: a tap shift is just a different row address into the
// halo.  The partial sums are added into the FP32 gradient with atomics once per CTA.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "net.cuh"

namespace tomo {
namespace net {

namespace {

constexpr int TD = 4, TH = 8, TW = 8;                       // output tile
constexpr int HD = TD + 2, HH = TH + 2, HW = TW + 2;        // halo tile
constexpr int kHalo = HD * HH * HW;                         // 600 voxels
constexpr int kTileVox = TD * TH * TW;                      // 256 voxels

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm_x4_t(unsigned addr, unsigned &r0, unsigned &r1, unsigned &r2, unsigned &r3)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}

__device__ __forceinline__ void mma16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
                 "{%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 16-byte asynchronous global -> shared copy; zeros where !in.
__device__ __forceinline__ void cp_async16(unsigned dst, const void *src, bool in)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}

struct TileCoord {
    int b, d0, h0, w0;
};

__device__ __forceinline__ TileCoord tile_of(long long t, const Vol &v)
{
    const int nw = (v.W + TW - 1) / TW, nh = (v.H + TH - 1) / TH, nd = (v.D + TD - 1) / TD;
    TileCoord c;
    c.w0 = (int)(t % nw) * TW;
    t /= nw;
    c.h0 = (int)(t % nh) * TH;
    t /= nh;
    c.d0 = (int)(t % nd) * TD;
    t /= nd;
    c.b = (int)t;
    return c;
}

__host__ __device__ inline long long tiles_of(const Vol &v)
{
    return (long long)v.B * ((v.D + TD - 1) / TD) * ((v.H + TH - 1) / TH) * ((v.W + TW - 1) / TW);
}

// Channels [ci0, ci0 + 16) of the halo tile (zero outside the volume): 2 x 16 B per voxel.
__device__ __forceinline__ void stage_halo(const bf16 *x, const Vol &v, int cin, int ci0, const TileCoord &tc,
                                           uint4 *dst)
{
    for (int i = threadIdx.x; i < kHalo * 2; i += blockDim.x) {
        const int hv = i >> 1, half = i & 1;
        const int hw = hv % HW, hh = (hv / HW) % HH, hd = hv / (HW * HH);
        const int d = tc.d0 + hd - 1, h = tc.h0 + hh - 1, w = tc.w0 + hw - 1;
        const bool in = d >= 0 && d < v.D && h >= 0 && h < v.H && w >= 0 && w < v.W;
        const long long vox = in ? (((long long)tc.b * v.D + d) * v.H + h) * v.W + w : 0;
        cp_async16(smem_u32(dst + i), x + vox * cin + ci0 + 8 * half, in);
    }
}

__device__ __forceinline__ int halo_index(int m, int dd, int dh, int dw)
{
    const int ww = m % TW, wh = (m / TW) % TH, wd = m / (TW * TH);
    return ((wd + dd) * HH + (wh + dh)) * HW + (ww + dw);
}

// wgrad: 9 warps, warp w owns taps 3w .. 3w+2; CTA owns 16 input channels (blockIdx.y) and
// NM output channels (blockIdx.z), and loops over voxel tiles (blockIdx.x strided).  A tile's
// operand loads (shared-memory bandwidth) would take a quarter of the kernel's time; the rest is
// waiting for its staging, so what counts is CTAs per SM and copies in flight: registers held to
// 4 CTAs an SM at NM = 16 and 3 at 32, staging by cp.async.  A gradient of 8 x 64^3 voxels:
// 6.15 -> 5.30 ms (2 CTAs an SM throughout: 5.37; 5 and 4, with spills: 6.87).
template <int NM>
__global__ void __launch_bounds__(288, NM == 16 ? 4 : NM == 32 ? 3 : 2) k_conv_wgrad(const bf16 *x, const bf16 *dy, float *dw, Vol v, int cin,
                                                    int cout)
{
    constexpr int MT = NM / 16;
    constexpr int DYS = NM + 8;  // padded row (elements): ldmatrix rows fall on distinct banks
    extern __shared__ uint4 sm[];
    uint4 *s_in = sm;
    bf16 *s_dy = reinterpret_cast<bf16 *>(sm + kHalo * 2);
    const int ci0 = blockIdx.y * 16, co0 = blockIdx.z * NM;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 3;
    float acc[3][MT][2][4];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < MT; b++)
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[a][b][c][e] = 0.f;
    const unsigned s_in_b = smem_u32(s_in);
    const long long ntiles = tiles_of(v);
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const TileCoord tc = tile_of(t, v);
        __syncthreads();
        stage_halo(x, v, cin, ci0, tc, s_in);
        for (int i = threadIdx.x; i < kTileVox * (NM / 8); i += blockDim.x) {
            const int r = i / (NM / 8), part = i % (NM / 8);
            const int ww = r % TW, wh = (r / TW) % TH, wd = r / (TW * TH);
            const int d = tc.d0 + wd, h = tc.h0 + wh, ws = tc.w0 + ww;
            const bool in = d < v.D && h < v.H && ws < v.W && co0 + part * 8 < cout;
            const long long vox = in ? (((long long)tc.b * v.D + d) * v.H + h) * v.W + ws : 0;
            cp_async16(smem_u32(s_dy + r * DYS + part * 8), dy + (in ? vox * cout + co0 + part * 8 : 0), in);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
#pragma unroll 1
        for (int kk = 0; kk < kTileVox / 16; kk++) {
            unsigned a[MT][4];
#pragma unroll
            for (int mt = 0; mt < MT; mt++) {
                const int row = kk * 16 + (q >> 1) * 8 + (lane & 7);
                const int col = mt * 16 + (q & 1) * 8;
                ldsm_x4_t(smem_u32(s_dy + row * DYS + col), a[mt][0], a[mt][1], a[mt][2], a[mt][3]);
            }
            const int m = kk * 16 + (q & 1) * 8 + (lane & 7);
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const int tap = warp * 3 + j;
                const int hidx = halo_index(m, tap / 9, (tap / 3) % 3, tap % 3);
                unsigned b0, b1, b2, b3;
                ldsm_x4_t(s_in_b + (hidx * 16 + (q >> 1) * 8) * 2, b0, b1, b2, b3);
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    mma16816(acc[j][mt][0], a[mt], b0, b1);
                    mma16816(acc[j][mt][1], a[mt], b2, b3);
                }
            }
        }
    }
    const int g = lane >> 2, c2 = (lane & 3) * 2;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int tap = warp * 3 + j;
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int nt = 0; nt < 2; nt++)
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int co = co0 + mt * 16 + g + (r >= 2 ? 8 : 0);
                    const int ci = ci0 + nt * 8 + c2 + (r & 1);
                    if (co < cout) atomicAdd(dw + ((long long)co * 27 + tap) * cin + ci, acc[j][mt][nt][r]);
                }
    }
}

__device__ __forceinline__ void unpack8(const uint4 &q, float (&f)[8])
{
    const __nv_bfloat162 *p = reinterpret_cast<const __nv_bfloat162 *>(&q);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float2 v = __bfloat1622float2(p[k]);
        f[2 * k] = v.x;
        f[2 * k + 1] = v.y;
    }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8])
{
    uint4 q;
    __nv_bfloat162 *p = reinterpret_cast<__nv_bfloat162 *>(&q);
#pragma unroll
    for (int k = 0; k < 4; k++) p[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
    return q;
}

// Sums over voxels per channel.  A thread keeps one 16-byte group of 8 channels and reads every
// stride-th voxel's; the block's 256 x 8 sums meet in shared memory.  (2-byte loads and a shared
// atomic per thread took 0.57 ms for the 14 layers of 8 x 64^3 voxels; now 0.17.)
__global__ void __launch_bounds__(256) k_bias_grad(const uint4 *dy, float *db, long long n8, int c8)
{
    __shared__ float sums[256 * 8];
    const long long nth = (long long)gridDim.x * blockDim.x, stride = nth - nth % c8;  // a multiple of c8
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    float s[8] = {};
    if (t < stride) {
#pragma unroll 4
        for (long long e = t; e < n8; e += stride) {
            float v[8];
            unpack8(__ldg(dy + e), v);
#pragma unroll
            for (int k = 0; k < 8; k++) s[k] += v[k];
        }
    }
#pragma unroll
    for (int k = 0; k < 8; k++) sums[threadIdx.x * 8 + k] = s[k];
    __syncthreads();
    if ((int)threadIdx.x >= 8 * c8) return;
    // channel threadIdx.x: the threads whose group it is in
    const int first = (int)(blockIdx.x * (long long)blockDim.x % c8);
    float v = 0.f;
    for (int i = ((int)threadIdx.x / 8 - first + c8) % c8; i < 256; i += c8) v += sums[i * 8 + threadIdx.x % 8];
    atomicAdd(db + threadIdx.x, v);
}

// coarse voxel index -> its 8 fine children
__device__ __forceinline__ long long fine_index(const Vol &f, long long cv, int k)
{
    const int cw = f.W / 2, ch = f.H / 2, cd = f.D / 2;
    const int w = (int)(cv % cw);
    long long r = cv / cw;
    const int h = (int)(r % ch);
    r /= ch;
    const int d = (int)(r % cd);
    const int b = (int)(r / cd);
    return (((long long)b * f.D + 2 * d + (k >> 2)) * f.H + 2 * h + ((k >> 1) & 1)) * f.W + 2 * w + (k & 1);
}

// Resampling.  Every kernel moves 8 channels (16 B) per thread and reads and writes each tensor
// once; the values are rounded where the separate operations they stand for round.  (One thread
// per 2-byte value, with the upsampled copies, the split concatenations and the ReLU masks as
// passes of their own, took 1.04 ms per gradient of 8 x 64^3 voxels; now 0.21.)

// f where the activation y is positive, else 0 (the gradient through ReLU).
__device__ __forceinline__ void relu_mask(const uint4 &y, float (&f)[8])
{
    float a[8];
    unpack8(y, a);
#pragma unroll
    for (int k = 0; k < 8; k++) f[k] = a[k] > 0.f ? f[k] : 0.f;
}

__global__ void k_pool_fwd(const uint4 *x, uint4 *y, Vol f, int c8)
{
    const long long n = f.voxels() / 8 * c8;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long cv = e / c8;
        const int ch = (int)(e - cv * c8);
        uint4 q[8];
#pragma unroll
        for (int k = 0; k < 8; k++) q[k] = __ldg(x + fine_index(f, cv, k) * c8 + ch);
        float s[8] = {};
#pragma unroll
        for (int k = 0; k < 8; k++) {
            float v[8];
            unpack8(q[k], v);
#pragma unroll
            for (int i = 0; i < 8; i++) s[i] += v[i];
        }
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] *= 0.125f;
        y[e] = pack8(s);
    }
}

// y = [x nearest-upsampled x2 | skip], per coarse voxel: its 8 fine voxels
__global__ void k_up_concat(const uint4 *x, int ca8, const uint4 *skip, int cb8, uint4 *y, Vol f)
{
    const int c8 = ca8 + cb8;
    const long long n = f.voxels() / 8 * c8;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long cv = e / c8;
        const int ch = (int)(e - cv * c8);
        uint4 q[8];
        if (ch < ca8) {
            const uint4 one = __ldg(x + cv * ca8 + ch);
#pragma unroll
            for (int k = 0; k < 8; k++) q[k] = one;
        } else {
#pragma unroll
            for (int k = 0; k < 8; k++) q[k] = __ldg(skip + fine_index(f, cv, k) * cb8 + (ch - ca8));
        }
#pragma unroll
        for (int k = 0; k < 8; k++) y[fine_index(f, cv, k) * c8 + ch] = q[k];
    }
}

// dx = relu'(x) sum over the 8 fine voxels of dy's first ca8 groups (of c8)
__global__ void k_up_bwd(const uint4 *dy, int c8, const uint4 *x, uint4 *dx, int ca8, Vol f)
{
    const long long n = f.voxels() / 8 * ca8;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long cv = e / ca8;
        const int ch = (int)(e - cv * ca8);
        uint4 q[8];
#pragma unroll
        for (int k = 0; k < 8; k++) q[k] = __ldg(dy + fine_index(f, cv, k) * c8 + ch);
        const uint4 act = __ldg(x + e);
        float s[8] = {};
#pragma unroll
        for (int k = 0; k < 8; k++) {
            float v[8];
            unpack8(q[k], v);
#pragma unroll
            for (int i = 0; i < 8; i++) s[i] += v[i];
        }
        relu_mask(act, s);
        dx[e] = pack8(s);
    }
}

// dx = relu'(x) (skip gradient: groups [off8, off8 + cb8) of dy, c8 per voxel, + the pooling
// path's dp / 8), per coarse voxel
__global__ void k_skip_bwd(const uint4 *dy, int c8, int off8, const uint4 *dp, const uint4 *x, uint4 *dx, int cb8, Vol f)
{
    const long long n = f.voxels() / 8 * cb8;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long cv = e / cb8;
        const int ch = (int)(e - cv * cb8);
        float g[8];
        unpack8(__ldg(dp + e), g);
#pragma unroll
        for (int i = 0; i < 8; i++) g[i] = __bfloat162float(__float2bfloat16_rn(0.125f * g[i]));
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const long long v = fine_index(f, cv, k);
            float s[8];
            unpack8(__ldg(dy + v * c8 + off8 + ch), s);
#pragma unroll
            for (int i = 0; i < 8; i++) s[i] += g[i];
            relu_mask(__ldg(x + v * cb8 + ch), s);
            dx[v * cb8 + ch] = pack8(s);
        }
    }
}

__device__ __forceinline__ double block_sum(double v, double *sh)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += sh[w];
    __syncthreads();
    return s;
}

// The head's 16 channels of a voxel, in two 16-byte loads.
__device__ __forceinline__ void load16(const bf16 *y, long long v, float (&f)[16])
{
    const uint4 *q = reinterpret_cast<const uint4 *>(y + v * 16);
    float a[8], b[8];
    unpack8(__ldg(q), a);
    unpack8(__ldg(q + 1), b);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        f[k] = a[k];
        f[8 + k] = b[k];
    }
}

__global__ void k_head_fwd(const bf16 *y, const float *wh, const float *bh, float *tau, const float *target,
                           long long n, double *acc)
{
    __shared__ double sh[32];
    double se = 0.0, cnt = 0.0;
    float w[16];
#pragma unroll
    for (int k = 0; k < 16; k++) w[k] = __ldg(wh + k);
    const float b = __ldg(bh);
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        float f[16];
        load16(y, v, f);
        float s = 1.0f + b;
#pragma unroll
        for (int k = 0; k < 16; k++) s += w[k] * f[k];
        tau[v] = s;
        if (target && target[v] > 0.f) {
            const double d = (double)s - (double)target[v];
            se += d * d;
            cnt += 1.0;
        }
    }
    if (!target) return;
    se = block_sum(se, sh);
    cnt = block_sum(cnt, sh);
    if (threadIdx.x == 0) {
        atomicAdd(acc, se);
        atomicAdd(acc + 1, cnt);
    }
}

// A thread sums its voxels' 17 gradients in registers, a warp by shuffles, and the block's warps
// meet in shared memory (a shared atomic per voxel and channel took 0.74 ms on 8 x 64^3 voxels;
// now 0.04).  dy goes out masked by the ReLU of y.
__global__ void __launch_bounds__(256) k_head_bwd(const bf16 *y, const float *wh, const float *tau, const float *target,
                                                  const double *acc, bf16 *dy, float *dwh, float *dbh, long long n)
{
    __shared__ float sw[17];
    if (threadIdx.x < 17) sw[threadIdx.x] = 0.f;
    __syncthreads();
    const float scale = acc[1] > 0.0 ? (float)(2.0 / acc[1]) : 0.f;
    float w[16], s[17] = {};
#pragma unroll
    for (int k = 0; k < 16; k++) w[k] = __ldg(wh + k);
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const float g = target[v] > 0.f ? scale * (tau[v] - target[v]) : 0.f;
        float f[16], d0[8], d1[8];
        load16(y, v, f);
        s[16] += g;
        if (g != 0.f)  // an infinite activation where there is no loss adds nothing, not 0 x inf
#pragma unroll
            for (int k = 0; k < 16; k++) s[k] += g * f[k];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            d0[k] = f[k] > 0.f ? g * w[k] : 0.f;
            d1[k] = f[8 + k] > 0.f ? g * w[8 + k] : 0.f;
        }
        uint4 *out = reinterpret_cast<uint4 *>(dy + v * 16);
        out[0] = pack8(d0);
        out[1] = pack8(d1);
    }
#pragma unroll
    for (int k = 0; k < 17; k++) {
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        if ((threadIdx.x & 31) == 0) atomicAdd(&sw[k], s[k]);
    }
    __syncthreads();
    if (threadIdx.x < 16) atomicAdd(dwh + threadIdx.x, sw[threadIdx.x]);
    if (threadIdx.x == 16) atomicAdd(dbh, sw[16]);
}

__global__ void k_adam(float *p, const float *g, float *m, float *v, long long n, float lr, float b1, float b2,
                       float eps, float c1, float c2)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const float gr = g[e];
        const float mm = b1 * m[e] + (1.f - b1) * gr;
        const float vv = b2 * v[e] + (1.f - b2) * gr * gr;
        m[e] = mm;
        v[e] = vv;
        p[e] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    }
}

struct JobGeo {
    int y, x, z;      // clamped window node
    bool inside;
    float dist, s, s_src;
};

__device__ __forceinline__ JobGeo job_geo(const Job &j, long long i, float h)
{
    JobGeo q;
    const int w = (int)(i % j.pw);
    const long long r = i / j.pw;
    const int hh = (int)(r % j.ph), d = (int)(r / j.ph);
    const int k = j.stride;  // network voxel (d, hh, w) samples window node (k d, k hh, k w)
    q.inside = d * k < j.wny && hh * k < j.wnx && w * k < j.nz;
    q.y = min(d * k, j.wny - 1);
    q.x = min(hh * k, j.wnx - 1);
    q.z = min(w * k, j.nz - 1);
    const float ex = q.x * h - j.sx, ey = q.y * h - j.sy, ez = q.z * h - j.sz;
    q.dist = sqrtf(ex * ex + ey * ey + ez * ez);
    const long long mstride = (long long)j.nz * j.model_nx;
    q.s = __ldg(j.slow + q.z + (long long)j.nz * (j.wx0 + q.x) + mstride * (j.wy0 + q.y));
    const int sz = min((int)(j.sz / h), j.nz - 1), sx = min((int)(j.sx / h), j.wnx - 1),
              sy = min((int)(j.sy / h), j.wny - 1);
    q.s_src = __ldg(j.slow + sz + (long long)j.nz * (j.wx0 + sx) + mstride * (j.wy0 + sy));
    return q;
}

__global__ void k_features(const Job *jobs, float h, bf16 *x16)
{
    const Job j = jobs[blockIdx.y];
    const long long n = (long long)j.pd * j.ph * j.pw;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const JobGeo q = job_geo(j, i, h);
        __align__(16) bf16 f[16];
#pragma unroll
        for (int k = 0; k < 16; k++) f[k] = __float2bfloat16_rn(0.f);
        f[0] = __float2bfloat16_rn(q.s / q.s_src - 1.0f);
        f[1] = __float2bfloat16_rn(q.dist / (64.0f * h * (float)j.stride));
        uint4 *dst = reinterpret_cast<uint4 *>(x16 + (j.out_off + i) * 16);
        dst[0] = reinterpret_cast<const uint4 *>(f)[0];
        dst[1] = reinterpret_cast<const uint4 *>(f)[1];
    }
}

__global__ void k_tau_target(const Job *jobs, float h, float *tau)
{
    const Job j = jobs[blockIdx.y];
    const long long n = (long long)j.pd * j.ph * j.pw;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const JobGeo q = job_geo(j, i, h);
        float t = 0.f;
        if (q.inside && q.dist >= h) {
            const float tt = j.T[q.z + (long long)j.nz * (q.x + (long long)j.wnx * q.y)];
            t = tt / (q.s_src * q.dist);
        }
        tau[j.out_off + i] = t;
    }
}

// Weight of window node x between the sampled nodes of an axis of n nodes at stride k (node
// c sits at min(c k, n - 1)).
__device__ __forceinline__ void axis_weight(int x, int k, int n, int &c0, int &c1, float &t)
{
    const int nc = (n + k - 1) / k;
    c0 = min(x / k, nc - 1);
    c1 = min(c0 + 1, nc - 1);
    const int p0 = c0 * k, p1 = min(c1 * k, n - 1);
    t = p1 > p0 ? (float)(x - p0) / (float)(p1 - p0) : 0.f;
}

// T = tau s_src distance at every window node, tau trilinear between the sampled nodes
// (kStrided) or read as it is (stride 1).
//
// The kernel writes 4 bytes a node and reads 1/k^3 of that, so it should run at the store
// rate; with one node per thread it was bound by the six 64-bit and six 32-bit integer
// divisions that took the node's index apart.  Here a thread owns one (z, y) of the window
// and walks a run of kTimeRun nodes along x: its z and y weights, its distance part and its
// four column pointers are formed once, x and its cell are the same for the whole block (a
// counter instead of a division), and the values interpolated along z are reloaded only
// where x enters a new cell.  Lanes follow z, the fastest axis, across column ends, so no
// lane idles on a depth that is not a multiple of 32.  64 windows of 201 x 201 x 101 at
// stride 4 (261 M nodes): the kernel 3.70 -> 0.52 ms (0.71 with IEEE root and
// division and runs of 32); issue in 76 % of the slots on 8 windows.
constexpr int kTimeRun = 64;

// kFast: the short root of common.cuh and 32-bit (z, y) pairs; else the IEEE root and 64 bits (a
// 64-bit division a thread: 2.81 ms for the prediction above instead of 2.79).  Squared distances
// of spacings in [2^-50, 2^30] lie in the short root's range, or below h^2, where the time is 0
// either way.
template <bool kStrided, bool kFast>
__global__ void __launch_bounds__(256) k_tau_to_time(const Job *jobs, float h, const float *tau, float *t_out)
{
    const Job j = jobs[blockIdx.z];
    const int k = kStrided ? j.stride : 1;
    typedef typename std::conditional<kFast, int, long long>::type Pair;
    const Pair q = blockIdx.x * (Pair)blockDim.x + threadIdx.x;  // (z, y) pair
    if (q >= (Pair)j.nz * j.wny) return;
    const int sz = min((int)(j.sz / h), j.nz - 1), sx = min((int)(j.sx / h), j.wnx - 1),
              sy = min((int)(j.sy / h), j.wny - 1);
    const float s_src =
        __ldg(j.slow + sz + (long long)j.nz * (j.wx0 + sx) + (long long)j.nz * j.model_nx * (j.wy0 + sy));
    const int y = (int)(q / j.nz), z = (int)(q - (Pair)y * j.nz);
    const float ey = y * h - j.sy, ez = z * h - j.sz;
    int z0 = z, z1 = z, y0 = y, y1 = y;
    float tz = 0.f, ty = 0.f;
    if (kStrided) {
        axis_weight(z, k, j.nz, z0, z1, tz);
        axis_weight(y, k, j.wny, y0, y1, ty);
    }
    // tau columns of the sampled depths and rows, at sampled x = 0; one step in x is pw
    const float *tj = tau + j.out_off;
    const float *p00 = tj + z0 + (long long)j.pw * j.ph * y0, *p10 = tj + z1 + (long long)j.pw * j.ph * y0;
    const float *p01 = tj + z0 + (long long)j.pw * j.ph * y1, *p11 = tj + z1 + (long long)j.pw * j.ph * y1;
    auto at = [&](const float *lo, const float *hi, int c) {
        return __ldg(lo + (long long)j.pw * c) * (1.f - tz) + __ldg(hi + (long long)j.pw * c) * tz;
    };
    const int nc = (j.wnx + k - 1) / k;
    for (int xa = blockIdx.y * kTimeRun; xa < j.wnx; xa += gridDim.y * kTimeRun) {
        const int xe = min(xa + kTimeRun, j.wnx);
        float *out = t_out + j.nat_off + z + (long long)j.nz * (xa + (long long)j.wnx * y);
        int c = xa / k, rem = xa - c * k;  // x = c k + rem
        int c1 = min(c + 1, nc - 1);
        Divisor den = divisor((float)(min(c1 * k, j.wnx - 1) - c * k));
        float c00 = 0.f, c01 = 0.f, c10 = 0.f, c11 = 0.f;
        if (kStrided) {
            c00 = at(p00, p10, c);
            c01 = at(p01, p11, c);
            c10 = at(p00, p10, c1);
            c11 = at(p01, p11, c1);
        }
        for (int x = xa; x < xe; x++, out += j.nz) {
            if (kStrided && rem == k) {  // the next cell: its lower corner is the last one's upper
                rem = 0;
                c = c1;
                c1 = min(c + 1, nc - 1);
                den = divisor((float)(min(c1 * k, j.wnx - 1) - c * k));
                c00 = c10;
                c01 = c11;
                if (c1 > c) {
                    c10 = at(p00, p10, c1);
                    c11 = at(p01, p11, c1);
                }
            }
            const float ex = x * h - j.sx;
            const float d2 = ex * ex + ey * ey + ez * ez, dist = kFast ? fsqrt(d2) : sqrtf(d2);
            float t = 0.f;
            if (dist >= h) {
                if (kStrided) {
                    const float tx = den.y > 0.f ? fdiv((float)rem, den) : 0.f;
                    const float c0 = c00 * (1.f - tx) + c10 * tx, cc = c01 * (1.f - tx) + c11 * tx;
                    t = (c0 * (1.f - ty) + cc * ty) * s_src * dist;
                } else {
                    t = __ldg(p00 + (long long)j.pw * x) * s_src * dist;
                }
            }
            __stcs(out, t);
            rem++;
        }
    }
}

__global__ void k_random_models(const TileModel *tiles, float *slow, int nx, int ny, int nz)
{
    const TileModel &tm = tiles[blockIdx.y];
    const long long n = (long long)tm.n * tm.n * nz;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int z = (int)(i % nz);
        const long long r = i / nz;
        const int x = (int)(r % tm.n), y = (int)(r / tm.n);
        int layer = 0;
        for (int k = 0; k < tm.nlayers - 1; k++)
            if ((float)z > tm.z0[k] + tm.gx[k] * x + tm.gy[k] * y) layer = k + 1;
        float v = tm.vel[layer];
        for (int a = 0; a < tm.nanom; a++) {
            const float dx = x - tm.ax[a], dy = y - tm.ay[a], dz = z - tm.az[a];
            v *= 1.0f + tm.aamp[a] * expf(-(dx * dx + dy * dy + dz * dz) / (2.0f * tm.asig[a] * tm.asig[a]));
        }
        const int gx = tm.x0 + x, gy = tm.y0 + y;
        if (gx < nx && gy < ny) slow[z + (long long)nz * (gx + (long long)nx * gy)] = 1.0f / v;
    }
}

int grid1(long long n, int threads)
{
    long long g = (n + threads - 1) / threads;
    if (g > 148LL * 64) g = 148LL * 64;
    return g < 1 ? 1 : (int)g;
}

template <int NM>
cudaError_t launch_wgrad(const bf16 *x, const bf16 *dy, float *dw, Vol v, int cin, int cout, cudaStream_t st)
{
    const size_t smem = (size_t)kHalo * 2 * sizeof(uint4) + (size_t)kTileVox * (NM + 8) * sizeof(bf16);
    cudaError_t e = cudaFuncSetAttribute(k_conv_wgrad<NM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const long long nt = tiles_of(v);
    const int ny = cin / 16, nz = (cout + NM - 1) / NM;
    // several times the resident CTAs (2-4 an SM), so that the last ones to finish are short
    // (4 / 8 / 12 per SM: 5.37 / 5.30 / 5.28 ms per gradient of 8 x 64^3 voxels)
    long long gx = (8 * 148LL + ny * nz - 1) / (ny * nz);
    if (gx > nt) gx = nt;
    if (gx < 1) gx = 1;
    k_conv_wgrad<NM><<<dim3((unsigned)gx, (unsigned)ny, (unsigned)nz), 288, smem, st>>>(x, dy, dw, v, cin, cout);
    return cudaGetLastError();
}

}  // namespace

cudaError_t conv_wgrad(const bf16 *x, const bf16 *dy, float *dw, Vol v, int cin, int cout, cudaStream_t st)
{
    if (cin % 16 || cout % 16 || cin < 16 || cout < 16) return cudaErrorInvalidValue;
    switch (cout >= 64 ? 64 : cout) {
    case 16: return launch_wgrad<16>(x, dy, dw, v, cin, cout, st);
    case 32: return launch_wgrad<32>(x, dy, dw, v, cin, cout, st);
    case 48: return launch_wgrad<48>(x, dy, dw, v, cin, cout, st);
    default: return launch_wgrad<64>(x, dy, dw, v, cin, cout, st);
    }
}

namespace {
const uint4 *q4(const bf16 *p) { return reinterpret_cast<const uint4 *>(p); }
uint4 *q4(bf16 *p) { return reinterpret_cast<uint4 *>(p); }
bool halves(const Vol &f) { return f.D % 2 == 0 && f.H % 2 == 0 && f.W % 2 == 0; }
}  // namespace

cudaError_t bias_grad(const bf16 *dy, float *db, long long voxels, int c, cudaStream_t st)
{
    if (c > 256 || c % 8) return cudaErrorInvalidValue;
    const long long n8 = voxels * c / 8, want = (n8 + 256 * 16 - 1) / (256 * 16);
    k_bias_grad<<<(unsigned)std::min<long long>(std::max<long long>(want, 1), 148 * 8), 256, 0, st>>>(q4(dy), db, n8, c / 8);
    return cudaGetLastError();
}

cudaError_t pool_fwd(const bf16 *x, bf16 *y, Vol f, int c, cudaStream_t st)
{
    if (!halves(f) || c % 8) return cudaErrorInvalidValue;
    k_pool_fwd<<<grid1(f.voxels() / 64 * c, 256), 256, 0, st>>>(q4(x), q4(y), f, c / 8);
    return cudaGetLastError();
}

cudaError_t up_concat(const bf16 *x, int ca, const bf16 *skip, int cb, bf16 *y, Vol f, cudaStream_t st)
{
    if (!halves(f) || ca % 8 || cb % 8) return cudaErrorInvalidValue;
    k_up_concat<<<grid1(f.voxels() / 64 * (ca + cb), 256), 256, 0, st>>>(q4(x), ca / 8, q4(skip), cb / 8, q4(y), f);
    return cudaGetLastError();
}

cudaError_t up_bwd(const bf16 *dy, int c, const bf16 *x, bf16 *dx, int ca, Vol f, cudaStream_t st)
{
    if (!halves(f) || c % 8 || ca % 8 || ca > c) return cudaErrorInvalidValue;
    k_up_bwd<<<grid1(f.voxels() / 64 * ca, 256), 256, 0, st>>>(q4(dy), c / 8, q4(x), q4(dx), ca / 8, f);
    return cudaGetLastError();
}

cudaError_t skip_bwd(const bf16 *dy, int c, const bf16 *dp, const bf16 *x, bf16 *dx, int cb, Vol f, cudaStream_t st)
{
    if (!halves(f) || c % 8 || cb % 8 || cb > c) return cudaErrorInvalidValue;
    k_skip_bwd<<<grid1(f.voxels() / 64 * cb, 256), 256, 0, st>>>(q4(dy), c / 8, (c - cb) / 8, q4(dp), q4(x), q4(dx), cb / 8, f);
    return cudaGetLastError();
}

cudaError_t head_fwd(const bf16 *y, const float *wh, const float *bh, float *tau, const float *target, long long voxels,
                     double *acc, cudaStream_t st)
{
    k_head_fwd<<<grid1(voxels, 256), 256, 0, st>>>(y, wh, bh, tau, target, voxels, acc);
    return cudaGetLastError();
}

cudaError_t head_bwd(const bf16 *y, const float *wh, const float *tau, const float *target, const double *acc, bf16 *dy,
                     float *dwh, float *dbh, long long voxels, cudaStream_t st)
{
    const long long want = (voxels + 255) / 256;
    k_head_bwd<<<(unsigned)std::min<long long>(want, 148 * 8), 256, 0, st>>>(y, wh, tau, target, acc, dy, dwh, dbh, voxels);
    return cudaGetLastError();
}

cudaError_t adam(float *p, const float *g, float *m, float *v, long long n, float lr, float b1, float b2, float eps,
                 int t, cudaStream_t st)
{
    const float c1 = 1.f - std::pow(b1, (float)t), c2 = 1.f - std::pow(b2, (float)t);
    k_adam<<<grid1(n, 256), 256, 0, st>>>(p, g, m, v, n, lr, b1, b2, eps, c1, c2);
    return cudaGetLastError();
}

cudaError_t features(const Job *jobs, int njobs, float h, bf16 *x16, long long max_vox, cudaStream_t st)
{
    if (njobs < 1 || njobs > 65535) return cudaErrorInvalidValue;
    k_features<<<dim3((unsigned)grid1(max_vox, 256) / 8 + 1, (unsigned)njobs), 256, 0, st>>>(jobs, h, x16);
    return cudaGetLastError();
}

cudaError_t tau_target(const Job *jobs, int njobs, float h, float *tau, long long max_vox, cudaStream_t st)
{
    if (njobs < 1 || njobs > 65535) return cudaErrorInvalidValue;
    k_tau_target<<<dim3((unsigned)grid1(max_vox, 256) / 8 + 1, (unsigned)njobs), 256, 0, st>>>(jobs, h, tau);
    return cudaGetLastError();
}

cudaError_t tau_to_time(const Job *jobs, int njobs, float h, int stride, const float *tau, float *t_out,
                        long long max_plane, int max_wnx, cudaStream_t st)
{
    if (njobs < 1 || njobs > 65535 || max_plane < 1 || max_wnx < 1) return cudaErrorInvalidValue;
    const int runs = (max_wnx + kTimeRun - 1) / kTimeRun;
    if (max_plane > 256LL * 0x7fffffff) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)((max_plane + 255) / 256), (unsigned)(runs < 65535 ? runs : 65535), (unsigned)njobs);
    const bool fast = h >= 0x1p-50f && h <= 0x1p30f && max_plane < (1LL << 31) - 256;
    auto fn = stride > 1 ? (fast ? k_tau_to_time<true, true> : k_tau_to_time<true, false>)
                         : (fast ? k_tau_to_time<false, true> : k_tau_to_time<false, false>);
    fn<<<grid, 256, 0, st>>>(jobs, h, tau, t_out);
    return cudaGetLastError();
}

cudaError_t random_models(const TileModel *tiles, int ntiles, float *slow, int nx, int ny, int nz, cudaStream_t st)
{
    if (ntiles < 1 || ntiles > 65535) return cudaErrorInvalidValue;
    k_random_models<<<dim3(64, (unsigned)ntiles), 256, 0, st>>>(tiles, slow, nx, ny, nz);
    return cudaGetLastError();
}

}  // namespace net
}  // namespace tomo
