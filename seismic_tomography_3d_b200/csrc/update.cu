// Model update on the device (sm_100a): trilinear coarse-to-fine of the CGLS solution,
// 3D Gaussian smoothing, masked slowness update, velocity output, and the data residual.
// FP32 arithmetic follows the reference operation order with round-to-nearest intrinsics
// (no FMA contraction), so results are bit-identical to Least_squares::model_update
// (src/tomography/least_squares/least_squares.cpp:498-570) and gaussian
// (src/utils/smoothing/gaussian.cpp:5-73).
#include "cgls.cuh"
#include "common.cuh"
#include "fim.cuh"

namespace tomo {

namespace {

__device__ __forceinline__ float flat_at(const float *a, long long n, long long i)
{
    return (i >= 0 && i < n) ? __ldg(a + i) : 0.0f;
}

int grid_for(long long n, int threads)
{
    long long g = (n + threads - 1) / threads;
    if (g > 148LL * 32) g = 148LL * 32;
    return g < 1 ? 1 : (int)g;
}

}  // namespace

// dm at every model node: trilinear in the CGLS solution (least_squares.cpp:505-540).
//
// A thread owns one (z, y) and walks a run of kDmRun nodes along x.  A node needs 9 IEEE
// divisions and 3 floors of per-axis quantities and 8 cell values; one node per thread
// computed them all, and took its 64-bit index apart by division.  Here the z and y weights
// are formed once per thread, the x weights once per block (shared memory), and the 8 values
// are reloaded only where x enters a new cell, so the 4-byte store a node is the bound.
// 401 x 401 x 201 nodes: 0.29 -> 0.06 ms.
constexpr int kDmRun = 32;

struct AxisWeight {
    float w;  // fraction between the cell's lower corner and the next one
    int c;    // cell index
};

__device__ __forceinline__ AxisWeight axis_weight(int n, float d, float dt)
{
    AxisWeight a;
    const float x = fmul((float)n, d), q = fdiv(x, dt), f = floorf(q);
    const float x0 = fmul(f, dt), x1 = fadd(fmul(f, dt), dt);
    a.w = fdiv(fsub(x, x0), fsub(x1, x0));
    a.c = (int)q;
    return a;
}

__global__ void __launch_bounds__(256)
    k_model_dm(const float *xdm, float *dm, int nx, int ny, int nz, float dx, float dy, float dz, float dxt, float dyt,
               float dzt, int nxt, int nyt, int nzt, UpdateMasks m)
{
    __shared__ AxisWeight sx[kDmRun];
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const bool mine = q < (long long)nz * ny;
    const int k = mine ? (int)(q / nz) : 0, i = mine ? (int)(q - (long long)k * nz) : 0;
    const AxisWeight wy = axis_weight(k, dy, dyt), wz = axis_weight(i, dz, dzt);
    const bool in_zy = i >= m.i_lo && i < nz - m.i_hi_off && k >= m.k_lo && k < ny - m.k_hi_off_dm;
    const long long nm = (long long)nxt * nyt * nzt, base = wz.c + (long long)wy.c * nxt * nzt;
    const long long step_y = (long long)nxt * nzt;
    for (int ja = blockIdx.y * kDmRun; ja < nx; ja += gridDim.y * kDmRun) {
        __syncthreads();
        if (threadIdx.x < kDmRun) sx[threadIdx.x] = axis_weight(ja + (int)threadIdx.x, dx, dxt);
        __syncthreads();
        if (!mine) continue;
        const int je = min(ja + kDmRun, nx);
        float *out = dm + i + (long long)nz * (ja + (long long)nx * k);
        float c000 = 0.f, c001 = 0.f, c100 = 0.f, c101 = 0.f, c010 = 0.f, c011 = 0.f, c110 = 0.f, c111 = 0.f;
        int cell = -1;
        for (int j = ja; j < je; j++, out += nz) {
            float v = 0.0f;
            if (in_zy && j >= m.j_lo && j < nx - m.j_hi_off_dm) {
                const AxisWeight wx = sx[j - ja];
                if (wx.c != cell) {
                    cell = wx.c;
                    const long long im = base + (long long)cell * nzt;
                    c000 = flat_at(xdm, nm, im);
                    c001 = flat_at(xdm, nm, im + 1);
                    c100 = flat_at(xdm, nm, im + nzt);
                    c101 = flat_at(xdm, nm, im + 1 + nzt);
                    c010 = flat_at(xdm, nm, im + step_y);
                    c011 = flat_at(xdm, nm, im + 1 + step_y);
                    c110 = flat_at(xdm, nm, im + nzt + step_y);
                    c111 = flat_at(xdm, nm, im + 1 + nzt + step_y);
                }
                v = trilinear_weights(c000, c001, c100, c101, c010, c011, c110, c111, wx.w, wy.w, wz.w);
            }
            *out = v;
        }
    }
}

// One output node per thread; taps summed in the reference's (y, x, z) loop order.  Only for
// filters of more than kMaxFused samples; the others are summed inside k_model_update.
__global__ void k_gaussian(const float *in, float *out, int nx, int ny, int nz, int samples, const float *kernel)
{
    const long long n = (long long)nx * ny * nz;
    const int init = samples / 2;
    for (long long index = blockIdx.x * (long long)blockDim.x + threadIdx.x; index < n;
         index += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(index / ((long long)nx * nz));
        const int j = (int)((index - (long long)k * nx * nz) / nz);
        const int i = (int)(index - (long long)j * nz - (long long)k * nx * nz);
        if (k < init || k >= ny - init || j < init || j >= nx - init || i < init || i >= nz - init) {
            out[index] = __ldg(in + index);
            continue;
        }
        float accum = 0.0f;
        for (int yk = 0; yk < samples; yk++)
            for (int xk = 0; xk < samples; xk++) {
                const float *row = in + (i - init) + (long long)(j - init + xk) * nz + (long long)(k - init + yk) * nx * nz;
                const float *kr = kernel + xk * samples + yk * samples * samples;
                for (int zk = 0; zk < samples; zk++) accum = fadd(accum, fmul(__ldg(row + zk), __ldg(kr + zk)));
            }
        out[index] = accum;
    }
}

// Smoothing with an S^3 filter (S = 1: none), slowness += dm, velocity = 1 / slowness, and the
// new slowness into the brick-major copy, in one pass.
//
// The filter is S^3 multiplies and adds a node in the reference's (y, x, z) order (no FMA),
// so FP32 issue is the bound (S = 5: 250 instructions a node, 0.23 ms for 32 M nodes) -- if
// the operands cost little.  One node per thread loaded 125 values and 125 weights for them
// (2.37 ms) and left three more passes over the model to k_model_apply and k_brick_model.
// Here a block stages a 32 (z) x kUpdX x 8 (y) tile of dm and its halo in shared memory, a
// thread owns kUpdX nodes along x, and for each y plane of the filter holds the plane's S^2
// weights in registers while the S values of each of the kUpdX + S - 1 rows serve the up to
// S outputs that need them: 1.6 shared loads per 10 FP32 instructions, conflict-free (lanes
// along z).  Each output still sums its taps in (y, x, z) order, so the result is the
// reference's bit for bit.  401 x 401 x 201 nodes, 5 samples: 2.91 -> 0.61 ms for the whole
// update (four kernels before, two now); this kernel 0.54 ms at 88 % of the issue slots.  The
// tile goes in by cp.async, all of a thread's 34 copies in flight (0.62 ms with plain loads).
constexpr int kUpdZ = 32, kUpdX = 16, kUpdY = 8;
constexpr int kMaxFused = 7;

template <int S>
__global__ void __launch_bounds__(kUpdZ *kUpdY)
    k_model_update(const float *dm, float *slowness, float *bricks, float *velocity, const float *kernel, int nx,
                   int ny, int nz, int nxx, int nyy, int nzz, UpdateMasks m)
{
    constexpr int H = S / 2, TZ = kUpdZ + 2 * H, TX = kUpdX + 2 * H, TY = kUpdY + 2 * H;
    __shared__ float tile[TY][TX][TZ];
    __shared__ float weights[S * S * S];
    const int tz = threadIdx.x, ty = threadIdx.y, tid = tz + kUpdZ * ty;
    const int tiles_z = (nz + kUpdZ - 1) / kUpdZ, tiles_x = (nx + kUpdX - 1) / kUpdX;
    const int i0 = (int)(blockIdx.x % tiles_z) * kUpdZ;
    const int j0 = (int)(blockIdx.x / tiles_z % tiles_x) * kUpdX, k0 = (int)(blockIdx.x / tiles_z / tiles_x) * kUpdY;
    // the thread's slowness values: in flight while the filter runs (read after the stores of
    // the epilogue began, each would wait for the one before)
    const int i = i0 + tz, k = k0 + ty;
    float s[kUpdX];
    if (i < nz && k < ny) {
#pragma unroll
        for (int r = 0; r < kUpdX; r++)
            s[r] = j0 + r < nx ? slowness[i + (long long)nz * (j0 + r + (long long)nx * k)] : 0.0f;
    }
    {
        // element e = tid + 256 it is (z, x, y), advanced without divisions
        constexpr int kStep = kUpdZ * kUpdY, kDz = kStep % TZ, kDx = kStep / TZ;
        static_assert(kDx + 1 <= TX, "one carry into y per step");
        const long long row = nz, plane = (long long)nx * nz;
        const bool inside = i0 >= H && i0 + kUpdZ + H <= nz && j0 >= H && j0 + kUpdX + H <= nx && k0 >= H &&
                            k0 + kUpdY + H <= ny;
        int z = tid % TZ, x = tid / TZ % TX, y = tid / (TZ * TX);
        const float *src = dm + (i0 - H + z) + row * (j0 - H + x) + plane * (k0 - H + y);
        unsigned dst = (unsigned)__cvta_generic_to_shared(&tile[0][0][0] + tid);
        for (int e = tid; e < TZ * TX * TY; e += kStep, dst += kStep * sizeof(float)) {
            const int zi = i0 - H + z, xj = j0 - H + x, yk = k0 - H + y;
            const bool in = inside || (zi >= 0 && zi < nz && xj >= 0 && xj < nx && yk >= 0 && yk < ny);
            // 4-byte asynchronous copy (0 bytes read: the cell is filled with zero)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(in ? src : dm), "r"(in ? 4 : 0)
                         : "memory");
            z += kDz;
            x += kDx;
            src += kDz + kDx * row;
            if (z >= TZ) {
                z -= TZ;
                x++;
                src += row - TZ;
            }
            if (x >= TX) {
                x -= TX;
                y++;
                src += plane - TX * row;
            }
        }
    }
    if (S > 1)
        for (int e = tid; e < S * S * S; e += kUpdZ * kUpdY) weights[e] = __ldg(kernel + e);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float acc[kUpdX];
#pragma unroll
    for (int r = 0; r < kUpdX; r++) acc[r] = 0.0f;
    if (S > 1) {
#pragma unroll 1
        for (int yk = 0; yk < S; yk++) {
            float w[S * S];
#pragma unroll
            for (int e = 0; e < S * S; e++) w[e] = weights[yk * S * S + e];
#pragma unroll
            for (int x = 0; x < kUpdX + S - 1; x++) {
                float v[S];
#pragma unroll
                for (int zk = 0; zk < S; zk++) v[zk] = tile[ty + yk][x][tz + zk];
#pragma unroll
                for (int r = 0; r < kUpdX; r++) {
                    if (x - r < 0 || x - r >= S) continue;
#pragma unroll
                    for (int zk = 0; zk < S; zk++) acc[r] = fadd(acc[r], fmul(v[zk], w[(x - r) * S + zk]));
                }
            }
        }
    }
    if (i >= nz || k >= ny) return;
    const bool in_zy = i >= m.i_lo && i < nz - m.i_hi_off && k >= m.k_lo && k < ny - m.k_hi_off_upd;
    const bool inner_zy = k >= H && k < ny - H && i >= H && i < nz - H;
    const int gbz = nzz / kBrick, gbx = nxx / kBrick;
    static_assert(kUpdX % kBrick == 0, "a thread's nodes start on a brick");
    float *brick = bricks + ((i >> 2) + (long long)gbz * ((j0 >> 2) + (long long)gbx * (k >> 2))) * kBrickNodes +
                   (i & 3) + 16 * (k & 3);
    const long long at = i + (long long)nz * (j0 + (long long)nx * k);
    const bool face_zy = i == nz - 1 || k == ny - 1;
#pragma unroll
    for (int r = 0; r < kUpdX; r++) {
        const int j = j0 + r;
        if (j >= nx) break;
        if (in_zy && j >= m.j_lo && j < nx - m.j_hi_off_upd) {
            // the filter leaves the nodes without a full neighbourhood as they are
            const float d = S > 1 && inner_zy && j >= H && j < nx - H ? acc[r] : tile[ty + H][r + H][tz + H];
            s[r] = fadd(s[r], d);
            slowness[at + (long long)nz * r] = s[r];
            brick[(long long)gbz * kBrickNodes * (r >> 2) + 4 * (r & 3)] = s[r];
            if (face_zy || j == nx - 1)  // a node on a far face is repeated into the padding
                for (int y = k; y < (k == ny - 1 ? nyy : k + 1); y++)
                    for (int x = j; x < (j == nx - 1 ? nxx : j + 1); x++)
                        for (int z = i; z < (i == nz - 1 ? nzz : i + 1); z++)
                            bricks[((z >> 2) + (long long)gbz * ((x >> 2) + (long long)gbx * (y >> 2))) * kBrickNodes +
                                   (z & 3) + 4 * (x & 3) + 16 * (y & 3)] = s[r];
        }
        if (velocity) velocity[at + (long long)nz * r] = fdiv(1.0f, s[r]);
    }
}

// B = [dobs - dcal ; 0] (B may be nullptr) and the FP64 partial sums of ||dobs - dcal||^2, one
// per block; k_norm_sum adds them.  Elements go to threads and partials to the sum in a fixed
// order.  (160,000 picks: 4 us; one block took 84 us for the norm alone.)
__global__ void __launch_bounds__(256) k_residual(const float *dobs, const float *dcal, float *B, int n, int n_total,
                                                  double *partials)
{
    __shared__ double sh[8];
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_total; i += gridDim.x * blockDim.x) {
        const float o = i < n ? dobs[i] : 0.0f, c = i < n ? dcal[i] : 0.0f;
        if (B) B[i] = fsub(o, c);
        const double d = (double)o - (double)c;
        acc += d * d;
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; w++) t += sh[w];
        partials[blockIdx.x] = t;
    }
}

__global__ void k_norm_sum(const double *partials, double *out)
{
    double acc = 0.0;
    for (int i = threadIdx.x; i < kNormBlocks; i += 32) acc += partials[i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if (threadIdx.x == 0) *out = acc;
}

cudaError_t model_dm(const float *xdm, float *dm, int nx, int ny, int nz, float dx, float dy, float dz, float dxt,
                     float dyt, float dzt, int nxt, int nyt, int nzt, UpdateMasks m, cudaStream_t st)
{
    const long long blocks = ((long long)nz * ny + 255) / 256;
    const int runs = (nx + kDmRun - 1) / kDmRun;
    if (blocks >= (1LL << 31)) return cudaErrorInvalidValue;
    k_model_dm<<<dim3((unsigned)blocks, (unsigned)(runs < 65535 ? runs : 65535)), 256, 0, st>>>(
        xdm, dm, nx, ny, nz, dx, dy, dz, dxt, dyt, dzt, nxt, nyt, nzt, m);
    return cudaGetLastError();
}

bool update_fuses(int samples) { return samples <= kMaxFused; }

cudaError_t gaussian_smooth(const float *in, float *out, int nx, int ny, int nz, int samples, const float *kernel,
                            cudaStream_t st)
{
    k_gaussian<<<grid_for((long long)nx * ny * nz, 256), 256, 0, st>>>(in, out, nx, ny, nz, samples, kernel);
    return cudaGetLastError();
}

cudaError_t model_update(const float *dm, float *slowness, float *bricks, float *velocity, int samples,
                         const float *kernel, int nx, int ny, int nz, int nxx, int nyy, int nzz, UpdateMasks m,
                         cudaStream_t st)
{
    const long long tiles = (long long)((nz + kUpdZ - 1) / kUpdZ) * ((nx + kUpdX - 1) / kUpdX) *
                            ((ny + kUpdY - 1) / kUpdY);
    if (tiles >= (1LL << 31)) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)tiles), block(kUpdZ, kUpdY);
    switch (samples) {
    case 1: k_model_update<1><<<grid, block, 0, st>>>(dm, slowness, bricks, velocity, kernel, nx, ny, nz, nxx, nyy, nzz, m); break;
    case 3: k_model_update<3><<<grid, block, 0, st>>>(dm, slowness, bricks, velocity, kernel, nx, ny, nz, nxx, nyy, nzz, m); break;
    case 5: k_model_update<5><<<grid, block, 0, st>>>(dm, slowness, bricks, velocity, kernel, nx, ny, nz, nxx, nyy, nzz, m); break;
    case 7: k_model_update<7><<<grid, block, 0, st>>>(dm, slowness, bricks, velocity, kernel, nx, ny, nz, nxx, nyy, nzz, m); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t data_residual(const float *dobs, const float *dcal, float *B, int n, int n_total, double *norm2,
                          cudaStream_t st)
{
    k_residual<<<kNormBlocks, 256, 0, st>>>(dobs, dcal, B, n, n_total, norm2 + 1);
    k_norm_sum<<<1, 32, 0, st>>>(norm2 + 1, norm2);
    return cudaGetLastError();
}

}  // namespace tomo
