// Shared device helpers for the tomography kernels (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace tomo {

constexpr float kInf = 1e6f;  // "not reached" value (src/eikonal/block_FIM/cuda_kernel.cuh:7)
constexpr unsigned kFull = 0xffffffffu;

// Device-side error word values (ctrl[kErr]).
enum DevErr : unsigned {
    kDevOk = 0,
    kDevBarrierTimeout = 1,
    kDevRoundCap = 2,
    kDevCapacity = 3,
};

// Control-block layout shared by the persistent kernels.
enum CtrlSlot : int {
    kCnt0 = 0, kCnt1 = 1, kCnt2 = 2,  // work-list counters (3-way rotation)
    kBarCount = 3, kBarGen = 4,       // grid barrier
    kErr = 5,                         // DevErr
    kRounds = 6,                      // rounds run (written by block 0)
    kCur0 = 7, kCur1 = 8, kCur2 = 9,  // per-round fetch cursors (3-way rotation)
    kCtrlWords = 16,
};

// Division by a divisor known in advance: with z = RN(1 / y), q = RN(a z), r = a - q y (exact)
// and RN(q + r z), the IEEE quotient in three operations (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990; Brisebarre, Muller and Raina,
// "Accelerating correctly rounded floating-point division when the divisor is known in
// advance", 2004).  q + r z is within 3 x 2^-25 ulp of a / y, so only quotients that near a
// midpoint could round the other way; tests/test_divide_cpu.py goes through all of them, for
// every divisor.  Valid for y in [kDivMin, kDivMax] and a = 0 (the sign of a zero quotient
// may differ) or 2^-80 <= |a| <= 2^80; other a give a quotient that is not correctly rounded
// (|a| smaller) or NaN (infinite a).
constexpr float kDivMin = 0x1p-40f, kDivMax = 0x1p40f;

struct Divisor {
    float y, z;
};

// On the host (IEEE division rounds to nearest).
inline Divisor prepare_divisor(float y) { return Divisor{y, 1.0f / y}; }

#ifdef __CUDACC__
__device__ __forceinline__ unsigned ld_volatile(const unsigned *p)
{
    return *reinterpret_cast<const volatile unsigned *>(p);
}

// Software grid barrier for a cooperatively launched (co-resident) grid.  The wait is
// bounded: after `spin_limit` polls it records kDevBarrierTimeout and returns false, so a
// lost block can never hang the GPU.  Returns false if any block recorded an error; every
// thread of a block gets the same answer (thread 0's read of the error word), so a block
// never splits over an error raised while it passes the barrier.
__device__ __forceinline__ bool grid_barrier(unsigned *ctrl, unsigned long long spin_limit)
{
    __shared__ unsigned err;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned nblocks = gridDim.x * gridDim.y * gridDim.z;
        const unsigned gen = ld_volatile(ctrl + kBarGen);
        __threadfence();
        const unsigned arrived = atomicAdd(ctrl + kBarCount, 1u);
        if (arrived == nblocks - 1) {
            atomicExch(ctrl + kBarCount, 0u);
            __threadfence();
            atomicAdd(ctrl + kBarGen, 1u);
        } else {
            unsigned long long spins = 0;
            while (ld_volatile(ctrl + kBarGen) == gen) {
                if (++spins > spin_limit) {
                    atomicCAS(ctrl + kErr, 0u, (unsigned)kDevBarrierTimeout);
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        err = ld_volatile(ctrl + kErr);
    }
    __syncthreads();
    return err == 0u;
}

// Grid-wide barrier on a monotone arrival counter: the k-th barrier of a launch (k = epoch,
// counted by every block) completes when ctrl[kBarCount] reaches (k + 1) * blocks.  There is
// no reset and no generation word, so the last block to arrive does no extra atomics.  The
// counter starts at 0 for the launch; the waits are bounded as in grid_barrier.
__device__ __forceinline__ bool grid_sync(unsigned *ctrl, unsigned &epoch, unsigned long long spin_limit)
{
    __shared__ unsigned err;  // the error word as thread 0 read it: one answer for the block
    __syncthreads();
    ++epoch;
    if (threadIdx.x == 0) {
        const unsigned target = epoch * (gridDim.x * gridDim.y * gridDim.z);
        __threadfence();
        atomicAdd(ctrl + kBarCount, 1u);
        unsigned long long spins = 0;
        while (ld_volatile(ctrl + kBarCount) < target) {
            if (++spins > spin_limit) {
                atomicCAS(ctrl + kErr, 0u, (unsigned)kDevBarrierTimeout);
                break;
            }
            __nanosleep(32);
        }
        __threadfence();
        err = ld_volatile(ctrl + kErr);
    }
    __syncthreads();
    return err == 0u;
}

// IEEE FP32 arithmetic that the compiler may not contract into FMAs: used wherever the
// reference's FP32 operation order is restated bit for bit.
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }

// The prepared division above.
__device__ __forceinline__ Divisor divisor(float y) { return Divisor{y, __frcp_rn(y)}; }

__device__ __forceinline__ float fdiv(float a, const Divisor &d)
{
    const float q = __fmul_rn(a, d.z);
    return __fmaf_rn(__fmaf_rn(-q, d.y, a), d.z, q);
}

// Square root: the hardware's reciprocal root r gives g = a r and h = r / 2, and one step with
// the exact residual a - g g corrects g (Markstein 1990): five operations, the IEEE root for
// every a in [2^-102, 2^126) (tests/test_sqrt_gpu.py goes through all of them) and NaN below
// zero.  Below 2^-102 it can be an ulp off, for subnormal a (whose reciprocal root is flushed to
// infinity) and infinite a it is NaN, and a = 0 is set apart.  Callers keep a in the range.
__device__ __forceinline__ float fsqrt(float a)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    const float g = __fmul_rn(a, r), h = __fmul_rn(0.5f, r);
    const float s = __fmaf_rn(__fmaf_rn(-g, g, a), h, g);
    return a == 0.0f ? a : s;
}

// trilinear (src/utils/interpolation/trilinear.cpp:3-20), same operation order, from the
// weights of the upper corners.
__device__ __forceinline__ float trilinear_weights(float c000, float c001, float c100, float c101, float c010,
                                                   float c011, float c110, float c111, float xd, float yd, float zd)
{
    const float c00 = fadd(fmul(c000, fsub(1.0f, xd)), fmul(c100, xd));
    const float c01 = fadd(fmul(c001, fsub(1.0f, xd)), fmul(c101, xd));
    const float c10 = fadd(fmul(c010, fsub(1.0f, xd)), fmul(c110, xd));
    const float c11 = fadd(fmul(c011, fsub(1.0f, xd)), fmul(c111, xd));
    const float c0 = fadd(fmul(c00, fsub(1.0f, yd)), fmul(c10, yd));
    const float c1 = fadd(fmul(c01, fsub(1.0f, yd)), fmul(c11, yd));
    return fadd(fmul(c0, fsub(1.0f, zd)), fmul(c1, zd));
}

// The same from the corners' coordinates.
__device__ __forceinline__ float trilinear_ref(float c000, float c001, float c100, float c101,
                                               float c010, float c011, float c110, float c111,
                                               float x0, float x1, float y0, float y1, float z0,
                                               float z1, float x, float y, float z)
{
    const float xd = fdiv(fsub(x, x0), fsub(x1, x0));
    const float yd = fdiv(fsub(y, y0), fsub(y1, y0));
    const float zd = fdiv(fsub(z, z0), fsub(z1, z0));
    return trilinear_weights(c000, c001, c100, c101, c010, c011, c110, c111, xd, yd, zd);
}

#endif  // __CUDACC__

}  // namespace tomo
