// FP64 matrix instruction and asynchronous copies shared by the FP64 GEMM
// kernels.  mma.sync m8n8k4 on FP64 reaches 36.8 of the card's 37 TFLOP/s from
// one warp per scheduler, where register-tiled FMAs need 32 warps an SM for
// 34.8: the operands of one instruction are two registers a thread, so a
// warp's tile needs few shared-memory reads and small tiles lose nothing.
#pragma once
#include <cstdint>

namespace gpx {

// D += A B, A 8 x 4 (lane holds row lane / 4, column lane % 4), B 4 x 8 (row
// lane % 4, column lane / 4), D 8 x 8 (row lane / 4, columns 2 (lane % 4) + {0, 1}).
// The result has the bits of fma(a3, b3, fma(a2, b2, fma(a1, b1, fma(a0, b0, d))))
// (1,280,000 random products compared), so a contraction issued in ascending
// order equals a scalar loop's.
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// 16 bytes global -> shared; zero-filled where !valid (src must still be a
// readable address).
__device__ __forceinline__ void cp_async_16(void* dst, const void* src, bool valid) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_fence() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_for() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Right-hand sides are cut into chunks of a multiple of 8 columns, at most
// `most`, of nearly equal width: R = 12 runs 16 columns, R = 40 runs 40, R = 96
// runs two chunks of 48, where a fixed 64-column tile would compute 64, 64 and 128.
inline int rhs_chunk(int R, int most) {
    const int chunks = (R + most - 1) / most;
    return ((R + chunks - 1) / chunks + 7) & ~7;
}

}  // namespace gpx
