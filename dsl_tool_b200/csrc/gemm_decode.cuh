// Device code shared by the weight-streaming kernels (gemm_decode.cu: one row group, gemm_decode_grouped.cu: row groups).
#pragma once
#include "gemm.cuh"
#include "ptx.cuh"

namespace dsl {

// Two accumulators (adjacent tokens) += partial product * scale: fma.rn.f32x2 is two IEEE fused multiply-adds.
__device__ __forceinline__ void dec_fma2(float& a0, float& a1, float p0, float p1, unsigned long long s2) {
    unsigned long long a, p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(a0), "f"(a1));
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(p0), "f"(p1));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(p), "l"(s2));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(a));
}

// Group-scaled FP8: one run (K groups [kb0, kb0 + len) of `tile`, one shared-memory stage each) into registers.
// This thread's lane of tensor memory is one weight row, i.e. one output column; acc[t] belongs to token t.  Per group
// acc = p * (sa * sb) + acc for block scales, acc = (p * sa) * sb + acc for per-column ones - the operations of the
// tiled kernels, in the order the producer visits the groups.  The activation scales of the TOK tokens are fetched
// DEPTH groups ahead (one token per lane) and handed round through a small per-warp buffer.
// `sa`: activation scales of the run's first token ([rows][S]; rows beyond are computed and never stored); `sb`: with block
// scales the S values of this column tile, else this thread's column of the [S][n] array.
template <int TOK, bool SB_BLOCK, int BUFS>
__device__ __forceinline__ bool promote_run(const float* __restrict__ sa_rows, int rows, const float* __restrict__ sb_ptr, int sb_pitch,
                                            int kb0, int len, int rot, int S, uint32_t tmem_lane, uint64_t* acc_full, uint64_t* acc_empty,
                                            volatile uint32_t* abort_flag, float* tscale, int lane, uint32_t& step, float (&acc)[TOK]) {
    constexpr int J = (TOK + 31) / 32;
    constexpr int DEPTH = TOK > 64 ? 2 : 4;
    float sa_q[DEPTH][J], sb_q[DEPTH];
    __syncwarp();       // `tscale` restarts at its first buffer: the last reads of the run before (any length) are behind every lane
    auto fetch = [&](int i, float (&sa)[J], float& sb) {
        int kb = i + rot;
        if (kb >= len) kb -= len;
        kb += kb0;
        sb = __ldg(SB_BLOCK ? sb_ptr + kb : sb_ptr + static_cast<size_t>(kb) * sb_pitch);
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int t = min(lane + 32 * j, rows - 1);
            sa[j] = __ldg(sa_rows + static_cast<size_t>(t) * S + kb);
        }
    };
#pragma unroll
    for (int t = 0; t < TOK; ++t) acc[t] = 0.f;
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) fetch(min(d, len - 1), sa_q[d], sb_q[d]);
#pragma unroll 1
    for (int i = 0; i < len; ++i, ++step) {
        float* ts = tscale + (i & 1) * TOK;
        const float sb = sb_q[0];
#pragma unroll
        for (int j = 0; j < J; ++j)
            if (TOK >= 32 || lane < TOK) ts[lane + 32 * j] = SB_BLOCK ? __fmul_rn(sa_q[0][j], sb) : sa_q[0][j];
#pragma unroll
        for (int d = 0; d + 1 < DEPTH; ++d) {
            sb_q[d] = sb_q[d + 1];
#pragma unroll
            for (int j = 0; j < J; ++j) sa_q[d][j] = sa_q[d + 1][j];
        }
        fetch(min(i + DEPTH, len - 1), sa_q[DEPTH - 1], sb_q[DEPTH - 1]);
        const uint32_t buf = step % BUFS;
        if (!mbar_wait(acc_full + buf, (step / BUFS) & 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) return false;
        __syncwarp();
        tc_fence_after();
        uint32_t v[2][16];
        tmem_ld_32x32b_x16(tmem_lane + buf * TOK, v[0]);
#pragma unroll
        for (int c = 0; c < TOK / 16; ++c) {
            tmem_ld_wait();
            if (c + 1 < TOK / 16) {
                tmem_ld_32x32b_x16(tmem_lane + buf * TOK + (c + 1) * 16, v[(c + 1) & 1]);
            } else {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty + buf);
            }
            const ulonglong2* s4 = reinterpret_cast<const ulonglong2*>(ts + c * 16);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const ulonglong2 s = s4[q];
                float* a = acc + c * 16 + q * 4;
                const uint32_t* p = v[c & 1] + q * 4;
                if (SB_BLOCK) {
                    dec_fma2(a[0], a[1], __uint_as_float(p[0]), __uint_as_float(p[1]), s.x);
                    dec_fma2(a[2], a[3], __uint_as_float(p[2]), __uint_as_float(p[3]), s.y);
                } else {
                    const float4 f = *reinterpret_cast<const float4*>(&s4[q]);
                    a[0] = fmaf(__fmul_rn(__uint_as_float(p[0]), f.x), sb, a[0]);
                    a[1] = fmaf(__fmul_rn(__uint_as_float(p[1]), f.y), sb, a[1]);
                    a[2] = fmaf(__fmul_rn(__uint_as_float(p[2]), f.z), sb, a[2]);
                    a[3] = fmaf(__fmul_rn(__uint_as_float(p[3]), f.w), sb, a[3]);
                }
            }
        }
    }
    return true;
}

}  // namespace dsl
