// Weight-streaming GEMM for row groups of few rows each (the experts of a mixture-of-experts layer at decode batch sizes):
//
//   C[m, n] = sum_k A[m, k] * B[g(m), n, k]       [epilogue as for the tiled kernels, gated activation and NVFP4 result included]
//
// The problem is bound by reading every group's weight once from HBM.  The tiled kernels pad a group's rows to 128 or 256,
// so their tensor-core time is that of a full batch and they read the weight at 4.6 TB/s; here the operand roles are swapped
// as in gemm_decode.cu: 128 weight rows (output columns) are the M side of tcgen05.mma and TOK = 32 or 64 of the group's
// rows the N side, which leaves the tensor core mostly idle and the ring of TMA loads (7-8 stages of 16 KB of weight) to set
// the pace.  There are usually more (group, column tile) pairs than SMs, so K is not cut: a CTA takes whole tiles, round robin,
// and its ring runs on from one tile into the next (with fewer pairs it is still ahead of the tiled kernels: 8 groups of 512
// columns, K = 4096, 8 rows each, call with quantiser, NVFP4 23 / 31 us, BF16 26 / 28 us).  64 experts of 3072 x 4096 NVFP4, eight rows each: 77 us = 5.9 TB/s of weight
// and scales (98 us, 4.6 TB/s, on the tiled kernel).  A group with more than TOK rows is several items on the same weight tile,
// neighbours in the order, so that all but the first find it in the L2.
//
// Roles per CTA (192 threads): warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 epilogue.  Group-scaled FP8 promotes every
// K group through registers (promote_run).  Every mbarrier
// wait is bounded.
#include <cuda_bf16.h>
#include <stdlib.h>

#include "gemm.cuh"
#include "gemm_decode.cuh"
#include "gemm_epilogue.cuh"
#include "gemm_tiles.cuh"
#include "ptx.cuh"

namespace dsl {
namespace dg {

constexpr int SFW_COL = 256;      // weight scale factors (the M side)
constexpr int SFX_COL = 272;      // activation scale factors (the N side)

template <int KIND, int TOK>
struct Cfg {
    static constexpr int W_STAGE = 128 * STAGE_KB;
    static constexpr int X_STAGE = TOK * STAGE_KB;
    static constexpr int SF_ATOMS = KIND == KIND_NVF4 ? 4 : (KIND == KIND_MXF4 ? 2 : 0);
    static constexpr int SF_STAGE = SF_ATOMS * 512;
    static constexpr int STAGE_BYTES = W_STAGE + X_STAGE + 2 * SF_STAGE;
    static constexpr int NUM_STAGES = 200 * 1024 / STAGE_BYTES > 8 ? 8 : 200 * 1024 / STAGE_BYTES;
    static constexpr int TURN_BYTES = 32 * 33 * 4;                       // per epilogue warp: 32 tokens x 32 columns, turned round
    static constexpr int ACC_BUFS = KIND == KIND_F8G ? 512 / TOK > 8 ? 8 : 512 / TOK : 2;
    static constexpr int OFF_W = 0;
    static constexpr int OFF_X = OFF_W + NUM_STAGES * W_STAGE;
    static constexpr int OFF_SFW = OFF_X + NUM_STAGES * X_STAGE;
    static constexpr int OFF_SFX = OFF_SFW + NUM_STAGES * SF_STAGE;
    static constexpr int OFF_BAR = OFF_SFX + NUM_STAGES * SF_STAGE;
    static constexpr int NUM_BARS = 2 * NUM_STAGES + 2 * ACC_BUFS;
    static constexpr int OFF_MISC = OFF_BAR + NUM_BARS * 8;
    static constexpr int OFF_TABLE = OFF_MISC + 16;                      // offs, first token block, first 128-row scale tile
    static constexpr int OFF_TSCALE = (OFF_TABLE + 3 * (DSL_MAX_GROUPS + 1) * 4 + 15) / 16 * 16;
    static constexpr int OFF_TURN = OFF_TSCALE + (KIND == KIND_F8G ? 4 * 2 * TOK * 4 : 0);
    static constexpr int SMEM_BYTES = OFF_TURN + 4 * TURN_BYTES + 1024;
    static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB shared-memory limit");
    static_assert(SMEM_BYTES > 116224, "two CTAs could share an SM and deadlock on tensor-memory allocation");
    static_assert(SF_ATOMS == 0 || TOK == 64, "items of block-scaled kinds must start at an even scale-factor column");
    static_assert(KIND == KIND_F8G || ACC_BUFS * TOK <= SFW_COL, "accumulators overlap the scale-factor columns");
};

struct Item {
    int group, tile, row0, rows, sf_tile, sf_col;   // sf_col: 32-row quarter of the scale tile the tokens start in
};

struct Walk {
    const int* offs;
    const int* blk0;
    const int* sft0;
    int groups, n_tiles, tok;
    __device__ __forceinline__ int total() const { return blk0[groups] * n_tiles; }
    __device__ __forceinline__ Item decode(int item) const {
        const int q = item / n_tiles;
        int lo = 0, hi = groups;        // last g with blk0[g] <= q: the group whose blocks contain q
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (blk0[mid] <= q) lo = mid; else hi = mid;
        }
        const int local = item - blk0[lo] * n_tiles;
        const int blocks = blk0[lo + 1] - blk0[lo];
        Item it;
        it.group = lo;
        it.tile = local / blocks;
        const int r = (local - it.tile * blocks) * tok;      // first row inside the group
        it.row0 = offs[lo] + r;
        it.rows = min(tok, offs[lo + 1] - it.row0);
        it.sf_tile = sft0[lo] + (r >> 7);
        it.sf_col = (r >> 5) & 3;
        return it;
    }
};

}  // namespace dg

template <int KIND, int TOK>
__global__ void __launch_bounds__(192, 1)
gemm_decode_grouped_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const GemmArgs args) {
    using C = dg::Cfg<KIND, TOK>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
    uint64_t* empty_bar = full_bar + C::NUM_STAGES;
    uint64_t* acc_full = empty_bar + C::NUM_STAGES;
    uint64_t* acc_empty = acc_full + C::ACC_BUFS;
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(smem + C::OFF_MISC);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + C::OFF_MISC + 4);
    int* s_offs = reinterpret_cast<int*>(smem + C::OFF_TABLE);
    int* s_blk0 = s_offs + (DSL_MAX_GROUPS + 1);
    int* s_sft0 = s_blk0 + (DSL_MAX_GROUPS + 1);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int groups = args.num_groups;

    if (threadIdx.x == 0) {
        for (int i = 0; i < C::NUM_STAGES; ++i) { mbar_init(full_bar + i, 1); mbar_init(empty_bar + i, 1); }
        for (int i = 0; i < C::ACC_BUFS; ++i) { mbar_init(acc_full + i, 1); mbar_init(acc_empty + i, 4); }
        *abort_flag = 0;
        fence_mbar_init();
        prefetch_tmap(&tmap_w);
        prefetch_tmap(&tmap_x);
    }
    if (C::SF_ATOMS > 0) {   // never let an uninitialised (possibly NaN) scale byte meet zero-filled data
        uint32_t* z = reinterpret_cast<uint32_t*>(smem + C::OFF_SFW);
        for (int i = threadIdx.x; i < C::NUM_STAGES * 2 * C::SF_STAGE / 4; i += blockDim.x) z[i] = 0u;
        fence_proxy_async_smem();
    }
    if (warp == 1) tmem_alloc(tmem_ptr, TMEM_COLS);
    // Everything above touches no global memory and may overlap the tail of the preceding kernel of the stream.  A successor
    // that opted in may be placed on an SM as soon as this kernel's CTA leaves it; it is let go only after the wait, because it
    // may fetch a weight that was complete before this kernel started (dsl_epilogue.b_is_static).
    griddep_wait();
    griddep_launch_dependents();
    load_group_offsets(s_offs, args.group_offsets, groups, args.m_total);
    __syncthreads();
    if (warp == 2) {   // tables, 32 groups at a time: running maximum (monotone offsets), then running sums of the blocks
        int high = s_offs[0], blocks = 0, tiles = 0;
        if (lane == 0) { s_blk0[0] = 0; s_sft0[0] = 0; }
        for (int g0 = 0; g0 < groups; g0 += 32) {
            const int g = g0 + lane;
            int end = g < groups ? s_offs[g + 1] : 0;
            end = max(end, high);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xFFFFFFFFu, end, o);
                if (lane >= o) end = max(end, v);
            }
            int begin = __shfl_up_sync(0xFFFFFFFFu, end, 1);
            if (lane == 0) begin = high;
            const int rows = g < groups ? end - begin : 0;
            int b = (rows + TOK - 1) / TOK, t = (rows + 127) / 128;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int vb = __shfl_up_sync(0xFFFFFFFFu, b, o), vt = __shfl_up_sync(0xFFFFFFFFu, t, o);
                if (lane >= o) { b += vb; t += vt; }
            }
            if (g < groups) {
                s_offs[g + 1] = end;
                s_blk0[g + 1] = blocks + b;
                s_sft0[g + 1] = tiles + t;
            }
            high = __shfl_sync(0xFFFFFFFFu, end, 31);
            blocks += __shfl_sync(0xFFFFFFFFu, b, 31);
            tiles += __shfl_sync(0xFFFFFFFFu, t, 31);
            __syncwarp();
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr;

    dg::Walk walk;
    walk.offs = s_offs;
    walk.blk0 = s_blk0;
    walk.sft0 = s_sft0;
    walk.groups = groups;
    walk.n_tiles = (args.n + 127) / 128;
    walk.tok = TOK;
    const int total = walk.total();
    const int S = (args.k_bytes + STAGE_KB - 1) / STAGE_KB;
    const int step_items = static_cast<int>(gridDim.x);

    if (warp == 0) {
        // ================= TMA producer =================
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < total && ok; t += step_items) {
                const dg::Item it = walk.decode(t);
                const size_t w_tile = static_cast<size_t>(it.group) * args.sfb_tiles_per_group + it.tile;
                for (int kb = 0; kb < S; ++kb) {
                    if (!mbar_wait(empty_bar + stage, phase ^ 1u, abort_flag, ST_TIMEOUT_PRODUCER)) { ok = false; break; }
                    const int atoms = C::SF_ATOMS > 0 ? min(C::SF_ATOMS, args.sf_katoms - kb * C::SF_ATOMS) : 0;
                    mbar_arrive_expect_tx(full_bar + stage, C::W_STAGE + C::X_STAGE + 2 * atoms * 512);
                    if (C::SF_ATOMS == 0 && args.b_kn) {    // blocks of 128 bytes of N x one stage of K, side by side
                        constexpr int ELEM = KIND == KIND_BF16 ? 2 : 1;
#pragma unroll
                        for (int j = 0; j < ELEM; ++j)
                            tma_load_3d(smem + C::OFF_W + stage * C::W_STAGE + j * (C::W_STAGE / ELEM), &tmap_w, full_bar + stage,
                                        it.tile * 128 * ELEM + j * 128, kb * (STAGE_KB / ELEM), it.group);
                    } else {
                        tma_load_3d(smem + C::OFF_W + stage * C::W_STAGE, &tmap_w, full_bar + stage, kb * STAGE_KB, it.tile * 128, it.group);
                    }
                    tma_load_2d(smem + C::OFF_X + stage * C::X_STAGE, &tmap_x, full_bar + stage, kb * STAGE_KB, it.row0);
                    if (C::SF_ATOMS > 0) {
                        const size_t katom0 = static_cast<size_t>(kb) * C::SF_ATOMS;
                        bulk_load(smem + C::OFF_SFW + stage * C::SF_STAGE, args.sfb + (w_tile * args.sf_katoms + katom0) * 512, atoms * 512,
                                  full_bar + stage);
                        bulk_load(smem + C::OFF_SFX + stage * C::SF_STAGE,
                                  args.sfa + (static_cast<size_t>(it.sf_tile) * args.sf_katoms + katom0) * 512, atoms * 512, full_bar + stage);
                    }
                    if (++stage == C::NUM_STAGES) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        uint32_t idesc = (static_cast<uint32_t>(TOK >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
        if (KIND == KIND_F8 || KIND == KIND_F8G) idesc |= 1u << 4;
        if (KIND == KIND_NVF4) idesc |= (1u << 7) | (1u << 10);
        if (KIND == KIND_MXF4) idesc |= (1u << 7) | (1u << 10) | (1u << 23);
        if (KIND == KIND_BF16) idesc |= (1u << 4) | (1u << 7) | (1u << 10);
        // weight given [K, N]: the M side is MN-major (bit 15), 32 bytes of K are 16 / 32 rows of 128 bytes
        const bool w_kn = C::SF_ATOMS == 0 && args.b_kn != 0;
        if (w_kn) idesc |= 1u << 15;
        const uint64_t w_step = w_kn ? (KIND == KIND_BF16 ? 16 * 128 : 32 * 128) >> 4 : 2;
        const uint32_t w_block = w_kn && KIND == KIND_BF16 ? C::W_STAGE / 2 : 0;
        int stage = 0;
        uint32_t phase = 0, step = 0;       // step: accumulator buffers filled so far (per item, or per K group for F8G)
        bool ok = true;
        for (int t = blockIdx.x; t < total && ok; t += step_items) {
            const int sf_col = C::SF_ATOMS > 0 ? walk.decode(t).sf_col : 0;
            for (int kb = 0; kb < S; ++kb) {
                const uint32_t buf = step % C::ACC_BUFS;
                if ((KIND == KIND_F8G || kb == 0) &&
                    !mbar_wait(acc_empty + buf, ((step / C::ACC_BUFS) & 1u) ^ 1u, abort_flag, ST_TIMEOUT_MMA)) { ok = false; break; }
                if (!mbar_wait(full_bar + stage, phase, abort_flag, ST_TIMEOUT_MMA)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * TOK;
                const uint64_t wdesc = make_desc_mn_sw128(smem_u32(smem + C::OFF_W + stage * C::W_STAGE), w_block);
                const uint64_t xdesc = make_desc_sw128(smem_u32(smem + C::OFF_X + stage * C::X_STAGE));
                if (elect_one()) {
                    if (C::SF_ATOMS > 0) {
                        const uint32_t sfw_addr = smem_u32(smem + C::OFF_SFW + stage * C::SF_STAGE);
                        const uint32_t sfx_addr = smem_u32(smem + C::OFF_SFX + stage * C::SF_STAGE);
#pragma unroll
                        for (int i = 0; i < C::SF_ATOMS; ++i) {
                            tc_cp_32x128b_warpx4(tmem_base + dg::SFW_COL + i * 4, make_desc_sf(sfw_addr + i * 512));
                            tc_cp_32x128b_warpx4(tmem_base + dg::SFX_COL + i * 4, make_desc_sf(sfx_addr + i * 512));
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t accum = ((KIND != KIND_F8G && kb > 0) || k > 0) ? 1u : 0u;
                        if (KIND == KIND_F8 || KIND == KIND_F8G) {
                            mma_f8f6f4(d_tmem, wdesc + w_step * k, xdesc + 2 * k, idesc, accum);
                        } else if (KIND == KIND_BF16) {
                            mma_f16(d_tmem, wdesc + w_step * k, xdesc + 2 * k, idesc, accum);
                        } else if (KIND == KIND_NVF4) {
                            mma_nvf4(d_tmem, wdesc + 2 * k, xdesc + 2 * k, idesc, tmem_base + dg::SFW_COL + k * 4,
                                     tmem_base + dg::SFX_COL + k * 4 + sf_col, accum);
                        } else {
                            const uint32_t sf_id = (k & 1) * 2;
                            const uint32_t id = idesc | (sf_id << 29) | (sf_id << 4);
                            mma_mxf4(d_tmem, wdesc + 2 * k, xdesc + 2 * k, id, tmem_base + dg::SFW_COL + (k >> 1) * 4,
                                     tmem_base + dg::SFX_COL + (k >> 1) * 4 + sf_col, accum);
                        }
                    }
                    tc_commit(empty_bar + stage);
                    if (KIND == KIND_F8G || kb == S - 1) tc_commit(acc_full + buf);
                }
                __syncwarp();
                if (KIND == KIND_F8G || kb == S - 1) ++step;
                if (++stage == C::NUM_STAGES) { stage = 0; phase ^= 1u; }
            }
        }
    } else {
        // ================= epilogue =================
        const int quad = warp & 3;
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
        float s1 = args.s1_dev != nullptr ? *args.s1_dev : args.s1;
        float s2 = args.s2_dev != nullptr ? *args.s2_dev : args.s2;
        if (args.scale_product) { s1 = s1 * s2; s2 = 1.0f; }
        const bool vec_ok = args.out_bf16 ? (args.ldc % 8 == 0) : (args.ldc % 4 == 0);
        float* turn = reinterpret_cast<float*>(smem + C::OFF_TURN + (warp - 2) * C::TURN_BYTES);
        const int nb128 = walk.n_tiles;
        uint32_t step = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < total && ok; t += step_items) {
            const dg::Item it = walk.decode(t);
            const int col0 = it.tile * 128 + quad * 32;
            // 32 tokens of this warp's 32 columns lie in `turn`, column by column as the accumulator has them; every lane
            // now takes one token's row of 32 columns, which is the shape the tiled kernels' epilogue works on.  (With the
            // lane as the column, a gated and quantised result costs every lane the arithmetic of the whole block: 32 rows
            // an expert, 64 experts: 355 us a layer, against 207 us for the tiled kernels.)
            auto finish = [&](int first) {
                __syncwarp();
                const int i = first + lane;
                if (i < it.rows && col0 < args.n) {
                    uint32_t v[32];
#pragma unroll
                    for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(turn[lane * 33 + c]);
                    const int row = it.row0 + i;
                    const float rs = args.row_scale != nullptr ? args.row_scale[row] : 1.0f;
                    store_chunk32(args, row, col0, it.group, v, s1, s2, rs, vec_ok, it.sf_tile, (it.sf_col << 5) + i);
                }
                __syncwarp();
            };
            if constexpr (KIND == KIND_F8G) {
                float acc[TOK];
                float* tscale = reinterpret_cast<float*>(smem + C::OFF_TSCALE) + (warp - 2) * 2 * TOK;
                const float* sa = args.gsa + static_cast<size_t>(it.row0) * S;
                ok = args.sb_block
                         ? promote_run<TOK, true, C::ACC_BUFS>(sa, it.rows, args.gsb + (static_cast<size_t>(it.group) * nb128 + it.tile) * S, 0, 0,
                                                               S, 0, S, tmem_lane, acc_full, acc_empty, abort_flag, tscale, lane, step, acc)
                         : promote_run<TOK, false, C::ACC_BUFS>(sa, it.rows,
                                                                args.gsb + static_cast<size_t>(it.group) * S * args.n + min(col0 + lane, args.n - 1),
                                                                args.n, 0, S, 0, S, tmem_lane, acc_full, acc_empty, abort_flag, tscale, lane,
                                                                step, acc);
                if (!ok) break;
#pragma unroll
                for (int c = 0; c < TOK; c += 32) {
                    if (c >= it.rows) break;
#pragma unroll
                    for (int i = 0; i < 32; ++i) turn[i * 33 + lane] = acc[c + i];
                    finish(c);
                }
            } else {
                const uint32_t buf = step % C::ACC_BUFS;
                if (!mbar_wait(acc_full + buf, (step / C::ACC_BUFS) & 1u, abort_flag, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
                ++step;
                __syncwarp();
                tc_fence_after();
#pragma unroll 1
                for (int c = 0; c < it.rows; c += 32) {
                    uint32_t v[32];
                    tmem_ld_32x32b_x32(tmem_lane + buf * TOK + c, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) turn[i * 33 + lane] = __uint_as_float(v[i]);
                    if (c + 32 >= it.rows) {        // everything is out of tensor memory: the next but one item may have it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(acc_empty + buf);
                    }
                    finish(c);
                }
            }
        }
    }

    // ---- common exit -------------------------------------------------------------------
    tc_fence_before();
    __syncthreads();
    const uint32_t aborted = *abort_flag;
    if (aborted != 0) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(2000);
        if (threadIdx.x == 0 && args.status != nullptr) atomicOr(args.status, aborted);
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// ---- host side ---------------------------------------------------------------------------
template <int KIND, int TOK>
static int launch_grouped_one(const void* A, const void* B, const GemmArgs& args, cudaStream_t st) {
    using C = dg::Cfg<KIND, TOK>;
    CUtensorMap tw, tx;
    if (args.b_kn) {
        constexpr int ELEM = KIND == KIND_BF16 ? 2 : 1;
        if (!make_tmap_kn(&tw, B, args.n, args.k_bytes / ELEM, args.num_groups, ELEM, STAGE_KB / ELEM)) return DSL_ERR_DRIVER;
    } else if (!make_tmap_u8(&tw, B, args.k_bytes, args.n, args.num_groups, STAGE_KB, 128)) {
        return DSL_ERR_DRIVER;
    }
    if (!make_tmap_u8(&tx, A, args.k_bytes, args.m_total, 0, STAGE_KB, TOK)) return DSL_ERR_DRIVER;
    static PerDeviceInt attr_set;   // per device; idempotent, a race here only repeats the same call
    const int dev = current_device_slot();
    if (dev < 0) return static_cast<int>(cudaErrorInvalidDevice);
    if (attr_set.v[dev].load(std::memory_order_acquire) == 0) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_decode_grouped_kernel<KIND, TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
        if (e != cudaSuccess) return static_cast<int>(e);
        attr_set.v[dev].store(1, std::memory_order_release);
    }
    const long long n_tiles = (args.n + 127) / 128;
    const long long max_groups = args.m_total < args.num_groups ? args.m_total : args.num_groups;      // groups that can have rows
    const long long max_items = ((args.m_total + TOK - 1) / TOK + max_groups) * n_tiles;
    const long long grid = max_items < sm_count() ? max_items : sm_count();
    static const bool pdl = [] { const char* e = getenv("DSLGEMM_PDL"); return !(e != nullptr && e[0] == '0'); }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(192);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return static_cast<int>(cudaLaunchKernelEx(&cfg, gemm_decode_grouped_kernel<KIND, TOK>, tw, tx, args));
}

template <int KIND>
static int launch_grouped_kind(const void* A, const void* B, const GemmArgs& args, cudaStream_t st) {
    // TOK at least twice the mean row count, so that few groups need a second pass over their weight.  FP4 kinds always take
    // 64: an item of 32 could start in an odd quarter of its scale tile, and the scale-factor column of the N side has to
    // be even.
    if constexpr (KIND != KIND_NVF4 && KIND != KIND_MXF4) {
        if (static_cast<long long>(args.m_total) <= 16ll * args.num_groups) return launch_grouped_one<KIND, 32>(A, B, args, st);
    }
    return launch_grouped_one<KIND, 64>(A, B, args, st);
}

// Mean rows a group up to which this kernel serves.  Whole layer, 64 experts, top 8, K = D = 4096, H = 1536, against the
// tiled kernels (us):      8 rows       16 rows      25 rows      32 rows
//   NVFP4              158 / 194    166 / 201    174 / 208    175 / 208
//   FP8 128x128 blocks 237 / 304    242 / 338    279 / 551    297 / 609
//   FP8 per tensor     243 / 285    249 / 293    261 / 301    267 / 343
//   BF16               418 / 489    442 / 508    445 / 519    431 / 660
// and with one row for each of eight experts 72 / 76, 79 / 92, 87 / 99, 99 / 136.
// The sizes of the groups are on the device, so the rule sees their mean only.  Skewed groups, the gate/up GEMM of that layer
// (64 groups, N = 3072, K = 4096, quantiser included, L2 cold; this kernel / the tiled kernels, us):
//                       512 rows:  even       all in 8   all in 1 | 2048 rows: even     half in 1  0.9 in 1   all in 8  all in 1
//   NVFP4                        111 / 122   41 / 49    38 / 42   |          123 / 136  134 / 140  145 / 142  76 / 66   76 / 62
//   FP8 128x128 blocks           149 / 230   44 / 54    42 / 34   |          173 / 239  194 / 245  224 / 249 114 / 60  112 / 56
//   FP8 per tensor               154 / 172   49 / 53    45 / 37   |          170 / 187  181 / 193  197 / 193  88 / 73   86 / 67
//   BF16                         267 / 308   65 / 73    58 / 36   |          273 / 321  300 / 329  331 / 323 114 / 79  112 / 60
// While the weights of most groups are read this kernel is ahead or even; it falls behind, to half the speed, only where nearly
// all rows sit in a few groups, whose weight the taller tiles of the other kernels read fewer times.
constexpr int kGroupedMeanRows = 32;

bool decode_grouped_served(const GemmArgs& args) {
    if (args.group_offsets == nullptr || (args.out_sf != nullptr && args.act == DSL_ACT_NONE)) return false;
    if (static_cast<long long>(args.m_total) > static_cast<long long>(kGroupedMeanRows) * args.num_groups) return false;
    const long long items = ((args.m_total + 31) / 32 + static_cast<long long>(args.num_groups)) * ((args.n + 127) / 128);
    return items <= (1ll << 30);                            // item counters in the kernel are 32-bit
}

int launch_gemm_decode_grouped(int kind, const void* A, const void* B, const GemmArgs& args, cudaStream_t st) {
    if (!decode_grouped_served(args)) return DSL_NOT_SERVED;
    switch (kind) {
        case KIND_F8: return launch_grouped_kind<KIND_F8>(A, B, args, st);
        case KIND_NVF4: return launch_grouped_kind<KIND_NVF4>(A, B, args, st);
        case KIND_MXF4: return launch_grouped_kind<KIND_MXF4>(A, B, args, st);
        case KIND_BF16: return launch_grouped_kind<KIND_BF16>(A, B, args, st);
        case KIND_F8G: return launch_grouped_kind<KIND_F8G>(A, B, args, st);
        default: return DSL_ERR_ENUM;
    }
}

}  // namespace dsl
