// dsl_moe_layer: the whole mixture-of-experts feed-forward layer of a GPU that holds every expert, in ONE call of the
// C ABI.  The layer is a chain of a dozen short launches around two grouped GEMMs; issued from the host language one by
// one, with a tensor allocated for every intermediate, the host takes longer than the GPU for anything up to about a
// thousand tokens (64 tokens, NVFP4: 313 us of host time for 200 us of kernels; 71 us here).  Here the intermediates are
// carved out of one scratch area and the launches go out back to back.  The kernels, their order and their arithmetic are
// those of the step-by-step form (moe.py), which expert-parallel ranks keep using.
#include <cuda_runtime.h>

#include "dslgemm.h"

namespace {

struct Carver {
    size_t at = 0;
    size_t take(size_t bytes) {
        const size_t here = at;
        at += (bytes + 255) / 256 * 256;
        return here;
    }
};

struct Layout {
    size_t ids, weights, counts, offsets, tile0, dest;      // routing
    size_t q, sf, gs, ws;                                   // tokens, quantised once
    size_t rows, row_sf;                                    // expert-sorted rows and their scales
    size_t h, hq, h_sf, h_gs;                               // hidden activation (bf16) and its quantised form
    size_t y, total;
    size_t row_sf_bytes, h_sf_bytes;
};

bool fp4(int format) { return format == DSL_W_NVFP4 || format == DSL_W_MXFP4; }

// `fused`: the gate/up GEMM quantises the hidden activation itself (NVFP4 with a calibrated scale)
Layout carve(int format, bool fused, int tokens, int k, int experts, int K, int H, int D) {
    Layout l{};
    Carver c;
    const size_t T = tokens, R = T * k;
    l.ids = c.take(R * 4);
    l.weights = c.take(R * 4);
    l.counts = c.take(dsl_moe_plan_scratch_bytes(static_cast<int>(R), experts));
    l.offsets = c.take((experts + 1) * 4);
    l.tile0 = c.take((experts + 1) * 4);
    l.dest = c.take(R * 4);
    l.gs = c.take(4);
    l.h_gs = c.take(4);
    l.ws = c.take(16);
    const int blk = format == DSL_W_NVFP4 ? 16 : 32;
    const size_t row_q = fp4(format) ? K / 2 : (format == DSL_W_BF16 ? 2 * static_cast<size_t>(K) : K);
    const size_t row_h = fp4(format) ? H / 2 : H;
    if (fp4(format)) {
        l.q = c.take(T * row_q);
        l.sf = c.take(dsl_sf_bytes(T, K / blk));
        l.row_sf_bytes = dsl_sf_bytes_grouped(R, K / blk, experts);
        l.h_sf_bytes = dsl_sf_bytes_grouped(R, H / blk, experts);
    } else if (format == DSL_W_FP8_BLOCK128) {
        l.q = c.take(T * row_q);
        l.sf = c.take(T * (K / 128) * 4);
        l.row_sf_bytes = R * (K / 128) * 4;
        l.h_sf_bytes = R * (H / 128) * 4;
    } else if (format == DSL_W_FP8) {
        l.q = c.take(T * row_q);
    }
    l.rows = c.take(R * row_q);
    l.row_sf = c.take(l.row_sf_bytes);
    if (!fused) l.h = c.take(R * H * 2);
    if (format != DSL_W_BF16) l.hq = c.take(R * row_h);
    l.h_sf = c.take(l.h_sf_bytes);
    l.y = c.take(R * D * 2);
    l.total = c.at;
    return l;
}

int check_layer(const dsl_weight* gu, const dsl_weight* dn, int tokens, int k) {
    if (gu == nullptr || dn == nullptr) return DSL_ERR_NULL;
    if (gu->format != dn->format || gu->format < DSL_W_FP8 || gu->format > DSL_W_BF16) return DSL_ERR_ENUM;
    if (gu->groups < 1 || gu->groups > DSL_MAX_GROUPS || gu->groups != dn->groups || gu->n <= 0 || gu->n % 2 != 0 || dn->k != gu->n / 2 ||
        gu->k <= 0 || dn->n <= 0)
        return DSL_ERR_SHAPE;
    const int K = gu->k, H = dn->k;
    const int multiple = fp4(gu->format) ? 32 : (gu->format == DSL_W_FP8_BLOCK128 ? 128 : (gu->format == DSL_W_FP8 ? 16 : 8));
    if (K % multiple != 0 || H % multiple != 0) return DSL_ERR_SHAPE;
    // scale rows are dispatched as 16-byte vectors
    if (gu->format == DSL_W_FP8_BLOCK128 && (K / 128) % 4 != 0) return DSL_ERR_SHAPE;
    if (tokens < 0 || k < 1 || k > 32 || k > gu->groups) return DSL_ERR_SHAPE;
    if (static_cast<long long>(tokens) * k > 0x7FFFFFFFll) return DSL_ERR_TOO_LARGE;
    return 0;
}

}  // namespace

extern "C" size_t dsl_moe_layer_scratch_bytes(const dsl_weight* gate_up, const dsl_weight* down, int tokens, int k, int fused_hidden) {
    if (check_layer(gate_up, down, tokens, k) != 0) return 0;
    return carve(gate_up->format, fused_hidden != 0, tokens, k, gate_up->groups, gate_up->k, down->k, down->n).total;
}

extern "C" int dsl_moe_layer(const void* x, int x_dtype, const void* logits, int logits_dtype, int tokens, int k, int renorm,
                             const dsl_weight* gate_up, const dsl_weight* down, const float* act_gs_dev, int fused_hidden,
                             float hidden_gs, void* scratch, size_t scratch_bytes, void* out, int out_dtype, uint32_t* status,
                             void* stream) {
    int rc = check_layer(gate_up, down, tokens, k);
    if (rc != 0) return rc;
    if (x == nullptr || logits == nullptr || out == nullptr || scratch == nullptr || gate_up->q == nullptr || down->q == nullptr)
        return DSL_ERR_NULL;
    const int format = gate_up->format, E = gate_up->groups, K = gate_up->k, H = down->k, D = down->n;
    if (x_dtype < DSL_F32 || x_dtype > DSL_F16 || (format == DSL_W_BF16 && x_dtype != DSL_BF16)) return DSL_ERR_ENUM;
    if (fused_hidden && (format != DSL_W_NVFP4 || H % 16 != 0)) return DSL_ERR_ENUM;
    if (format != DSL_W_BF16 && (gate_up->scale == nullptr || down->scale == nullptr)) return DSL_ERR_NULL;
    if (format == DSL_W_NVFP4 && (gate_up->global_scale == nullptr || down->global_scale == nullptr)) return DSL_ERR_NULL;
    if ((reinterpret_cast<uintptr_t>(scratch) & 255u) != 0) return DSL_ERR_ALIGN;
    const Layout l = carve(format, fused_hidden != 0, tokens, k, E, K, H, D);
    if (scratch_bytes < l.total) return DSL_ERR_TOO_LARGE;
    if (tokens == 0) return 0;
    uint8_t* base = static_cast<uint8_t*>(scratch);
    auto u8 = [&](size_t off) { return base + off; };
    auto i32 = [&](size_t off) { return reinterpret_cast<int*>(base + off); };
    auto f32 = [&](size_t off) { return reinterpret_cast<float*>(base + off); };
    const int R = tokens * k;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define DSL_STEP(call) do { rc = (call); if (rc != 0) return rc; } while (0)
    // Routing and plan go out after the quantiser where there is one: they are launched as programmatic dependents (moe.cu),
    // the quantiser, a kernel of other chains too, is not.
    auto route_and_plan = [&]() -> int {
        const int r = dsl_moe_route(logits, logits_dtype, tokens, E, k, renorm, i32(l.ids), f32(l.weights), stream);
        return r != 0 ? r : dsl_moe_plan(i32(l.ids), R, E, i32(l.counts), i32(l.offsets), i32(l.tile0), i32(l.dest), stream);
    };
    const int* offs = i32(l.offsets);
    dsl_epilogue up{}, dn{};
    up.scale_a_host = up.scale_b_host = dn.scale_a_host = dn.scale_b_host = 1.0f;
    up.b_is_static = dn.b_is_static = 1;
    up.activation = DSL_ACT_SWIGLU;
    up.out_dtype = dn.out_dtype = DSL_BF16;
    uint8_t* y = u8(l.y);
    const uint8_t* wu = static_cast<const uint8_t*>(gate_up->q);
    const uint8_t* wd = static_cast<const uint8_t*>(down->q);
    if (fp4(format)) {
        const int fmt = format == DSL_W_NVFP4 ? DSL_FP4_NV : DSL_FP4_MX;
        const int blk = fmt == DSL_FP4_NV ? 16 : 32;
        float* gs = act_gs_dev != nullptr ? const_cast<float*>(act_gs_dev) : f32(l.gs);
        DSL_STEP(dsl_quant_fp4(x, x_dtype, tokens, K, fmt, fmt == DSL_FP4_NV ? gs : nullptr, act_gs_dev != nullptr, u8(l.q), u8(l.sf),
                               nullptr, 0, u8(l.ws), stream));
        DSL_STEP(route_and_plan());
        // Scale bytes of rows no group owns only reach result rows that nobody stores; those past the last K block meet
        // zero-filled elements, where a NaN pattern would spread, so they alone have to be cleared.
        if ((K / blk) % 4 != 0) DSL_STEP(static_cast<int>(cudaMemsetAsync(u8(l.row_sf), 0, l.row_sf_bytes, st)));
        DSL_STEP(dsl_moe_dispatch_fp4(u8(l.q), u8(l.sf), i32(l.ids), i32(l.dest), i32(l.offsets), i32(l.tile0), tokens, k, K, fmt, 0, E,
                                      u8(l.rows), u8(l.row_sf), stream));
        if (fmt == DSL_FP4_NV) {
            up.scale_a_dev = gs;
            up.scale_b_dev = gate_up->global_scale;
            dn.scale_b_dev = down->global_scale;
        }
        if (fused_hidden) {
            if ((H / blk) % 4 != 0) DSL_STEP(static_cast<int>(cudaMemsetAsync(u8(l.h_sf), 0, l.h_sf_bytes, st)));
            up.out_dtype = DSL_OUT_NVFP4;
            up.out_sf = u8(l.h_sf);
            up.out_gs_host = hidden_gs;
            dn.scale_a_host = hidden_gs;
            DSL_STEP(dsl_gemm_fp4(u8(l.rows), wu, u8(l.row_sf), static_cast<const uint8_t*>(gate_up->scale), fmt, u8(l.hq), H, R,
                                  gate_up->n, K, offs, E, &up, status, stream));
        } else {
            DSL_STEP(dsl_gemm_fp4(u8(l.rows), wu, u8(l.row_sf), static_cast<const uint8_t*>(gate_up->scale), fmt, u8(l.h), H, R,
                                  gate_up->n, K, offs, E, &up, status, stream));
            DSL_STEP(dsl_quant_fp4(u8(l.h), DSL_BF16, R, H, fmt, fmt == DSL_FP4_NV ? f32(l.h_gs) : nullptr, 0, u8(l.hq), u8(l.h_sf),
                                   i32(l.offsets), E, u8(l.ws), stream));
            if (fmt == DSL_FP4_NV) dn.scale_a_dev = f32(l.h_gs);
        }
        DSL_STEP(dsl_gemm_fp4(u8(l.hq), wd, u8(l.h_sf), static_cast<const uint8_t*>(down->scale), fmt, y, D, R, D, H, offs, E, &dn, status,
                              stream));
    } else if (format == DSL_W_FP8) {
        DSL_STEP(dsl_quant_fp8(x, x_dtype, tokens, K, DSL_FP8_PER_TENSOR, f32(l.gs), 0, u8(l.q), u8(l.ws), stream));
        DSL_STEP(route_and_plan());
        DSL_STEP(dsl_moe_dispatch_rows(u8(l.q), i32(l.ids), i32(l.dest), i32(l.offsets), tokens, k, K, 0, E, u8(l.rows), stream));
        up.scale_a_dev = f32(l.gs);
        up.scale_b_dev = static_cast<const float*>(gate_up->scale);
        DSL_STEP(dsl_gemm_fp8(u8(l.rows), wu, u8(l.h), H, R, gate_up->n, K, offs, E, &up, status, stream));
        DSL_STEP(dsl_quant_fp8(u8(l.h), DSL_BF16, R, H, DSL_FP8_PER_TENSOR, f32(l.h_gs), 0, u8(l.hq), u8(l.ws), stream));
        dn.scale_a_dev = f32(l.h_gs);
        dn.scale_b_dev = static_cast<const float*>(down->scale);
        DSL_STEP(dsl_gemm_fp8(u8(l.hq), wd, y, D, R, D, H, offs, E, &dn, status, stream));
    } else if (format == DSL_W_FP8_BLOCK128) {
        DSL_STEP(dsl_quant_fp8(x, x_dtype, tokens, K, DSL_FP8_GROUP_1X128, f32(l.sf), 0, u8(l.q), u8(l.ws), stream));
        DSL_STEP(route_and_plan());
        DSL_STEP(dsl_moe_dispatch_rows(u8(l.q), i32(l.ids), i32(l.dest), i32(l.offsets), tokens, k, K, 0, E, u8(l.rows), stream));
        DSL_STEP(dsl_moe_dispatch_rows(u8(l.sf), i32(l.ids), i32(l.dest), i32(l.offsets), tokens, k, K / 128 * 4ll, 0, E, u8(l.row_sf), stream));
        DSL_STEP(dsl_gemm_fp8_groupwise(u8(l.rows), wu, f32(l.row_sf), static_cast<const float*>(gate_up->scale), 1, u8(l.h), H, R,
                                        gate_up->n, K, offs, E, &up, status, stream));
        DSL_STEP(dsl_quant_fp8(u8(l.h), DSL_BF16, R, H, DSL_FP8_GROUP_1X128, f32(l.h_sf), 0, u8(l.hq), u8(l.ws), stream));
        DSL_STEP(dsl_gemm_fp8_groupwise(u8(l.hq), wd, f32(l.h_sf), static_cast<const float*>(down->scale), 1, y, D, R, D, H, offs, E, &dn,
                                        status, stream));
    } else {
        DSL_STEP(route_and_plan());
        DSL_STEP(dsl_moe_dispatch_rows(x, i32(l.ids), i32(l.dest), i32(l.offsets), tokens, k, 2ll * K, 0, E, u8(l.rows), stream));
        DSL_STEP(dsl_gemm_bf16(u8(l.rows), wu, u8(l.h), H, R, gate_up->n, K, offs, E, &up, status, stream));
        DSL_STEP(dsl_gemm_bf16(u8(l.h), wd, y, D, R, D, H, offs, E, &dn, status, stream));
    }
    DSL_STEP(dsl_moe_combine(y, DSL_BF16, i32(l.ids), i32(l.dest), i32(l.offsets), f32(l.weights), tokens, k, D, 0, E, out, out_dtype, stream));
#undef DSL_STEP
    return 0;
}
