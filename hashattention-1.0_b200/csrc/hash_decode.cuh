// Decode-time hash encoder: one CTA per (query head, side) evaluates the head's 3-layer MLP
// (128 -> 128 -> 128 -> 32, SiLU between, sign at the end) for the new query / new key of every
// sequence of its batch slice, packs the 32 sign bits with one warp ballot, and appends the
// new key's code (and the K / V rows) to the paged caches.
//
// Follows USA.q_embedding / USA.k_embedding with hard=True
// (hashattention/hashattention_llama.py:204-226) in fp32 arithmetic.
#pragma once

#include "common.cuh"

namespace ha {

constexpr int kHashDecodeThreads = 512;

struct HashDecodeParams {
    const __nv_bfloat16* q;      // [B][Hq][128]
    const __nv_bfloat16* k_new;  // [B][Hkv][128] or null (query side only)
    const __nv_bfloat16* v_new;  // [B][Hkv][128] or null
    const void* w[2];            // side 0 = query MLPs, side 1 = key MLPs
    const float* bias[2];
    __nv_bfloat16* k_pages;
    __nv_bfloat16* v_pages;
    uint32_t* hash_pages;
    const int32_t* page_table;
    const int32_t* seq_lens;
    uint32_t* q_codes;   // [B][Hq]
    float* preact_dbg;   // [B][2][Hq][32] or null
    __nv_bfloat16* q_stage;  // [B][Hq][128] or null: a device copy of q for the attention kernels, written when
                             // q itself lives in mapped host memory (read once here instead of by every gather CTA)
    int32_t* status;
    int B, Hkv, max_pages, num_pages, batch_per_cta;
    int layers;          // 3, 2 or 1 Linear layers (see ha_hash_weights_t.num_layers)
};

// Eight consecutive weights of one row, as stored, and their dot product with eight inputs.
template <typename WT>
struct Row8;

template <>
struct Row8<__nv_bfloat16> {
    uint4 raw;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) {
        raw = __ldg(reinterpret_cast<const uint4*>(p));
    }
    __device__ __forceinline__ float dot(const float (&x)[8]) const {
        float s = bf16_lo(raw.x) * x[0];
        s = fmaf(bf16_hi(raw.x), x[1], s);
        s = fmaf(bf16_lo(raw.y), x[2], s);
        s = fmaf(bf16_hi(raw.y), x[3], s);
        s = fmaf(bf16_lo(raw.z), x[4], s);
        s = fmaf(bf16_hi(raw.z), x[5], s);
        s = fmaf(bf16_lo(raw.w), x[6], s);
        s = fmaf(bf16_hi(raw.w), x[7], s);
        return s;
    }
    __device__ __forceinline__ void unpack(float (&e)[8]) const {
        e[0] = bf16_lo(raw.x); e[1] = bf16_hi(raw.x); e[2] = bf16_lo(raw.y); e[3] = bf16_hi(raw.y);
        e[4] = bf16_lo(raw.z); e[5] = bf16_hi(raw.z); e[6] = bf16_lo(raw.w); e[7] = bf16_hi(raw.w);
    }
};

template <>
struct Row8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) {
        a = __ldg(reinterpret_cast<const float4*>(p));
        b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    }
    __device__ __forceinline__ float dot(const float (&x)[8]) const {
        float s = a.x * x[0];
        s = fmaf(a.y, x[1], s);
        s = fmaf(a.z, x[2], s);
        s = fmaf(a.w, x[3], s);
        s = fmaf(b.x, x[4], s);
        s = fmaf(b.y, x[5], s);
        s = fmaf(b.z, x[6], s);
        s = fmaf(b.w, x[7], s);
        return s;
    }
    __device__ __forceinline__ void unpack(float (&e)[8]) const {
        e[0] = a.x; e[1] = a.y; e[2] = a.z; e[3] = a.w;
        e[4] = b.x; e[5] = b.y; e[6] = b.z; e[7] = b.w;
    }
};

__device__ __forceinline__ float half_warp_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

__device__ __forceinline__ float silu(float x) { return x / (1.0f + expf(-x)); }

// Sums of N rows (N = 1 or 4) over the 16 lanes of a half-warp. With four rows a lane hands half of its rows to its partner
// and keeps the other half in the first two steps of the butterfly, so they take 5 shuffles instead of 16 and every lane
// ends up with the sum of one row, row spread_row<N>(sub). Each row is added up in the order of half_warp_sum.
template <int N>
__device__ __forceinline__ float spread_sum(const float (&s)[N], int sub) {
    static_assert(N == 1 || N == 4, "one row, or four");
    if constexpr (N == 1) {
        return half_warp_sum(s[0]);
    } else {
        const bool upper8 = (sub & 8) != 0, upper4 = (sub & 4) != 0;
        float r[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float send = upper8 ? s[i] : s[i + 2], keep = upper8 ? s[i + 2] : s[i];
            r[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
        const float send = upper4 ? r[0] : r[1], keep = upper4 ? r[1] : r[0];
        float t = keep + __shfl_xor_sync(0xffffffffu, send, 4);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        return t + __shfl_xor_sync(0xffffffffu, t, 1);
    }
}
// the row whose sum lane `sub` of a half-warp ends up with; 16 / N lanes hold the same one, the first of them has
// sub % (16 / N) == 0
template <int N>
__device__ __forceinline__ int spread_row(int sub) { return sub / (16 / N); }

// Thread mapping: 16 warps; a half-warp (16 lanes x 8 columns) covers one 128-wide weight row.
// In the two hidden layers a warp owns 8 consecutive output rows: load j of a lane belongs to
// row 2j + (lane >> 4) of them. In the last layer it owns 2 rows in the same way.
constexpr int kMlpWarps = kHashDecodeThreads / 32;  // 16
constexpr int kHid = kHidden / kMlpWarps / 2;       // rows per half-warp in a hidden layer: 4
constexpr int kOut = kCodeBits / kMlpWarps / 2;     // ... in the last one: 1

// One head's MLP held in the registers of a 512-thread CTA.
template <typename WT>
struct MlpRegs {
    Row8<WT> w0[kHid], w1[kHid], w2[kOut];
    float b0, b1, b2;  // biases of the rows whose sums this lane ends up with

    // All three layers are fetched back to back so that their DRAM latency is paid once.
    __device__ __forceinline__ void load(const WT* W, const float* bias, int warp, int lane) {
        const int half = lane >> 4, sub = lane & 15, col = sub * 8;
#pragma unroll
        for (int j = 0; j < kHid; ++j) {
            const int row = warp * (2 * kHid) + 2 * j + half;
            w0[j].load(W + row * kHeadDim + col);
            w1[j].load(W + kHidden * kHeadDim + row * kHidden + col);
        }
#pragma unroll
        for (int j = 0; j < kOut; ++j)
            w2[j].load(W + kHidden * kHeadDim + kHidden * kHidden + (warp * (2 * kOut) + 2 * j + half) * kHidden + col);
        b0 = __ldg(bias + warp * (2 * kHid) + 2 * spread_row<kHid>(sub) + half);
        b1 = __ldg(bias + kHidden + warp * (2 * kHid) + 2 * spread_row<kHid>(sub) + half);
        b2 = __ldg(bias + 2 * kHidden + warp * (2 * kOut) + 2 * spread_row<kOut>(sub) + half);
    }
};

struct MlpSmem {
    __align__(16) float h0[kHidden];
    __align__(16) float h1[kHidden];
    float out[kCodeBits];
};

__device__ __forceinline__ void unpack_x8(const uint4 raw, float (&x)[8]) {
    x[0] = bf16_lo(raw.x); x[1] = bf16_hi(raw.x);
    x[2] = bf16_lo(raw.y); x[3] = bf16_hi(raw.y);
    x[4] = bf16_lo(raw.z); x[5] = bf16_hi(raw.z);
    x[6] = bf16_lo(raw.w); x[7] = bf16_hi(raw.w);
}

__device__ __forceinline__ void load_x8(const float* s, float (&x)[8]) {
    const float4 lo = *reinterpret_cast<const float4*>(s);
    const float4 hi = *reinterpret_cast<const float4*>(s + 4);
    x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w;
    x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
}

// One layer: the row sums of the warp's rows plus bias; a lane returns the one it ended up with.
template <typename WT, int N>
__device__ __forceinline__ float mlp_rows(const Row8<WT> (&w)[N], float bias, const float (&x)[8], int lane) {
    float s[N];
#pragma unroll
    for (int j = 0; j < N; ++j) s[j] = w[j].dot(x);
    return spread_sum<N>(s, lane & 15) + bias;
}
// stores a lane's row of a layer (one of the lanes that hold it)
template <int N>
__device__ __forceinline__ void mlp_store(float v, float* dst, int warp, int lane) {
    const int half = lane >> 4, sub = lane & 15;
    if (sub % (16 / N) == 0) dst[warp * (2 * N) + 2 * spread_row<N>(sub) + half] = v;
}

// Evaluates the MLP on one 128-element bf16 row, of which `raw` holds this lane's 8 elements
// (load_x_row). Must be called by all threads of the CTA; on
// return (after its last barrier) sm.out[0..32) holds the final-layer pre-activations.
// `between` runs after the first layer (a place to issue loads whose address depends on a value
// that was requested before the call). The caller may call mlp_eval again without a further
// barrier: each buffer is rewritten only after barriers that every reader of the previous
// round has passed.
//
// layers: 3 = all of W0, W1, W2; 2 = W0 then W2 (Linear-SiLU-Linear, hashattention_llama.py:112-120);
// 1 = W2 alone (:121-127).
template <typename WT, typename F>
__device__ __forceinline__ void mlp_eval(const MlpRegs<WT>& r, const uint4 raw,
                                         MlpSmem& sm, int warp, int lane, F&& between, int layers = 3) {
    const int col = (lane & 15) * 8;
    float x[8];
    unpack_x8(raw, x);
    if (layers >= 2) mlp_store<kHid>(silu(mlp_rows(r.w0, r.b0, x, lane)), sm.h0, warp, lane);
    between();
    if (layers >= 2) {
        __syncthreads();
        load_x8(sm.h0 + col, x);
    } else {
        __syncthreads();  // no hidden layer separates this call's write of `out` from the previous call's readers
    }
    if (layers == 3) {
        mlp_store<kHid>(silu(mlp_rows(r.w1, r.b1, x, lane)), sm.h1, warp, lane);
        __syncthreads();
        load_x8(sm.h1 + col, x);
    }
    mlp_store<kOut>(mlp_rows(r.w2, r.b2, x, lane), sm.out, warp, lane);
    __syncthreads();
}

// mlp_eval for two rows at once (`sm[0]`, `sm[1]`): the same weights in registers feed both rows, and the two
// dependent chains (dot, shuffle reduction, SiLU, barrier) interleave, so the pair costs little more than one row.
template <typename WT, typename F>
__device__ __forceinline__ void mlp_eval2(const MlpRegs<WT>& r, const uint4 raw_a, const uint4 raw_b,
                                          MlpSmem (&sm)[2], int warp, int lane, F&& between, int layers = 3) {
    const int col = (lane & 15) * 8;
    float xa[8], xb[8];
    unpack_x8(raw_a, xa);
    unpack_x8(raw_b, xb);
    if (layers >= 2) {
        const float a = mlp_rows(r.w0, r.b0, xa, lane), b = mlp_rows(r.w0, r.b0, xb, lane);
        mlp_store<kHid>(silu(a), sm[0].h0, warp, lane);
        mlp_store<kHid>(silu(b), sm[1].h0, warp, lane);
    }
    between();
    __syncthreads();
    if (layers >= 2) {
        load_x8(sm[0].h0 + col, xa);
        load_x8(sm[1].h0 + col, xb);
    }
    if (layers == 3) {
        const float a = mlp_rows(r.w1, r.b1, xa, lane), b = mlp_rows(r.w1, r.b1, xb, lane);
        mlp_store<kHid>(silu(a), sm[0].h1, warp, lane);
        mlp_store<kHid>(silu(b), sm[1].h1, warp, lane);
        __syncthreads();
        load_x8(sm[0].h1 + col, xa);
        load_x8(sm[1].h1 + col, xb);
    }
    const float a = mlp_rows(r.w2, r.b2, xa, lane), b = mlp_rows(r.w2, r.b2, xb, lane);
    mlp_store<kOut>(a, sm[0].out, warp, lane);
    mlp_store<kOut>(b, sm[1].out, warp, lane);
    __syncthreads();
}

// This lane's 8 consecutive elements (columns 8 * (lane % 16) ...) of a 128-element bf16 row.
__device__ __forceinline__ uint4 load_x_row(const __nv_bfloat16* xrow, int lane) {
    return *reinterpret_cast<const uint4*>(xrow + (lane & 15) * 8);
}

// kPairs: a CTA with two or more sequences evaluates them two at a time; with one sequence per CTA the
// single-row loop is a little leaner.
template <typename WT, bool kPairs>
__global__ void __launch_bounds__(kHashDecodeThreads)
hash_decode_kernel(const HashDecodeParams p) {
    const int h = blockIdx.x;                // query head whose MLP this CTA evaluates
    const int side = blockIdx.y;             // 0 = query net, 1 = key net
    const int Hq = p.Hkv * kGroup;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    MlpRegs<WT> regs;
    regs.load(static_cast<const WT*>(p.w[side]) + (size_t)h * kMlpElems,
              p.bias[side] + (size_t)h * kMlpBias, warp, lane);
    __shared__ MlpSmem sm[2];

    const int b_begin = blockIdx.z * p.batch_per_cta;
    const int b_end = min(p.B, b_begin + p.batch_per_cta);
    const int kvh = h / kGroup, g = h % kGroup;

    // The input rows may be products of the kernel in front, so they are read after the wait; asking L2 for their
    // lines beforehand is harmless either way (L2 is where that kernel's stores land) and saves the DRAM trip when
    // the rows were written long ago. Not for rows in mapped host memory (q_stage given), which L2 does not hold.
    if (p.q_stage == nullptr) {
        for (int i = tid; i < 2 * (b_end - b_begin); i += kHashDecodeThreads) {
            const int b = b_begin + (i >> 1);
            const __nv_bfloat16* row = side == 0 ? p.q + ((size_t)b * Hq + h) * kHeadDim
                                                 : p.k_new + ((size_t)b * p.Hkv + kvh) * kHeadDim;
            prefetch_l2(row + (i & 1) * (kHeadDim / 2));
            if (side == 1 && g == 0 && p.v_new != nullptr)
                prefetch_l2(p.v_new + ((size_t)b * p.Hkv + kvh) * kHeadDim + (i & 1) * (kHeadDim / 2));
        }
    }

    pdl_wait();
    pdl_launch_dependents();

    if constexpr (kPairs) {
        // The sequences of this CTA are evaluated two at a time (the pair shares every weight register and its two
        // dependent chains interleave); the input rows, the V rows of the append and (key side) the sequence lengths
        // of a pair are requested together, the page-table entries of the append slots underneath the MLP arithmetic.
        auto x_row = [&](int b) {
            return side == 0 ? p.q + ((size_t)b * Hq + h) * kHeadDim : p.k_new + ((size_t)b * p.Hkv + kvh) * kHeadDim;
        };
        // The group's first key head also appends the K and V rows: lanes 0-15 of warp 0 hold the K row already (it
        // is the MLP's input), lanes 16-31 request the V row together with it - the inputs may live in mapped
        // host memory, where a second read at the end of the kernel would cost another trip over the bus.
        const bool appends = side == 1 && g == 0 && p.v_new != nullptr && warp == 0;
        auto v_part = [&](int b) {
            return *(reinterpret_cast<const uint4*>(p.v_new + ((size_t)b * p.Hkv + kvh) * kHeadDim) + (lane - 16));
        };
        // what warp 0 does with a finished row: code out, and (key side) the append
        auto finish = [&](int b, const MlpSmem& m, const uint4 raw, const uint4 v_raw, int S, int page) {
            const float pre = m.out[lane];
            // bit i = 1 iff output i > 0 (efficiency/kernels/torchatt.py:35-36: relu(sign(x)))
            const uint32_t code = __ballot_sync(0xffffffffu, pre > 0.0f);
            if (p.preact_dbg != nullptr)
                p.preact_dbg[(((size_t)b * 2 + side) * Hq + h) * kCodeBits + lane] = pre;
            if (side == 0) {
                if (lane == 0) p.q_codes[(size_t)b * Hq + h] = code;
                return;
            }
            if (S < 1 || S > p.max_pages * kPage) {
                if (lane == 0) report(p.status, HA_ERR_BAD_SEQ_LEN);
                return;
            }
            if (page < 0 || page >= p.num_pages) {
                if (lane == 0) report(p.status, HA_ERR_BAD_PAGE);
                return;
            }
            const size_t slot = ((size_t)page * p.Hkv + kvh) * kPage + (S - 1) % kPage;
            if (lane == 0) p.hash_pages[slot * kGroup + g] = code;
            // the group's first head also appends the K and V rows (256 B each)
            if (appends) {
                uint4* d = lane < 16 ? reinterpret_cast<uint4*>(p.k_pages + slot * kHeadDim) + lane
                                     : reinterpret_cast<uint4*>(p.v_pages + slot * kHeadDim) + (lane - 16);
                *d = lane < 16 ? raw : v_raw;
            }
        };
        auto page_of = [&](int b, int S) {
            return p.page_table[(size_t)b * p.max_pages + min(max(S - 1, 0) / kPage, p.max_pages - 1)];
        };
        for (int b = b_begin; b < b_end; b += 2) {
            const bool two = b + 1 < b_end;
            const int b1 = two ? b + 1 : b;
            const uint4 raw0 = load_x_row(x_row(b), lane), raw1 = load_x_row(x_row(b1), lane);
            uint4 v0 = make_uint4(0u, 0u, 0u, 0u), v1 = v0;
            if (appends && lane >= 16) {
                v0 = v_part(b);
                v1 = v_part(b1);
            }
            int S0 = 1, S1 = 1, page0 = 0, page1 = 0;
            if (side == 1) {
                S0 = p.seq_lens[b];
                S1 = p.seq_lens[b1];
            }
            if (side == 0 && p.q_stage != nullptr && warp == 0 && lane < 16) {
                *reinterpret_cast<uint4*>(p.q_stage + ((size_t)b * Hq + h) * kHeadDim + lane * 8) = raw0;
                if (two) *reinterpret_cast<uint4*>(p.q_stage + ((size_t)b1 * Hq + h) * kHeadDim + lane * 8) = raw1;
            }
            if (two) {
                mlp_eval2(regs, raw0, raw1, sm, warp, lane, [&] {
                    if (side == 1) {
                        page0 = page_of(b, S0);
                        page1 = page_of(b1, S1);
                    }
                }, p.layers);
            } else {
                mlp_eval(regs, raw0, sm[0], warp, lane, [&] {
                    if (side == 1) page0 = page_of(b, S0);
                }, p.layers);
            }
            if (warp != 0) continue;
            finish(b, sm[0], raw0, v0, S0, page0);
            if (two) finish(b1, sm[1], raw1, v1, S1, page1);
        }
    } else {
        // The input row and (key side) the sequence length of the next sequence are requested while the
        // current one is evaluated; the page-table entry of the append slot, whose address depends on
        // the length, is fetched underneath the MLP arithmetic.
        auto x_row = [&](int b) {
            return side == 0 ? p.q + ((size_t)b * Hq + h) * kHeadDim : p.k_new + ((size_t)b * p.Hkv + kvh) * kHeadDim;
        };
        // The group's first key head also appends the K and V rows: lanes 0-15 of warp 0 hold the K row already (it
        // is the MLP's input), lanes 16-31 request the V row together with it - the inputs may live in mapped
        // host memory, where a second read at the end of the kernel would cost another trip over the bus.
        const bool appends = side == 1 && g == 0 && p.v_new != nullptr && warp == 0;
        auto v_part = [&](int b) {
            return *(reinterpret_cast<const uint4*>(p.v_new + ((size_t)b * p.Hkv + kvh) * kHeadDim) + (lane - 16));
        };
        uint4 raw_next = make_uint4(0u, 0u, 0u, 0u), v_next = make_uint4(0u, 0u, 0u, 0u);
        int S_next = 1;
        if (b_begin < b_end) {
            raw_next = load_x_row(x_row(b_begin), lane);
            if (appends && lane >= 16) v_next = v_part(b_begin);
            if (side == 1) S_next = p.seq_lens[b_begin];
        }
        for (int b = b_begin; b < b_end; ++b) {
            const uint4 raw = raw_next, v_raw = v_next;
            const int S = S_next;
            if (b + 1 < b_end) {
                raw_next = load_x_row(x_row(b + 1), lane);
                if (appends && lane >= 16) v_next = v_part(b + 1);
                if (side == 1) S_next = p.seq_lens[b + 1];
            }
            if (side == 0 && p.q_stage != nullptr && warp == 0 && lane < 16)
                *reinterpret_cast<uint4*>(p.q_stage + ((size_t)b * Hq + h) * kHeadDim + lane * 8) = raw;
            int page = 0;
            mlp_eval(regs, raw, sm[0], warp, lane, [&] {
                if (side == 1) {
                    const int pidx = min(max(S - 1, 0) / kPage, p.max_pages - 1);
                    page = p.page_table[(size_t)b * p.max_pages + pidx];
                }
            }, p.layers);
            if (warp != 0) continue;

            const float pre = sm[0].out[lane];
            // bit i = 1 iff output i > 0 (efficiency/kernels/torchatt.py:35-36: relu(sign(x)))
            const uint32_t code = __ballot_sync(0xffffffffu, pre > 0.0f);
            if (p.preact_dbg != nullptr)
                p.preact_dbg[(((size_t)b * 2 + side) * Hq + h) * kCodeBits + lane] = pre;
            if (side == 0) {
                if (lane == 0) p.q_codes[(size_t)b * Hq + h] = code;
                continue;
            }
            if (S < 1 || S > p.max_pages * kPage) {
                if (lane == 0) report(p.status, HA_ERR_BAD_SEQ_LEN);
                continue;
            }
            const int tok = S - 1;
            if (page < 0 || page >= p.num_pages) {
                if (lane == 0) report(p.status, HA_ERR_BAD_PAGE);
                continue;
            }
            const size_t slot = ((size_t)page * p.Hkv + kvh) * kPage + tok % kPage;
            if (lane == 0) p.hash_pages[slot * kGroup + g] = code;
            // the group's first head also appends the K and V rows (256 B each)
            if (appends) {
                uint4* d = lane < 16 ? reinterpret_cast<uint4*>(p.k_pages + slot * kHeadDim) + lane
                                     : reinterpret_cast<uint4*>(p.v_pages + slot * kHeadDim) + (lane - 16);
                *d = lane < 16 ? raw : v_raw;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// Batched variant: a CTA evaluates 16 sequences of its (head, side) at once, each layer a GEMM of 16 rows on the tensor
// cores (mma.sync m16n8k16; the 128 rows of a tcgen05 tile would be seven eighths padding). Weights stay in registers (but
// for 72 bytes a thread that the build for fp32 weights spills) in the form in which the matrix instruction takes them: a warp
// owns one or two n-tiles (8 outputs) of a hidden layer, and in the last layer n-tile w % 4 over a part of the inputs. The
// order of the inputs inside a product is free, so a lane's share of 32 inputs is 8 consecutive ones: one 16-byte load each of
// weights and activations feeds two k-steps.
// Precision: products of two bf16 are exact. An activation is split into three bf16 (24 bits of mantissa), an fp32 weight
// too; of their nine products the three smallest are left out, the larger two of them at most 2^-22 of the whole each (cut
// off parts lie below 2^-7 and 2^-15 of it). The products of the leading parts are summed up by the matrix instruction over
// 16 inputs only and from there in fp32 additions, so that its truncation stays below theirs. Errors of the
// pre-activations against 64 bits, beside those of the encoder above: at hm_min_rows.
// What bounds it: latencies - weights, rows, three GEMMs with a barrier each - at about a third of the issue slots. Against
// the form before, whose fp32 multiply-adds from transposed fp32 weights in shared memory took 3/4 of its time: 12 - 32 sequences x 8 kv-heads 10.9 -> 4.6 us, 64
// 18.5 -> 8.0, 100 32.5 -> 14.0; fp32 weights 13.4 -> 8.0 (with parts rounded by cvt instead of truncated 9.5), 21.1 ->
// 13.6 and 36.0 -> 24.2. With 16 warps for bf16 weights 4.65 and 8.5.
// ------------------------------------------------------------------------------------------
constexpr int kHmRows = 16;             // sequences per CTA and pass
// Warps: each of them reads the 16 rows of activations, so fewer are better (8); fp32 weights, split into parts on the
// way, want more of them at work and half the registers each.
template <typename WT> constexpr int kHmWarps = sizeof(WT) == 4 ? 16 : 8;
constexpr int kHmBlocks = kHidden / 32;             // blocks of 32 inputs: 4
constexpr int kHmParts = 3;             // bf16 parts of an activation
constexpr int kHmPitch = kHidden + 32;  // elements: 16-byte reads of two neighbouring rows hit different banks
// Sequences per CTA from which the batched kernel is used. One encoder with 8 kv-heads (two CTAs per head and side), this
// kernel / the one above, us: bf16 weights 4.5 / 3.9 with 2 rows per CTA, 4.5 / 5.4 with 3, 4.4 / 6.2 with 4, 4.4 / 7.7 with
// 5; fp32 weights 8.0 / 7.1 with 4, 8.0 / 8.7 with 5. But up to 5 rows, where the kernel above is the alternative, only where
// the sums are no further from 64 bits than there, rms in units of 1e-9: bf16 weights 7.2 / 7.6 with three layers, 17.5 / 18.8
// with two, 28.6 / 26.9 with one; fp32 weights 10.8 / 8.6, 24.1 / 23.0, 34.2 / 46.6. (The form before this one had 19.9,
// 41.9, 39.5 and 20.6, 46.0, 118.)
inline int hm_min_rows(bool bf16_weights, int layers) { return bf16_weights && layers >= 2 ? 3 : 6; }
struct HmSmem {
    __align__(16) __nv_bfloat16 x[1][kHmRows][kHmPitch];
    __align__(16) __nv_bfloat16 act[2][kHmParts][kHmRows][kHmPitch];
    float part[4][kHmRows][kCodeBits];  // sums of the last layer over the warps' parts of the inputs
};

// Eight consecutive weights of one row as bf16 pairs: word(i, s) is part s of the weights 2 i and 2 i + 1
template <typename WT>
struct HmWeights;
template <>
struct HmWeights<__nv_bfloat16> {
    static constexpr int kParts = 1;
    uint4 raw;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { raw = __ldg(reinterpret_cast<const uint4*>(p)); }
    __device__ __forceinline__ void pin() {}
    __device__ __forceinline__ void words(int i, uint32_t (&w)[1]) const { w[0] = i == 0 ? raw.x : (i == 1 ? raw.y : (i == 2 ? raw.z : raw.w)); }
};
// a and b as three bf16 each, by truncation: 8 bits of the mantissa at a time, 24 in all, so the sum of the parts is exact
__device__ __forceinline__ void split3(float a, float b, uint32_t (&w)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        w[i] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);  // the upper halves, a's in the low half
        a -= bf16_lo(w[i]);
        b -= bf16_hi(w[i]);
    }
}
template <>
struct HmWeights<float> {
    static constexpr int kParts = 3;
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) {
        a = __ldg(reinterpret_cast<const float4*>(p));
        b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    }
    __device__ __forceinline__ void pin() {
        asm volatile("" : "+f"(a.x), "+f"(a.y), "+f"(a.z), "+f"(a.w), "+f"(b.x), "+f"(b.y), "+f"(b.z), "+f"(b.w));
    }
    __device__ __forceinline__ void words(int i, uint32_t (&w)[3]) const {
        if (i == 0) split3(a.x, a.y, w);
        else if (i == 1) split3(a.z, a.w, w);
        else if (i == 2) split3(b.x, b.y, w);
        else split3(b.z, b.w, w);
    }
};

__device__ __forceinline__ void mma_16x8x16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// acc = the 16 rows of A (kA bf16 parts) times TILES n-tiles of weights, over the input blocks [blk0, blk0 + BLOCKS). A lane
// ends up with rows lane / 4 and lane / 4 + 8, outputs 2 (lane % 4) and the next one, of each tile.
template <int kA, int TILES, int BLOCKS, typename WT>
__device__ __forceinline__ void hm_gemm(float (&acc)[TILES][4], const __nv_bfloat16 (*A)[kHmRows][kHmPitch], int blk0,
                                        const HmWeights<WT> (&w)[TILES][BLOCKS], int lane) {
    constexpr int kW = HmWeights<WT>::kParts;
    float small[2][TILES][4];  // products of which one factor is not a leading part, by magnitude
#pragma unroll
    for (int n = 0; n < TILES; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = small[0][n][i] = small[1][n][i] = 0.f;
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) {
        uint4 lo[kA], hi[kA];  // rows lane / 4 and lane / 4 + 8, inputs [8 (lane % 4), + 8) of the block
#pragma unroll
        for (int s = 0; s < kA; ++s) {
            const __nv_bfloat16* src = &A[s][lane / 4][(blk0 + k) * 32 + (lane % 4) * 8];
            lo[s] = *reinterpret_cast<const uint4*>(src);
            hi[s] = *reinterpret_cast<const uint4*>(src + 8 * kHmPitch);
        }
#pragma unroll
        for (int n = 0; n < TILES; ++n) {
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                uint32_t b0[kW], b1[kW];
                w[n][k].words(2 * kk, b0);
                w[n][k].words(2 * kk + 1, b1);
#pragma unroll
                for (int s = 0; s < kA; ++s) {
                    const uint32_t a[4] = {kk ? lo[s].z : lo[s].x, kk ? hi[s].z : hi[s].x, kk ? lo[s].w : lo[s].y, kk ? hi[s].w : hi[s].y};
#pragma unroll
                    for (int v = 0; v < kW && s + v <= 2; ++v) {
                        if (s + v == 0) {
                            float d[4] = {0.f, 0.f, 0.f, 0.f};
                            mma_16x8x16(d, a, b0[0], b1[0]);
#pragma unroll
                            for (int i = 0; i < 4; ++i) acc[n][i] += d[i];
                        } else {
                            mma_16x8x16(small[s + v - 1][n], a, b0[v], b1[v]);
                        }
                    }
                }
            }
        }
    }
#pragma unroll
    for (int n = 0; n < TILES; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] += small[0][n][i] + small[1][n][i];
}

// bias + SiLU of a hidden layer's accumulators -> the next layer's input, in three bf16 parts. (An activation that is not
// finite has a NaN among its parts, with which every sum of the row becomes one.)
template <int TILES>
__device__ __forceinline__ void hm_activate(__nv_bfloat16 (*dst)[kHmRows][kHmPitch], const float (&acc)[TILES][4],
                                            const float2 (&bias)[TILES], int warp, int lane) {
#pragma unroll
    for (int n = 0; n < TILES; ++n) {
        const int col = (warp * TILES + n) * 8 + (lane % 4) * 2;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint32_t w[3];
            split3(silu(acc[n][2 * half] + bias[n].x), silu(acc[n][2 * half + 1] + bias[n].y), w);
#pragma unroll
            for (int s = 0; s < kHmParts; ++s) *reinterpret_cast<uint32_t*>(&dst[s][lane / 4 + 8 * half][col]) = w[s];
        }
    }
}

// The hash function of one row by one warp in plain fp32, lane = output bit; `h`: 256 floats of scratch. For the rows that
// the matrix form cannot take, because a layer overflows, or the row or the weights hold an infinity or a NaN: they end in
// sums that are not finite (see hm_activate), which is looked for in the last layer alone and costs the others nothing (32
// sequences 4.25 us, without it 4.24; with a mark per row and hidden layer 4.41).
template <typename WT>
__device__ __forceinline__ float hm_plain_row(const __nv_bfloat16* x, float* h, const WT* W, const float* bias, int layers, int lane) {
    auto row = [&](const float* in, const WT* w, float b) {
        float s = 0.f;
#pragma unroll 1
        for (int i = 0; i < kHidden; ++i) s = fmaf(in[i], (float)w[i], s);
        return s + b;
    };
    float *in = h, *next = h + kHidden;
#pragma unroll 1
    for (int i = lane; i < kHidden; i += 32) in[i] = __bfloat162float(x[i]);
    __syncwarp();
#pragma unroll 1
    for (int l = 0; l < layers - 1; ++l) {  // W0, or W0 and W1
#pragma unroll 1
        for (int o = lane; o < kHidden; o += 32) next[o] = silu(row(in, W + (l * kHidden + o) * kHidden, __ldg(bias + l * kHidden + o)));
        __syncwarp();
        float* t = in;
        in = next;
        next = t;
    }
    const float pre = row(in, W + (2 * kHidden + lane) * kHidden, __ldg(bias + 2 * kHidden + lane));
    __syncwarp();
    return pre;
}

// Eight elements of an input row. Rows handed over for their codes alone may lie on 8-byte boundaries (the branch goes the
// same way in every thread); where K and V are appended, or attention follows, all tensors lie on 16-byte ones.
__device__ __forceinline__ uint4 hm_load16(const __nv_bfloat16* p) {
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) return *reinterpret_cast<const uint4*>(p);
    const uint2 lo = *reinterpret_cast<const uint2*>(p), hi = *reinterpret_cast<const uint2*>(p + 4);
    return make_uint4(lo.x, lo.y, hi.x, hi.y);
}

template <typename WT>
__global__ void __launch_bounds__(kHmWarps<WT> * 32, 1) hash_decode_batched_kernel(const HashDecodeParams p) {
    constexpr int kHmTiles = kHidden / (8 * kHmWarps<WT>);  // n-tiles per warp in a hidden layer: 2 or 1
    constexpr int kSplit = kHmWarps<WT> / 4;                // warps that share an n-tile of the last layer: 2 or 4
    __shared__ HmSmem sm;
    const int h = blockIdx.x, side = blockIdx.y;
    const int Hq = p.Hkv * kGroup;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kvh = h / kGroup, g = h % kGroup;
    const int b_begin = blockIdx.z * p.batch_per_cta;
    const int b_end = min(p.B, b_begin + p.batch_per_cta);
    const int half = lane >> 4, sub = lane & 15;  // a half of one of the first eight warps loads and finishes row 2 warp + half
    auto x_row = [&](int b) {
        return side == 0 ? p.q + ((size_t)b * Hq + h) * kHeadDim : p.k_new + ((size_t)b * p.Hkv + kvh) * kHeadDim;
    };

    // ---- weights and biases: constants, fetched before the dependency wait
    const WT* W = static_cast<const WT*>(p.w[side]) + (size_t)h * kMlpElems;
    const float* bias = p.bias[side] + (size_t)h * kMlpBias;
    HmWeights<WT> w0[kHmTiles][kHmBlocks], w1[kHmTiles][kHmBlocks], w2[1][kHmBlocks / kSplit];
    float2 b0[kHmTiles], b1[kHmTiles];
    const int tile2 = warp % 4, blk2 = warp / 4 * (kHmBlocks / kSplit);  // last layer: n-tile and first block of inputs
#pragma unroll
    for (int n = 0; n < kHmTiles; ++n) {
        const int row = (warp * kHmTiles + n) * 8;
        const WT* src = W + (size_t)(row + lane / 4) * kHidden + (lane % 4) * 8;
#pragma unroll
        for (int k = 0; k < kHmBlocks; ++k) {
            w0[n][k].load(src + k * 32);
            w1[n][k].load(src + kHidden * kHeadDim + k * 32);
        }
        const float* b = bias + row + (lane % 4) * 2;  // (biases may lie on any word: single loads)
        b0[n] = make_float2(__ldg(b), __ldg(b + 1));
        b1[n] = make_float2(__ldg(b + kHidden), __ldg(b + kHidden + 1));
    }
#pragma unroll
    for (int k = 0; k < kHmBlocks / kSplit; ++k)
        w2[0][k].load(W + 2 * kHidden * kHidden + (size_t)(tile2 * 8 + lane / 4) * kHidden + (blk2 + k) * 32 + (lane % 4) * 8);
    const float b2 = __ldg(bias + 2 * kHidden + lane);
    {
        // (the rows may still be written by the kernel in front: only their lines are asked for; not for rows in mapped host
        // memory, which L2 does not hold. A step of 16 sequences from host buffers takes 53.9 us with and without.)
        const int b = b_begin + 2 * warp + half;
        if (p.q_stage == nullptr && b < b_end && warp < kHmRows / 2 && sub < 2) prefetch_l2(x_row(b) + sub * (kHeadDim / 2));
    }

    pdl_wait();
    pdl_launch_dependents();

    for (int r0 = b_begin; r0 < b_end; r0 += kHmRows) {
        // (the parts of fp32 weights are made anew in every pass: kept, they would take three quarters of the registers)
#pragma unroll
        for (int n = 0; n < kHmTiles; ++n)
#pragma unroll
            for (int k = 0; k < kHmBlocks; ++k) {
                w0[n][k].pin();
                w1[n][k].pin();
            }
        // ---- the input rows, 8 elements per lane; key side: the append slot, and the V row the group's first head appends
        const int row = 2 * warp + half, b = r0 + row;
        const bool live = row < kHmRows && b < b_end;
        const bool appends = live && side == 1 && g == 0 && p.v_new != nullptr;
        uint4 raw = make_uint4(0u, 0u, 0u, 0u), v_raw = raw;
        int S = 1, page = 0;
        if (live) {
            raw = hm_load16(x_row(b) + sub * 8);
            if (appends) v_raw = *(reinterpret_cast<const uint4*>(p.v_new + ((size_t)b * p.Hkv + kvh) * kHeadDim) + sub);
            if (side == 1) {
                S = p.seq_lens[b];
                page = p.page_table[(size_t)b * p.max_pages + min(max(S - 1, 0) / kPage, p.max_pages - 1)];
            }
            if (side == 0 && p.q_stage != nullptr) *(reinterpret_cast<uint4*>(p.q_stage + ((size_t)b * Hq + h) * kHeadDim) + sub) = raw;
        }
        if (row < kHmRows) *reinterpret_cast<uint4*>(&sm.x[0][row][sub * 8]) = raw;
        __syncthreads();
        // layers: 3 = W0, W1, W2; 2 = W0, W2; 1 = W2
        float acc[kHmTiles][4], last[1][4];
        if (p.layers >= 2) {
            hm_gemm<1>(acc, sm.x, 0, w0, lane);
            hm_activate(sm.act[0], acc, b0, warp, lane);
            __syncthreads();
        }
        if (p.layers == 3) {
            hm_gemm<kHmParts>(acc, sm.act[0], 0, w1, lane);
            hm_activate(sm.act[1], acc, b1, warp, lane);
            __syncthreads();
        }
        if (p.layers == 1) hm_gemm<1>(last, sm.x, blk2, w2, lane);
        else hm_gemm<kHmParts>(last, sm.act[p.layers - 2], blk2, w2, lane);
        {
            float(*part)[kCodeBits] = sm.part[warp / 4];
            const int col = tile2 * 8 + (lane % 4) * 2;
            *reinterpret_cast<float2*>(&part[lane / 4][col]) = make_float2(last[0][0], last[0][1]);
            *reinterpret_cast<float2*>(&part[lane / 4 + 8][col]) = make_float2(last[0][2], last[0][3]);
        }
        __syncthreads();
        // ---- codes: lane = output bit, the warp's two rows; bit i = 1 iff output i > 0 (efficiency/kernels/torchatt.py:35-36:
        //      relu(sign(x))). Every buffer is written again only behind a barrier that its readers have passed.
        if (warp >= kHmRows / 2) continue;
        float pre0 = b2, pre1 = b2;
#pragma unroll
        for (int i = 0; i < kSplit; ++i) {
            pre0 += sm.part[i][2 * warp][lane];
            pre1 += sm.part[i][2 * warp + 1][lane];
        }
        if (__any_sync(0xffffffffu, !isfinite(pre0) || !isfinite(pre1))) {
            // (the activations have been read: this warp's share of their place, until it reaches the next pass's barrier)
            float* scratch = reinterpret_cast<float*>(&sm.act) + warp * 2 * kHidden;
            static_assert(sizeof(sm.act) >= kHmRows / 2 * 2 * kHidden * sizeof(float), "scratch of the first eight warps");
            if (__any_sync(0xffffffffu, !isfinite(pre0))) pre0 = hm_plain_row(sm.x[0][2 * warp], scratch, W, bias, p.layers, lane);
            if (__any_sync(0xffffffffu, !isfinite(pre1))) pre1 = hm_plain_row(sm.x[0][2 * warp + 1], scratch, W, bias, p.layers, lane);
        }
        const uint32_t code0 = __ballot_sync(0xffffffffu, pre0 > 0.0f), code1 = __ballot_sync(0xffffffffu, pre1 > 0.0f);
        const uint32_t code = half == 0 ? code0 : code1;
        if (p.preact_dbg != nullptr) {
            const int first = r0 + 2 * warp;
            if (first < b_end) p.preact_dbg[(((size_t)first * 2 + side) * Hq + h) * kCodeBits + lane] = pre0;
            if (first + 1 < b_end) p.preact_dbg[(((size_t)(first + 1) * 2 + side) * Hq + h) * kCodeBits + lane] = pre1;
        }
        if (live && side == 0) {
            if (sub == 0) p.q_codes[(size_t)b * Hq + h] = code;
        } else if (live && (S < 1 || S > p.max_pages * kPage)) {
            if (sub == 0) report(p.status, HA_ERR_BAD_SEQ_LEN);
        } else if (live && (page < 0 || page >= p.num_pages)) {
            if (sub == 0) report(p.status, HA_ERR_BAD_PAGE);
        } else if (live) {
            const size_t slot = ((size_t)page * p.Hkv + kvh) * kPage + (S - 1) % kPage;
            if (sub == 0) p.hash_pages[slot * kGroup + g] = code;
            if (appends) {  // 256 B each
                *(reinterpret_cast<uint4*>(p.k_pages + slot * kHeadDim) + sub) = raw;
                *(reinterpret_cast<uint4*>(p.v_pages + slot * kHeadDim) + sub) = v_raw;
            }
        }
        __syncwarp();
    }
}

// Prefill key-hash build on the CUDA cores, exact fp32 arithmetic: CTA (h, page, b) keeps the
// key MLP of query head h in registers and walks the tokens of one cache page.
// Follows USA.k_embedding(hard=True) over the cached keys
// (hashattention/hashattention_llama.py:204-214).
struct HashPrefillParams {
    const __nv_bfloat16* k_pages;
    uint32_t* hash_pages;
    const void* wk;
    const float* bk;
    const int32_t* page_table;
    const int32_t* seq_lens;
    const int32_t* first_token;  // [B] or null
    int32_t* status;
    int B, Hkv, max_pages, num_pages;
    int layers;  // 3, 2 or 1 Linear layers
};

template <typename WT>
__global__ void __launch_bounds__(kHashDecodeThreads)
hash_prefill_simt_kernel(const HashPrefillParams p) {
    const int h = blockIdx.x, pg = blockIdx.y, b = blockIdx.z;
    const int kvh = h / kGroup, g = h % kGroup;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    const int S = p.seq_lens[b];  // 0 is legal here: nothing cached yet, nothing to encode
    if (S < 0 || S > p.max_pages * kPage) {
        if (tid == 0 && h == 0 && pg == 0) report(p.status, HA_ERR_BAD_SEQ_LEN);
        return;
    }
    const int first = p.first_token != nullptr ? max(0, p.first_token[b]) : 0;
    const int t_begin = max(pg * kPage, first), t_end = min((pg + 1) * kPage, S);
    if (t_begin >= t_end) return;
    const int page = p.page_table[(size_t)b * p.max_pages + pg];
    if (page < 0 || page >= p.num_pages) {
        if (tid == 0) report(p.status, HA_ERR_BAD_PAGE);
        return;
    }

    MlpRegs<WT> regs;
    regs.load(static_cast<const WT*>(p.wk) + (size_t)h * kMlpElems, p.bk + (size_t)h * kMlpBias,
              warp, lane);
    __shared__ MlpSmem sm;
    pdl_wait();  // the keys may have been written by the kernel before this one

    const size_t slot0 = ((size_t)page * p.Hkv + kvh) * kPage;
    uint4 raw_next = load_x_row(p.k_pages + (slot0 + t_begin % kPage) * kHeadDim, lane);
    for (int t = t_begin; t < t_end; ++t) {
        const size_t slot = slot0 + t % kPage;
        const uint4 raw = raw_next;  // the next token's row is requested while this one is evaluated
        if (t + 1 < t_end) raw_next = load_x_row(p.k_pages + (slot + 1) * kHeadDim, lane);
        mlp_eval(regs, raw, sm, warp, lane, [] {}, p.layers);
        if (warp == 0) {
            const float pre = sm.out[lane];
            const uint32_t code = __ballot_sync(0xffffffffu, pre > 0.0f);
            if (lane == 0) p.hash_pages[slot * kGroup + g] = code;
        }
    }
}

}  // namespace ha
