// Prefill key-hash build on the 5th-generation tensor cores (tcgen05, sm_100a only), warp-specialised.
//
// For every cached key x (128 bf16) and every query head h of its kv-head the hash MLP
//     code = signbits( W2 . silu( W1 . silu( W0 x + b0 ) + b1 ) + b2 )
// is a chain of three GEMMs over a tile of 128 tokens. The (head, tile) pairs of a call, head-major, are cut
// into one contiguous range per CTA (one CTA per SM, equal cost); a CTA keeps the three weight
// matrices of its current head (72 KB bf16) in shared memory in the K-major 128-byte-swizzled layout the
// UMMA shared-memory descriptors describe, and reloads them where its range crosses into the next head.
//
// Roles of the 19 warps of a CTA:
//   * warps 0 and 1, the issuers: warp s issues the tcgen05.mma of the tiles in slot s (one elected thread of it) and
//     commits to mbarriers;
//   * warps 2-17, the epilogue: a thread owns one token row (its tensor-memory lane) and one 32-column slice of a
//     hidden layer. It reads its accumulator columns (tcgen05.ld), adds the bias, applies SiLU in fp32, splits
//     the activation into a hi and a lo bf16 (hi + lo carries 16 mantissa bits) and writes both back with
//     tcgen05.st over the columns it has just read: the next GEMM takes its A operand from tensor memory (two
//     MMAs per k-step, hi and lo against the same weights). The last 32 activations of layer 1 go to shared memory
//     instead: the 32 layer-2 columns take their place. The sign bits of a tile are packed by the four warps of one
//     slice, in turn;
//   * warp 18, the loader: one thread copies the 128 x 128 key tile (two TMA box copies, written in the same
//     swizzle) into a ring of shared-memory buffers ahead of the arithmetic.
// Two tiles are in flight, one per slot of 256 tensor-memory columns: layer 0's accumulator and activations in the first
// 128, layer 1's and the 32 of layer 2 in the others. So layer 0 of a slot's next tile needs nothing that layer 2 of the
// present one still uses, and is issued right behind layer 1. The epilogue warps take
//     layer 1 of tile j, layer 0 of tile j + 2 (the same slot), layer 1 of tile j + 1, layer 0 of tile j + 3, ...
// and find nearly every accumulator complete: a GEMM has the two phases of the other slot to run under.
//
// What bounds it: per pair of activations 3 special-function operations (24 clocks of a scheduler's unit) and about 20
// instructions, shared by four epilogue warps per scheduler (the registers allow no more): that arithmetic alone takes 28
// clocks a pair with four warps, 31 with two; in the kernel it takes about 36. At its longest the build runs into the
// 1,000 W limit. Against the form before (one issuing thread; layer 0 of the next tile behind layer 2; all 16 warps packing
// 8 bits of a tile's codes; ranges of equal tile counts), both in turn: 4 x 131072 tokens x 32 heads, repeated for seconds,
// 2889 -> 2724 us (in short bursts 1.09 x), 20011 tokens 109 -> 99, with fp32 weights 144 -> 126, the last 1000 tokens of
// 6 sequences 47.7 -> 39.3. Of that, electing the issuing thread inside the MMA's asm (operands stay in uniform registers:
// 30 clocks of issue instead of 71) gave 4 % at 20011 tokens, the ranges by cost 15 % at 6 x 1000 tokens.
// Slower: announcing activations slice by slice (four short bursts of MMAs instead of one: 0.76 x), two groups of eight
// epilogue warps taking turns (0.77 - 0.98 x), code packing in the issuing warps (0.87 - 0.98 x) or in four warps of their
// own at 80 registers (1.03 x with bf16 weights, 0.93 x with fp32), an exponential by polynomial for a quarter of the
// pairs (0.95 x), products of single values instead of pairs (0.96 x).
//
// The hi/lo split keeps the pre-activations within ~1e-6 of fp32 arithmetic, which is what makes
// the packed codes match the reference bit for bit outside the |x| < 1e-5 band.
//
// fp32 weights (hash_prefill_tc_kernel<float>) are split the same way when a head is loaded: a hi and a lo bf16 copy
// in shared memory, every GEMM multiplies by both (layer 0: X Whi + X Wlo; hidden layers: hi Whi + lo Whi + hi Wlo),
// and the key-tile ring shrinks from three tiles to one to make room.
//
// Follows USA.k_embedding(hard=True) (hashattention/hashattention_llama.py:204-214).
//
// Every wait is bounded: if a barrier never completes, the waiting thread records HA_ERR_TIMEOUT and raises a
// CTA-wide flag that ends every other wait; the CTA then waits (bounded) for the tensor core and its copies,
// frees its tensor memory and returns.
#pragma once

#include <cuda.h>  // CUtensorMap (the type only: the encoder is looked up at run time)

#include "common.cuh"

namespace ha {

constexpr int kTcEpiWarps = 16;                       // four 32-column slices x four quarters of the 128 tensor-memory lanes
constexpr int kTcEpiThreads = kTcEpiWarps * 32;
constexpr int kTcMmaWarp = 0;                         // warps 0 and 1 issue the GEMMs of slot 0 and slot 1
constexpr int kTcEpiWarp0 = 2;                        // epilogue warps kTcEpiWarp0 .. kTcEpiWarp0 + kTcEpiWarps - 1
constexpr int kTcLoadWarp = kTcEpiWarp0 + kTcEpiWarps;
constexpr int kTcThreads = (kTcLoadWarp + 1) * 32;
constexpr int kTcCodeWarps = 4;                       // warps that pack the codes of a tile: those of one column slice
constexpr int kTcTile = 128;                          // tokens per tile = TMEM lanes
constexpr uint32_t kTcBlockBytes = 128 * 128;         // one K-half of a 128-row operand: 128 rows x 128 B
constexpr uint32_t kTcW2BlockBytes = 32 * 128;        // one K-half of W2 (32 rows)
constexpr uint32_t kTcOffW0 = 0;
constexpr uint32_t kTcOffW1 = kTcOffW0 + 2 * kTcBlockBytes;
constexpr uint32_t kTcOffW2 = kTcOffW1 + 2 * kTcBlockBytes;
constexpr uint32_t kTcWBytes = kTcOffW2 + 2 * kTcW2BlockBytes;  // one copy of a head's weights: 72 KB
constexpr int kTcMaxXBufs = 3;
constexpr int kTcInfoRing = 16;  // tile records the loader keeps for the epilogue (it runs at most 8 tiles ahead of their use)
// Where the codes of a tile go: byte offset of row 0's code word in the hash pages, and the rows [row_lo, row_hi) of the
// tile that hold tokens to encode (none for a tile on a bad page). Written by the loader, read by the epilogue warps.
struct TcTileInfo {
    unsigned long long word0;
    int row_lo, row_hi;
};
static_assert(sizeof(TcTileInfo) == 16, "tile record");
// mbarriers (8 bytes each), by index.
// One "full" barrier per buffer and issuer (tile i: barrier i % (2 buffers)): an issuer waits for every phase of its barriers,
// as a test by parity needs; with one barrier per buffer it would meet every second phase only.
constexpr int kTcBarXFull = 0;                               // [2 x key-tile ring] the loader's expect-tx arrival + the bytes of the two copies
constexpr int kTcBarXEmpty = kTcBarXFull + 2 * kTcMaxXBufs;  // [key-tile ring] commit: layer 0 has read the tile
constexpr int kTcBarAcc = kTcBarXEmpty + kTcMaxXBufs;      // [2 slots][3 layers] commit: accumulator complete
constexpr int kTcBarAct = kTcBarAcc + 6;                 // [2 slots][2 layers] 16 warps: the activations of a hidden layer are written
constexpr int kTcBarRead = kTcBarAct + 4;                // [2 slots] 4 warps: the layer-2 columns are read
constexpr int kTcBarDrained = kTcBarRead + 2;            // 16 epilogue warps + 2 issuers: no GEMM reads the old weights any more
constexpr int kTcBarWeights = kTcBarDrained + 1;         // 16 epilogue warps: the next head's weights are in place
constexpr int kTcBarFinal = kTcBarWeights + 1;           // 2 commits: every GEMM of the CTA has completed
constexpr int kTcNumBars = kTcBarFinal + 1;
static_assert(kTcNumBars <= 32, "barrier block");
// Shared memory of a CTA. bf16 weights: one copy of the head's weights and a ring of three key tiles. fp32 weights are
// split into a hi and a lo bf16 copy (W = hi + lo to 16 mantissa bits; every GEMM multiplies by both), and the ring
// holds one tile.
template <bool kSplitW>
struct TcLayout {
    static constexpr int kXBufs = kSplitW ? 1 : 3;
    static constexpr uint32_t kOffWLo = kTcWBytes;  // the lo copy (split weights only)
    static constexpr uint32_t kOffX = kSplitW ? 2 * kTcWBytes : kTcWBytes;
    static constexpr uint32_t kOffAct = kOffX + kXBufs * 2 * kTcBlockBytes;   // [2 slots] the last 32 layer-1 activations of a tile
    static constexpr uint32_t kOffBias = kOffAct + 2 * kTcBlockBytes;  // 288 floats
    static constexpr uint32_t kOffBar = kOffBias + 1280;
    static constexpr uint32_t kOffTmem = kOffBar + 8 * 32;   // tmem base (4 B), abort flag (4 B)
    static constexpr uint32_t kOffInfo = kOffTmem + 16;      // ring of kTcInfoRing tile records (16 B each)
    static constexpr uint32_t kSmemBytes = kOffInfo + kTcInfoRing * 16 + 1024;  // + slack to align the base to 1024 B
    static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");
};
constexpr uint32_t kTcTmemCols = 512;
constexpr int kTcSpinLimit = 1 << 16;   // tries of a wait ...
constexpr uint32_t kTcTryNs = 20000;    // ... each of which may suspend the thread for up to this long
constexpr int kTcFinalPolls = 1 << 22;  // polls of a wait that must not give up with the others
// What the start of a head inside a CTA's range costs (drain, new weights, refill), in tiles. 6 x 1000 tokens x 32 heads
// (about 11 tiles per CTA) take 51.4 us if it is counted as 0, 49.4 as 1, 47.7 as 2 and as 3; 20011 tokens: no difference.
constexpr int kTcHeadTiles = 2;

struct HashPrefillTcParams {
    const __nv_bfloat16* k_pages;
    uint32_t* hash_pages;
    const void* wk;            // [Hq][36864] bf16 or fp32
    const float* bk;           // [Hq][288]
    const int32_t* page_table;
    const int32_t* seq_lens;
    const int32_t* first_token;  // [B] or null
    int32_t* status;
    int B, Hkv, max_pages, num_pages;
};

__device__ __forceinline__ uint32_t tc_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Byte offset of 16-byte chunk `chunk` (0..7) of row `row` inside one K-half block of a K-major
// operand with 128-byte swizzle: rows are 128 B apart, 8-row groups 1024 B apart, and the chunk
// index is XORed with the row's position in its group.
__device__ __forceinline__ uint32_t tc_swizzled(uint32_t row, uint32_t chunk) {
    return (row >> 3) * 1024u + (row & 7u) * 128u + ((chunk ^ (row & 7u)) << 4);
}

// Shared-memory matrix descriptor (K-major, SWIZZLE_128B, 8-row groups 1024 B apart) in two parts: only the low word
// depends on the address, and the descriptor of a later k-step of the operand follows by adding the k-step's offset in
// 16-byte units (the sum stays inside the address field).
__device__ __forceinline__ uint32_t tc_desc_lo(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | (1u << 16); }
__device__ __forceinline__ uint64_t tc_desc(uint32_t lo) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(64u | (1u << 14) | (2u << 29)));
    return d;
}
// k-step ks (16 inputs = 32 bytes of the 128-byte rows, four per K-half block) of an operand, in 16-byte units
__host__ __device__ constexpr uint32_t tc_koff(uint32_t ks, uint32_t block_bytes) { return (ks >> 2) * (block_bytes >> 4) + (ks & 3) * 2; }

// Instruction descriptor: bf16 x bf16 -> fp32, both operands K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t tc_idesc(uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// The warp executes these together and one elected thread of it (the same one each time) issues. Elected inside the asm,
// the operands stay warp-uniform for the compiler.
// D (tensor memory) (+)= A (shared memory) . B (shared memory)
__device__ __forceinline__ void tc_mma_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

// D (tensor memory) (+)= A (tensor memory: lane = row, two bf16 per column, K = 16 in 8 columns) . B (shared memory)
__device__ __forceinline__ void tc_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}\n" ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile(
        "{\n\t"
        ".reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
        "}\n" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Has phase `parity` of the mbarrier completed? (does not block)
__device__ __forceinline__ bool tc_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}

// Bounded wait for phase `parity` of the mbarrier; false if it ran out or another thread of the CTA gave up.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int32_t* status) {
    for (int spin = 0; spin < kTcSpinLimit; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(bar), "r"(parity), "r"(kTcTryNs) : "memory");
        if (done) return true;
        if (*abort_flag != 0) return false;
    }
    report(status, HA_ERR_TIMEOUT);
    *abort_flag = 1;
    return false;
}

// 16 accumulator columns of this thread's lane: issue, and the wait that makes the registers readable (it waits for
// every read the thread has issued). The wait takes the registers as operands, so that nothing that reads them can be
// scheduled in front of it.
__device__ __forceinline__ void tc_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tc_ld16_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :: "memory");
}

// 16 words per thread, written over the columns of this thread's lane (complete after tcgen05.wait::st) or, if to_smem, as
// four 16-byte chunks of shared memory. One asm under two predicates: as two branches of the program the compiler copies
// all 16 registers for one of them.
__device__ __forceinline__ void tc_put16(uint32_t taddr, const uint32_t (&r)[16], bool to_smem, uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %17, 0;\n\t"
        "@!p tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};\n\t"
        "@p st.shared.v4.b32 [%18], {%0, %1, %2, %3};\n\t"
        "@p st.shared.v4.b32 [%19], {%4, %5, %6, %7};\n\t"
        "@p st.shared.v4.b32 [%20], {%8, %9, %10, %11};\n\t"
        "@p st.shared.v4.b32 [%21], {%12, %13, %14, %15};\n\t}"
        :: "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
           "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
           "r"(taddr), "r"(to_smem ? 1u : 0u), "r"(s0), "r"(s1), "r"(s2), "r"(s3)
        : "memory");
}

// TMA: the box at element column x, row y of the key cache -> shared memory, bytes counted on the mbarrier (the
// copy reads this GPU's memory only and has this CTA as its single destination).
__device__ __forceinline__ void tc_tma_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}

// two fp32 -> one word of two bf16 (round to nearest even): a in the low half, b in the high half
__device__ __forceinline__ uint32_t tc_pack_bf16(float a, float b) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
    return d;
}

// Weight chunks of a head: 16 bytes of the bf16 operand each, row-major (16 per 128-wide row), the three matrices back to
// back as they are stored. Thread t of the epilogue's 512 takes chunks t, t + 512, ...: 9 in all.
constexpr int kTcWChunks = kMlpElems / 8 / kTcEpiThreads;
static_assert(kTcWChunks * kTcEpiThreads * 8 == kMlpElems, "weight chunks per thread");
// where chunk i of the head lies in shared memory: K-major, 128-byte swizzle, two K-half blocks per matrix
__device__ __forceinline__ uint32_t tc_w_offset(int i) {
    const uint32_t row = (uint32_t)i >> 4, c16 = (uint32_t)i & 15u;  // rows 0..127: W0, 128..255: W1, 256..287: W2
    const uint32_t base = row < 128 ? kTcOffW0 : (row < 256 ? kTcOffW1 : kTcOffW2);
    return base + (c16 >> 3) * (row < 256 ? kTcBlockBytes : kTcW2BlockBytes) + tc_swizzled(row < 256 ? row & 127u : row - 256u, c16 & 7u);
}
// All of a thread's loads are issued before the first store (fp32 weights: in three parts, for the registers).
__device__ __forceinline__ void tc_load_weights(unsigned char* dst, unsigned char*, const __nv_bfloat16* W, int t) {
    uint4 v[kTcWChunks];
#pragma unroll
    for (int j = 0; j < kTcWChunks; ++j) v[j] = __ldg(reinterpret_cast<const uint4*>(W) + t + j * kTcEpiThreads);
#pragma unroll
    for (int j = 0; j < kTcWChunks; ++j) *reinterpret_cast<uint4*>(dst + tc_w_offset(t + j * kTcEpiThreads)) = v[j];
}
// fp32 weights become a hi and a lo bf16 (hi + lo carries 16 mantissa bits), written to two copies of the operands.
__device__ __forceinline__ void tc_load_weights(unsigned char* dst, unsigned char* dst_lo, const float* W, int t) {
#pragma unroll
    for (int part = 0; part < 3; ++part) {
        float4 v[2 * kTcWChunks / 3];
#pragma unroll
        for (int j = 0; j < kTcWChunks / 3; ++j) {
            const float4* src = reinterpret_cast<const float4*>(W) + 2 * (t + (part * (kTcWChunks / 3) + j) * kTcEpiThreads);
            v[2 * j] = __ldg(src);
            v[2 * j + 1] = __ldg(src + 1);
        }
#pragma unroll
        for (int j = 0; j < kTcWChunks / 3; ++j) {
            const float w[8] = {v[2 * j].x, v[2 * j].y, v[2 * j].z, v[2 * j].w, v[2 * j + 1].x, v[2 * j + 1].y, v[2 * j + 1].z, v[2 * j + 1].w};
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                hi[k] = tc_pack_bf16(w[2 * k], w[2 * k + 1]);
                lo[k] = tc_pack_bf16(w[2 * k] - bf16_lo(hi[k]), w[2 * k + 1] - bf16_hi(hi[k]));
            }
            const uint32_t off = tc_w_offset(t + (part * (kTcWChunks / 3) + j) * kTcEpiThreads);
            *reinterpret_cast<uint4*>(dst + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(dst_lo + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
    }
}

// bias + SiLU + hi/lo split of 16 accumulator columns v (bit patterns of fp32) of one row. The 16 words that take their
// place are the A operand of one k-step of the next GEMM: words 0..7 hold the hi halves of the activations (two per
// word, the even one in the low half), words 8..15 their lo halves.
__device__ __forceinline__ void tc_activate16(const uint32_t (&v)[16], const float* bias, uint32_t (&out)[16]) {
    const f32x2 nlog2e = pack2(-1.4426950408889634f, -1.4426950408889634f), one = pack2(1.0f, 1.0f);
#pragma unroll
    for (int pr = 0; pr < 8; ++pr) {
        const float2 bb = *reinterpret_cast<const float2*>(bias + 2 * pr);  // the same address in every lane: a broadcast
        const f32x2 x = add2(pack2(__uint_as_float(v[2 * pr]), __uint_as_float(v[2 * pr + 1])), pack2(bb.x, bb.y));
        float t0, t1;
        unpack2(mul2(x, nlog2e), t0, t1);
        // SiLU x / (1 + e^-x) with the hardware exp2 and ONE reciprocal for the pair: 1 / (a0 a1) times a1 and a0.
        // e is held below 2^60 so that the product stays finite (the activation is below 1e-16 in magnitude there).
        float e0, e1, r;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(fminf(t0, 60.0f)));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(fminf(t1, 60.0f)));
        float a0, a1;
        unpack2(add2(pack2(e0, e1), one), a0, a1);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a0 * a1));
        const f32x2 y = mul2(x, mul2(pack2(a1, a0), pack2(r, r)));
        float y0, y1;
        unpack2(y, y0, y1);
        const uint32_t hi = tc_pack_bf16(y0, y1);
        float l0, l1;  // y - hi, exact: the multiply-add takes the bf16 halves of hi as they are
        asm("{\n\t.reg .b16 h0, h1;\n\tmov.b32 {h0, h1}, %2;\n\t"
            "fma.rn.f32.bf16 %0, h0, %3, %4;\n\tfma.rn.f32.bf16 %1, h1, %3, %5;\n\t}"
            : "=f"(l0), "=f"(l1) : "r"(hi), "h"((unsigned short)0xBF80), "f"(y0), "f"(y1));
        out[pr] = hi;
        out[pr + 8] = tc_pack_bf16(l0, l1);
    }
}

// The (head, token tile) pairs of the whole call, head-major and counting only tiles that hold tokens to encode, are cut
// into gridDim.x contiguous ranges of equal cost: a tile costs 1, and so that a CTA whose range crosses into the next head
// (drain, new weights, refill) gets fewer tiles, the start of a head costs kTcHeadTiles. Unless there are no more tiles than
// CTAs: then equal counts give each of them one tile at most, while ranges by cost give some of them two (96 tiles, 3 x 100
// tokens x 32 heads, equal counts / by cost: 12.4 / 13.5 us, with fp32 weights 13.9 / 15.7).
__device__ __forceinline__ void tc_seq_tiles(const HashPrefillTcParams& p, int b, bool reporter, int& S, int& first, int& lo, int& hi) {
    // a sequence's tiles to encode: [first_token / 128, ceil(S / 128)); none if its length is out of range
    S = __ldg(p.seq_lens + b);
    first = p.first_token != nullptr ? max(0, __ldg(p.first_token + b)) : 0;
    if (S < 0 || S > p.max_pages * kPage) {
        if (reporter) report(p.status, HA_ERR_BAD_SEQ_LEN);
        S = 0;
    }
    lo = first / kTcTile;
    hi = max(lo, (S + kTcTile - 1) / kTcTile);
}
struct TcRange {
    int head0, rem0, head1, rem1;  // the CTA's range starts rem0 / gridDim.x into head head0, ends rem1 / gridDim.x into head1
    int per_head, total;           // tiles per head; tiles of the range
    int skip, first_end;           // tiles of head0 in front of the range; end of head0, in tiles of the range
    // what does not depend on the sequences
    __device__ explicit TcRange(int Hq) {
        head0 = Hq * (int)blockIdx.x / (int)gridDim.x;
        rem0 = Hq * (int)blockIdx.x - head0 * (int)gridDim.x;
        head1 = Hq * ((int)blockIdx.x + 1) / (int)gridDim.x;
        rem1 = Hq * ((int)blockIdx.x + 1) - head1 * (int)gridDim.x;
    }
    // tiles of head h in front of the place rem / gridDim.x into it. A head that starts inside a CTA's range has
    // kTcHeadTiles empty places in front (none if a CTA has one tile at most).
    static __device__ int before(long long per_head, int h, int Hq, int rem) {
        const bool one_each = per_head * Hq <= (long long)gridDim.x;
        const int empty = one_each || (long long)h * (int)gridDim.x % Hq == 0 ? 0 : kTcHeadTiles;
        const long long places = per_head + empty;
        const long long at = places < (1ll << 32) / 65536 ? (long long)((uint32_t)places * (uint32_t)rem / gridDim.x) : places * rem / gridDim.x;
        return (int)max(0ll, at - empty);
    }
    // by a whole warp, lane = sequence
    __device__ void count(const HashPrefillTcParams& p, int lane, bool reporter) {
        long long T = 0;
        for (int b = lane; b < p.B; b += 32) {
            int S, first, lo, hi;
            tc_seq_tiles(p, b, reporter, S, first, lo, hi);
            T += hi - lo;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) T += __shfl_xor_sync(0xffffffffu, T, d);
        const int Hq = p.Hkv * kGroup;
        skip = before(T, head0, Hq, rem0);
        total = (int)((head1 - head0) * T + before(T, head1, Hq, rem1) - skip);
        per_head = (int)T;
        first_end = per_head - skip;
    }
};

// Walks over the tiles of a CTA's range (one thread; built by the whole warp).
struct TcItem {
    int h, S, first, t0, store;
    size_t slot0;  // (page * Hkv + kv head) * page size + offset of the tile's first token
};
struct TcCursor {
    const HashPrefillTcParams& p;
    int h, b, tile, hi, S, first;
    __device__ TcCursor(const HashPrefillTcParams& p_, const TcRange& r, int lane) : p(p_), h(r.head0), b(0), tile(0), hi(0), S(0), first(0) {
        // the sequence in which tile r.skip of the head lies
        long long before = 0;
        for (int b0 = 0; b0 < p.B && r.total > 0; b0 += 32) {
            int S_ = 0, first_ = 0, lo = 0, hi_ = 0;
            if (b0 + lane < p.B) tc_seq_tiles(p, b0 + lane, true, S_, first_, lo, hi_);
            long long incl = hi_ - lo;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const long long u = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += u;
            }
            const uint32_t reached = __ballot_sync(0xffffffffu, before + incl > r.skip);
            if (reached != 0) {
                const int l = __ffs(reached) - 1;
                const int at = lo + (int)(r.skip - (before + incl - (hi_ - lo)));
                b = b0 + l;
                tile = __shfl_sync(0xffffffffu, at, l);
                hi = __shfl_sync(0xffffffffu, hi_, l);
                S = __shfl_sync(0xffffffffu, S_, l);
                first = __shfl_sync(0xffffffffu, first_, l);
                break;
            }
            before += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    // The next tile (to be called `total` times). A tile on a bad page is reported, read from page 0 and not stored.
    __device__ TcItem next() {
        const int Hq = p.Hkv * kGroup;
        for (int guard = 0; tile >= hi && guard <= p.B * Hq; ++guard) {  // on to the next sequence, or the next head
            if (++b >= p.B) {
                b = 0;
                ++h;
            }
            int lo;
            tc_seq_tiles(p, b, true, S, first, lo, hi);
            tile = lo;
        }
        TcItem it;
        it.h = min(h, Hq - 1); it.S = S; it.first = first; it.t0 = tile * kTcTile; it.store = tile < hi ? 1 : 0;
        int page = __ldg(p.page_table + (size_t)b * p.max_pages + min(it.t0 / kPage, p.max_pages - 1));
        ++tile;
        if (page < 0 || page >= p.num_pages) {
            report(p.status, HA_ERR_BAD_PAGE);
            page = 0;
            it.store = 0;
        }
        it.slot0 = ((size_t)page * p.Hkv + it.h / kGroup) * kPage + it.t0 % kPage;
        return it;
    }
};

template <typename WT>
__global__ void __launch_bounds__(kTcThreads, 1) hash_prefill_tc_kernel(const HashPrefillTcParams p,
                                                                        const __grid_constant__ CUtensorMap k_map) {
    constexpr bool kSplitW = sizeof(WT) == 4;  // fp32 weights: hi and lo copies, every GEMM multiplies by both
    using L = TcLayout<kSplitW>;
    constexpr int kTcXBufs = L::kXBufs;
    constexpr uint32_t kTcOffX = L::kOffX, kTcOffBias = L::kOffBias, kTcOffBar = L::kOffBar, kTcOffTmem = L::kOffTmem;
    constexpr uint32_t kTcOffInfo = L::kOffInfo;
    extern __shared__ unsigned char tc_smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Hq = p.Hkv * kGroup;
    float* s_bias = reinterpret_cast<float*>(smem + kTcOffBias);
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + kTcOffTmem);
    volatile int* s_abort = reinterpret_cast<volatile int*>(smem + kTcOffTmem + 4);
    TcTileInfo* s_info = reinterpret_cast<TcTileInfo*>(smem + kTcOffInfo);
    const uint32_t sbase = tc_smem_u32(smem);
    const uint32_t bars = sbase + kTcOffBar;
    auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };

    // The weights of head h, by thread t of the epilogue. The first head of a CTA follows from its index alone, so its
    // weights are fetched before the dependency wait.
    auto load_head = [&](int h, int t) {
        tc_load_weights(smem, smem + L::kOffWLo, static_cast<const WT*>(p.wk) + (size_t)h * kMlpElems, t);
        if (t < kMlpBias) s_bias[t] = __ldg(p.bk + (size_t)h * kMlpBias + t);
    };
    TcRange range(Hq);
    if (warp >= kTcEpiWarp0 && warp < kTcLoadWarp) load_head(range.head0, tid - kTcEpiWarp0 * 32);
    if (tid == 0) {
        auto init = [&](int first, int n, uint32_t count) {
            for (int i = first; i < first + n; ++i)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar(i)), "r"(count));
        };
        init(kTcBarXFull, 2 * kTcMaxXBufs, 1);
        init(kTcBarXEmpty, kTcMaxXBufs, 1);
        init(kTcBarAcc, 6, 1);
        init(kTcBarAct, 4, kTcEpiWarps);
        init(kTcBarRead, 2, kTcCodeWarps);
        init(kTcBarDrained, 1, kTcEpiWarps + 2);
        init(kTcBarWeights, 1, kTcEpiWarps);
        init(kTcBarFinal, 1, 2);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kTcMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(s_tmem)), "r"(kTcTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *s_tmem;
    pdl_wait();  // the weights above are constants; everything below may depend on the previous kernel

    // every lane waits for itself; the warp then agrees, so that the warp-wide instructions that follow are never
    // executed by a part of it
    auto wait = [&](int b, uint32_t parity) {
        const bool ok = tc_wait(bar(b), parity, s_abort, p.status);
        return __all_sync(0xffffffffu, ok) != 0;
    };

    range.count(p, lane, warp == kTcLoadWarp);
    const int total = range.total, per_head = range.per_head, first_end = range.first_end;

    if (warp >= kTcEpiWarp0 && warp < kTcLoadWarp) {
        // ---- epilogue warps ----------------------------------------------------------------------------------
        const uint32_t sl = (uint32_t)(warp - kTcEpiWarp0) >> 2;  // this warp's 32-column slice of a hidden layer
        const uint32_t row = (uint32_t)(warp & 3) * 32 + lane;    // token row of the tile = tensor-memory lane
        const uint32_t t_base = tmem + (((uint32_t)(warp & 3) * 32u) << 16);
        uint32_t changes = 0;
        bool ok = true, have = false;  // have: the first half of the next phase's slice has been requested
        uint32_t rx[16], ry[16];
        auto slice_col = [&](uint32_t slot, uint32_t layer) { return t_base + slot * 256u + layer * 128u + 32u * sl; };
        // One hidden layer of the slot's tile number k: this warp's slice of the accumulator -> hi/lo activations, in two halves
        // of 16 columns, rx and ry. Each is requested one half ahead of its arithmetic, the first one in the middle of the
        // phase before if its accumulator is complete by then (`have`).
        auto hidden = [&](uint32_t slot, uint32_t layer, uint32_t k, bool want_next, uint32_t next_slot, uint32_t next_layer, uint32_t next_k) {
            const uint32_t col = slice_col(slot, layer);
            if (!have) {
                if (!wait(kTcBarAcc + 3 * (int)slot + (int)layer, k & 1)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                tc_ld16_issue(col, rx);
            }
            const float* bias = s_bias + layer * kHidden + 32 * sl;
            const bool to_smem = layer == 1 && sl == 3;
            // k-steps 6 and 7 of layer 2's A operand: hi halves in chunks 0-1 and 2-3 of the row, lo halves in 4-5 and 6-7
            const uint32_t chunk0 = sbase + L::kOffAct + slot * kTcBlockBytes + tc_swizzled(row, 0);
            uint32_t out[16];
            tc_ld16_wait(rx);
            tc_ld16_issue(col + 16u, ry);
            tc_activate16(rx, bias, out);
            tc_put16(col, out, to_smem, chunk0, chunk0 ^ 0x10u, chunk0 ^ 0x40u, chunk0 ^ 0x50u);
            tc_ld16_wait(ry);
            have = false;
            if (want_next && __all_sync(0xffffffffu, tc_test(bar(kTcBarAcc + 3 * (int)next_slot + (int)next_layer), next_k & 1)) != 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                tc_ld16_issue(slice_col(next_slot, next_layer), rx);
                have = true;
            }
            tc_activate16(ry, bias + 16, out);
            tc_put16(col + 16u, out, to_smem, chunk0 ^ 0x20u, chunk0 ^ 0x30u, chunk0 ^ 0x60u, chunk0 ^ 0x70u);
            if (to_smem) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(bar(kTcBarAct + 2 * (int)slot + (int)layer));
            return true;
        };
        // The codes of tile i, number k of its slot: thread = token row. Where they go is in the tile's record (read behind the
        // wait, which orders it behind the loader's write). Only every second phase of the barrier is waited for here, but
        // the one before is known to be complete: layer 1 of this tile was issued behind the arrivals below.
        auto codes = [&](uint32_t slot, uint32_t k, int i) {
            if (!wait(kTcBarAcc + 3 * (int)slot + 2, k & 1)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t col = t_base + slot * 256u + 224u;
            uint32_t r[16];  // (rx may hold the next phase's columns)
            tc_ld16_issue(col, ry);
            tc_ld16_issue(col + 16u, r);
            tc_ld16_wait(ry);
            tc_ld16_wait(r);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(bar(kTcBarRead + (int)slot));
            const TcTileInfo info = s_info[i % kTcInfoRing];
            const float4* b2 = reinterpret_cast<const float4*>(s_bias + 2 * kHidden);
            uint32_t code = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float4 bb = b2[q];
                const uint32_t* w = q < 4 ? ry + 4 * q : r + 4 * (q - 4);
                code |= (__uint_as_float(w[0]) + bb.x > 0.0f ? 1u : 0u) << (4 * q);
                code |= (__uint_as_float(w[1]) + bb.y > 0.0f ? 2u : 0u) << (4 * q);
                code |= (__uint_as_float(w[2]) + bb.z > 0.0f ? 4u : 0u) << (4 * q);
                code |= (__uint_as_float(w[3]) + bb.w > 0.0f ? 8u : 0u) << (4 * q);
            }
            if ((int)row >= info.row_lo && (int)row < info.row_hi)
                *reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(p.hash_pages) + info.word0 + row * (kGroup * 4)) = code;
            return true;
        };
        uint32_t k_cur = 0, k_oth = 0;  // tiles in front of the one at hand in its slot, and of the following one in the other slot
        for (int s0 = 0, seg = 0; s0 < total && ok; ++seg) {
            const int s1 = min(total, s0 == 0 ? first_end : s0 + per_head);  // end of this head's tiles
            if (s0 > 0) {
                // the weights change: the issuers and every epilogue warp meet (all GEMMs of the old head have completed and
                // its codes are packed), then the epilogue warps load together
                __syncwarp();
                if (lane == 0) tc_arrive(bar(kTcBarDrained));
                if (!(ok = wait(kTcBarDrained, changes & 1))) break;
                load_head(range.head0 + seg, tid - kTcEpiWarp0 * 32);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc_arrive(bar(kTcBarWeights));
                if (!(ok = wait(kTcBarWeights, changes & 1))) break;
                ++changes;
            }
            // tile j of the head is in slot j % 2; rounds -2 and -1 only start the first two tiles
            const int n = s1 - s0;
            uint32_t slot = 0;
            --k_cur;
            --k_oth;
            for (int j = -2; j < n && ok; ++j) {
#pragma unroll 1
                for (int layer = j >= 0 ? 1 : 0; layer >= (j + 2 < n ? 0 : 1) && ok; --layer) {
                    const bool same = layer == 1 && j + 2 < n;            // next: layer 0 of the slot's next tile
                    const bool other = !same && j + 1 >= 0 && j + 1 < n;  // next: layer 1 of the other slot's tile
                    ok = hidden(slot, (uint32_t)layer, layer == 1 ? k_cur : k_cur + 1, same || other, same ? slot : slot ^ 1u,
                                same ? 0u : 1u, same ? k_cur + 1 : k_oth);
                }
                if (ok && j >= 0 && ((uint32_t)(s0 + j) & 3u) == sl) ok = codes(slot, k_cur, s0 + j);
                const uint32_t k = k_cur + 1;  // on to the other slot
                k_cur = k_oth;
                k_oth = k;
                slot ^= 1u;
            }
            if (slot != 0) {  // the next head starts in slot 0 whatever the number of tiles
                const uint32_t k = k_cur;
                k_cur = k_oth;
                k_oth = k;
            }
            s0 = s1;
        }
    } else if (warp < kTcEpiWarp0) {
        // ---- issuers: all lanes run the loop with the same values, one elected thread issues ---------------------
        const uint32_t slot = __shfl_sync(0xffffffffu, (uint32_t)warp, 0);
        const uint32_t w0_lo = tc_desc_lo(sbase + kTcOffW0), w1_lo = tc_desc_lo(sbase + kTcOffW1);
        const uint32_t w2_lo = tc_desc_lo(sbase + kTcOffW2), x_lo = tc_desc_lo(sbase + kTcOffX);
        const uint32_t act_lo = tc_desc_lo(sbase + L::kOffAct + slot * kTcBlockBytes);
        constexpr uint32_t kWLo = L::kOffWLo >> 4;  // from a descriptor of the hi copy to the lo copy
        const uint32_t r0 = __shfl_sync(0xffffffffu, tmem, 0) + slot * 256u, r1 = r0 + 128u, d3 = r1 + 96u;
        uint32_t changes = 0, k = 0;  // head changes; tiles of the slot so far
        bool ok = true;
        auto wait_mma = [&](int b, uint32_t parity) {
            const bool done = wait(b, parity);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return done;
        };
        auto layer0 = [&](int i) {
            const uint32_t buf = (uint32_t)i % kTcXBufs;
            if (!wait_mma(kTcBarXFull + i % (2 * kTcXBufs), ((uint32_t)i / (2 * kTcXBufs)) & 1)) return false;
            const uint32_t xb = x_lo + buf * (2 * kTcBlockBytes >> 4);
#pragma unroll
            for (uint32_t ks = 0; ks < 8; ++ks) {
                const uint64_t xdesc = tc_desc(xb + tc_koff(ks, kTcBlockBytes));
                tc_mma_ss(r0, xdesc, tc_desc(w0_lo + tc_koff(ks, kTcBlockBytes)), tc_idesc(128), ks == 0 ? 0u : 1u);
                if constexpr (kSplitW)
                    tc_mma_ss(r0, xdesc, tc_desc(w0_lo + kWLo + tc_koff(ks, kTcBlockBytes)), tc_idesc(128), 1u);
            }
            tc_commit(bar(kTcBarXEmpty + (int)buf));
            tc_commit(bar(kTcBarAcc + 3 * (int)slot + 0));
            return true;
        };
        for (int s0 = 0; s0 < total && ok;) {
            const int s1 = min(total, s0 == 0 ? first_end : s0 + per_head);
            if (s0 > 0) {  // the next head's weights
                if (lane == 0) tc_arrive(bar(kTcBarDrained));
                if (!(ok = wait_mma(kTcBarWeights, changes & 1))) break;
                ++changes;
            }
            if (s0 + (int)slot < s1) ok = layer0(s0 + (int)slot);
            for (int i = s0 + (int)slot; i < s1 && ok; i += 2, ++k) {
                // layer 1 overwrites the columns of the last tile's layer 2
                if (k > 0 && !(ok = wait_mma(kTcBarRead + (int)slot, (k - 1) & 1))) break;
                if (!(ok = wait_mma(kTcBarAct + 2 * (int)slot, k & 1))) break;
#pragma unroll
                for (uint32_t ks = 0; ks < 8; ++ks) {
                    const uint32_t b_lo = w1_lo + tc_koff(ks, kTcBlockBytes);
                    tc_mma_ts(r1, r0 + 16 * ks, tc_desc(b_lo), tc_idesc(128), ks == 0 ? 0u : 1u);
                    tc_mma_ts(r1, r0 + 16 * ks + 8, tc_desc(b_lo), tc_idesc(128), 1u);
                    if constexpr (kSplitW) tc_mma_ts(r1, r0 + 16 * ks, tc_desc(b_lo + kWLo), tc_idesc(128), 1u);  // hi activations x lo weights
                }
                tc_commit(bar(kTcBarAcc + 3 * (int)slot + 1));
                // layer 0 of the slot's next tile follows in the tensor core's order: its accumulator takes the columns
                // layer 1 has just read its activations from
                if (i + 2 < s1 && !(ok = layer0(i + 2))) break;
                if (!(ok = wait_mma(kTcBarAct + 2 * (int)slot + 1, k & 1))) break;
#pragma unroll
                for (uint32_t ks = 0; ks < 8; ++ks) {
                    const uint32_t b_lo = w2_lo + tc_koff(ks, kTcW2BlockBytes);
                    if (ks < 6) {
                        tc_mma_ts(d3, r1 + 16 * ks, tc_desc(b_lo), tc_idesc(32), ks == 0 ? 0u : 1u);
                        tc_mma_ts(d3, r1 + 16 * ks + 8, tc_desc(b_lo), tc_idesc(32), 1u);
                        if constexpr (kSplitW) tc_mma_ts(d3, r1 + 16 * ks, tc_desc(b_lo + kWLo), tc_idesc(32), 1u);
                    } else {  // the last 32 activations are in shared memory: hi of both k-steps, then lo
                        const uint32_t a_lo = act_lo + (ks - 6) * 2;
                        tc_mma_ss(d3, tc_desc(a_lo), tc_desc(b_lo), tc_idesc(32), 1u);
                        tc_mma_ss(d3, tc_desc(a_lo + 4), tc_desc(b_lo), tc_idesc(32), 1u);
                        if constexpr (kSplitW) tc_mma_ss(d3, tc_desc(a_lo), tc_desc(b_lo + kWLo), tc_idesc(32), 1u);
                    }
                }
                tc_commit(bar(kTcBarAcc + 3 * (int)slot + 2));
            }
            s0 = s1;
        }
        // the tensor core has finished everything issued above (after a time-out: one more bounded wait)
        tc_commit(bar(kTcBarFinal));
        for (int spin = 0; spin < kTcFinalPolls && __all_sync(0xffffffffu, tc_test(bar(kTcBarFinal), 0)) == 0; ++spin) {}
    } else {
        // ---- loader ------------------------------------------------------------------------------------------
        // One thread: a tile is two TMA box copies (the two K-halves, 64 elements x 128 rows each, written in the
        // 128-byte swizzle) that complete on a barrier; the ring runs ahead of the arithmetic.
        TcCursor cur(p, range, lane);
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&k_map) : "memory");
            int i = 0;
            for (; i < total; ++i) {
                const uint32_t buf = (uint32_t)i % kTcXBufs;
                const TcItem it = cur.next();
                if (!tc_wait(bar(kTcBarXEmpty + (int)buf), ((uint32_t)(i / kTcXBufs) & 1) ^ 1, s_abort, p.status)) break;
                {  // the tile's record for the code warps, published by the arrival below
                    TcTileInfo info;
                    info.word0 = ((unsigned long long)it.slot0 * kGroup + (unsigned)(it.h % kGroup)) * 4ull;
                    info.row_lo = max(0, it.first - it.t0);
                    info.row_hi = it.store ? min(kTcTile, it.S - it.t0) : 0;
                    s_info[i % kTcInfoRing] = info;
                }
                const uint32_t full = bar(kTcBarXFull + i % (2 * kTcXBufs)), dst = sbase + kTcOffX + buf * 2 * kTcBlockBytes;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"(2 * kTcBlockBytes) : "memory");
                tc_tma_load(dst, &k_map, 0, (int)it.slot0, full);
                tc_tma_load(dst + kTcBlockBytes, &k_map, 64, (int)it.slot0, full);
            }
            // no copy is left in flight when the CTA ends (they have all landed unless the CTA gave up early)
            for (int j = max(0, i - kTcXBufs); j < i; ++j)
                for (int spin = 0; spin < kTcFinalPolls && !tc_test(bar(kTcBarXFull + j % (2 * kTcXBufs)), (uint32_t)(j / (2 * kTcXBufs)) & 1); ++spin) {}
        }
        __syncwarp();
    }

    // ---- release tensor memory ---------------------------------------------------------------------------
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kTcMmaWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcTmemCols) : "memory");
    }
}

}  // namespace ha
