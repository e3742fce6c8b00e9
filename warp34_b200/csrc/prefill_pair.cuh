// Chunked-prefill attention on the 5th-generation tensor cores at the accuracy of fp32 dequant-then-attend:
// every operand is fed to tcgen05.mma as fp16 value + fp16 rounding residual.  Included by tq4_attention.cu
// (shares the PTX wrappers, the geometry helpers and the epilogue).
//
// Replaces paged_attention_prefill_mma_f16_kernel<64 / 128> (crates/warp34-kernels/csrc/ops/
// op_paged_attn.cu:594-1128) for head_dim 256, 16-token pages, canonical packing of TQ4, FP8 E4M3 or Q8_0 rows.
//
// A cluster of two CTAs (cta_group::2, one SM each) owns 256 query rows (256 / gqa tokens x gqa heads of one kv
// head), 128 rows per CTA, and walks the keys its rows can see in blocks of 64.  The two SMs share every K and V
// tile: each CTA dequantises half of it (K: 32 of the 64 keys; V: 128 of the 256 channels) and the MMA reads both
// halves, so a code is dequantised once per 256 query rows.
//
//   warps 0-3   consumers: thread = query row = TMEM lane: scores from TMEM, online softmax with a lazily moved
//               reference maximum, P written over the scores it came from as fp16 value and residual (16 columns each per 32 keys)
//   warps 4-7   K producers, warps 8-11 V producers: lane = key, warp = 32 of the stage's 128 channels
//   warp 12     (CTA 0) issues every MMA; the scores of block j + 1 ahead of the output product of block j
//   warp 13     bulk-copies the raw (page, head) runs
//
//   S[256 x 64]   = Q'hi Khi^T + Q'lo Khi^T + Q'hi Klo^T      A in TMEM (Q'hi) or shared memory (Q'lo)
//   O[256 x 256] += Phi Vhi + Plo Vhi + Phi Vlo               A in TMEM
//
// K and V elements are row scale x centroid (or code): hi = fp16(d c), lo = fp16(d c - hi), about 22 bits together as long as
// lo is not far below fp16's normal range.  Where a sample of a tile's rows is small (PpScales: below about 2^-3), K or V
// is therefore held divided by a power of two for the whole tile, which the consumers take out again in fp32: a factor
// of the scores for K, of the normalised output for V.  (Without it 21 % of the outputs of a TQ4 chunk over K of magnitude 2^-10
// under Q of magnitude 2^10 were not the nearest fp16 value, against 3 % at magnitude 1, and one missed 2e-3 + 1e-2 |b| by 16 %.
// A power of two for every key or every 32 keys took 10 to 35 % more time on long contexts: each block then waits for its scales.)
// What bounds it: the tensor pipe under the power cap.  Six (TQ4) or five (8-bit) products per visible pair instead of
// two; 8 x 2048 tokens after 8192 (16 / 4 heads) take 5.6 ms = 440 TFLOP/s of attention = 1320 TFLOP/s issued, against
// 21.6 ms for register MMAs (mma.sync) over the same operands.  A pair rather than one CTA because dequantising once per
// 128 rows would cost as many shared-memory cycles as the MMAs take.  The MMAs are issued by one elected thread
// (elect.sync; with `lane == 0` as the condition each issue took about 45 cycles and the kernel 6.4 ms), and cross-CTA
// arrivals use the default semantics (cluster-scope release / acquire put a memory barrier in front of each).
// For 8-bit layers the query is neither rotated nor scaled: it is the fp16 operand as it arrives and has no residual.
#pragma once

namespace w34 {

constexpr int kPpRows = 256;                         // query rows of a pair
constexpr int kPpCtaRows = 128;
constexpr int kPpKeys = 64;                          // keys of a block = 4 pages
constexpr int kPpWarps = 14;
constexpr int kPpThreads = kPpWarps * 32;
constexpr int kPpStages = 3;                         // half-block stages of K and of V
constexpr uint32_t kPpPart = 2u * 32u * 128u;        // 8192: [2 blocks of 64 channels][32 keys][128 B], value or residual
constexpr uint32_t kPpStage = 2u * kPpPart;          // value + residual
constexpr uint32_t kPpQLoBytes = 4u * kPpCtaRows * 128u;   // 65536: [4 blocks of 64 channels][128 rows][128 B]
constexpr uint32_t kPpLutBytes = 256u * 128u;        // byte -> (value pair, residual pair), 16 lane copies of 8 bytes
constexpr int kPpRawStages = 2;
// Table factor: close to the fp16 grid (see kLutScale), and small enough that scale x centroid stays finite for every
// fp16 scale.
constexpr float kPpLutScale = 0.25f * kLutScale;
constexpr float kPpRescaleThreshold = 8.0f;          // log2 units: the reference maximum may lag by this much
constexpr float kPpShift = 6.0f;                     // P is carried times 2^6: at most 2^14, subnormal only below 2^-20
constexpr uint32_t kPpColO = 0, kPpColS = 256, kPpColQ = 384;
constexpr int kPpOutStride = 260;                    // floats per row of the epilogue staging: 256 columns, l, m
constexpr int kPpMaxSplits = 24;                     // at most 32: a lane per split in the merge

template <int FMT> struct PpFormat;
// has_keys: whether a row of mass l has a result.  A row whose query or keys hold a NaN has a NaN mass: it comes out as NaN on TQ4
// layers and as zeros on 8-bit ones, as it does from the kernels that serve smaller batches of them.
template <> struct PpFormat<WARP34_KV_FORMAT_TQ4> {
    static constexpr uint32_t kRow = kTq4RowBytes;
    static constexpr bool kRotated = true;
    static __device__ __forceinline__ bool has_keys(float l) { return !(l <= 0.0f); }
};
template <> struct PpFormat<WARP34_KV_FORMAT_FP8_E4M3> {
    static constexpr uint32_t kRow = kHeadDim + 8;
    static constexpr bool kRotated = false;
    static __device__ __forceinline__ bool has_keys(float l) { return l > 0.0f; }
};
template <> struct PpFormat<WARP34_KV_FORMAT_Q8_0> {
    static constexpr uint32_t kRow = 4 * 68;
    static constexpr bool kRotated = false;
    static __device__ __forceinline__ bool has_keys(float l) { return l > 0.0f; }
};

// A row's scales, as bits: non-negative floats order like them.
template <int FMT> struct PpScales {
    static constexpr uint32_t kFirst = FMT == WARP34_KV_FORMAT_FP8_E4M3 ? (uint32_t)kHeadDim : 0u;
    // How large a row is, from its scale: about its root mean square (TQ4: the centroids' is 1/16), or its largest element.
    static __device__ __forceinline__ float magnitude(uint32_t bits) {
        if (FMT == WARP34_KV_FORMAT_TQ4) return __half2float(__ushort_as_half((unsigned short)bits)) * 0.0625f;
        return __uint_as_float(bits) * (FMT == WARP34_KV_FORMAT_FP8_E4M3 ? 448.0f : 127.0f);
    }
    // The first scale of a row in global memory, without its sign.
    static __device__ __forceinline__ uint32_t first(const uint8_t* row) {
        return FMT == WARP34_KV_FORMAT_TQ4 ? *reinterpret_cast<const uint16_t*>(row + kFirst) & 0x7fffu : *reinterpret_cast<const uint32_t*>(row + kFirst) & 0x7fffffffu;
    }
    // The exponent of the power of two by which rows of this magnitude are divided: 0 from 2^-3 on (the tile of a TQ4 row holds a
    // quarter of it, and the residual's step of 2^-24 is then 2^-19 of a typical element; of an 8-bit row's largest element it is 2^-21),
    // so that ordinary activations pass as they are, and for zeros, NaN and infinities; smaller rows are brought to [1, 2).
    static __device__ __forceinline__ int exponent(uint32_t bits) {
        const float m = magnitude(bits);
        return m > 0.0f && m < 0.125f ? max((int)(__float_as_uint(m) >> 23) - 127, -60) : 0;
    }
    // Rows divided by 2^e are finite, scale and elements, up to here.
    static __device__ __forceinline__ bool fits(uint32_t bits, int e) { return e == 0 || !(magnitude(bits) >= 2048.0f * __uint_as_float((uint32_t)(127 + e) << 23)); }
};
__device__ __forceinline__ float power_of_two(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }

template <int FMT> struct PpSmem {
    static constexpr uint32_t kRun = kPageTokens * PpFormat<FMT>::kRow;      // one (page, head) run
    static constexpr uint32_t kRawK = 2u * kRun, kRawV = 4u * kRun;
    static constexpr uint32_t kRaw = kRawK + kRawV;
    static constexpr uint32_t kOffK = 0;
    static constexpr uint32_t kOffV = kOffK + kPpStages * kPpStage;
    static constexpr uint32_t kOffQLo = kOffV + kPpStages * kPpStage;
    static constexpr uint32_t kOffRaw = kOffQLo + (PpFormat<FMT>::kRotated ? kPpQLoBytes : 0u);
    static constexpr uint32_t kOffLut = (kOffRaw + kPpRawStages * kRaw + 127u) & ~127u;
    static constexpr uint32_t kOffBars = kOffLut + (PpFormat<FMT>::kRotated ? kPpLutBytes : 0u);
    static constexpr uint32_t kBytes = kOffBars + 288u;
    static_assert(kPpCtaRows * kPpOutStride * 4 <= (int)kOffLut, "epilogue staging must end before the table");
    static_assert(kPpCtaRows * 512 <= (int)kOffQLo, "Q' staging fits the tile stages");
    static_assert(!PpFormat<FMT>::kRotated || (kPpCtaRows / 4 + kPpWarps) * 2048 <= (int)kOffQLo, "so do the rows that change lanes behind it");
    static_assert(kBytes <= 227u * 1024u, "shared memory");
};

// barrier slots (8 bytes each).  Full / PReady: waited for by the MMA warp of CTA 0, arrivals from both CTAs.
// Empty, S, Pv: one arrival per CTA from the MMA warp's commits.  Raw*: within a CTA.
enum { kPpFullK = 0, kPpFullV = kPpFullK + kPpStages, kPpEmptyK = kPpFullV + kPpStages, kPpEmptyV = kPpEmptyK + kPpStages,
       kPpS = kPpEmptyV + kPpStages, kPpPReady = kPpS + 2, kPpPv = kPpPReady + 2, kPpDrain = kPpPv + 2, kPpRawKFull,
       kPpRawKFree = kPpRawKFull + kPpRawStages, kPpRawVFull = kPpRawKFree + kPpRawStages,
       kPpRawVFree = kPpRawVFull + kPpRawStages, kPpBarCount = kPpRawVFree + kPpRawStages };
static_assert(kPpBarCount * 8 <= 224, "barrier slots end before the words behind them");

// ---- CTA-pair wrappers ------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// One lane of a converged warp, chosen by the hardware: the compiler then knows that the branch runs in one thread.
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
    return ok != 0;
}
__device__ __forceinline__ void cluster_sync_all() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc2_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc2_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc2_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc2_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc2_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// One arrival on this barrier slot of both CTAs when every MMA issued so far by this thread has completed.
__device__ __forceinline__ void tc2_commit_both(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t (&r)[16], uint32_t taddr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

struct PrefillPairParams {
    warp34_kv_layer_layout layout;
    warp34_attention_batch batch;
    const void* q_in;
    void* attn_out;
    int io_bf16;
    int num_q_heads;
    int gqa;
    int tok_per_tile;      // 256 / gqa
    int skip_tokens;       // requests of at most this many tokens are left alone
    // The scores are multiplied by score_scale, which is positive.  TQ4: 1, and sm_scale * log2(e) / kPpLutScale is folded into Q' as
    // q_scale.  8-bit: |sm_scale| * log2(e), and q_scale is its sign; 1 and 0 where sm_scale is 0.
    float q_scale, score_scale;
    int32_t* status;       // may be null; bit 0: a wait gave up, bit 1: shared-memory window misaligned
    OutputGate og;
    // A chunk of few tiles after a long context: blockIdx.z takes one of `splits` equal ranges of a tile's key blocks and
    // leaves [split][token][q head][256] un-normalised rows and [split][token][q head]{m, l}; prefill_merge_kernel finishes.
    int splits;
    float* parts;
    float2* parts_ml;
};

// ---- rotation of a tile's rows, four at a time -------------------------------------------------------
// Eight lanes hold a row, 32 columns each, so that five of the eight levels of the 256-point transform are register arithmetic; between two
// such layouts the columns change lanes through shared memory.  (A row over a whole warp takes 40 shuffles; those of a tile's 128 rows kept
// the SM busy for 16 000 cycles before the first product and for as long again behind the last: 31 of the 46 thousand cycles of a
// tile of one block.)
//   chunks: lane j of a row, register 8 i + e: column 8 (j + 8 i) + e         quads: lane l, register 4 j + e: column 8 (j + 8 (l / 2)) + 4 (l % 2) + e
// Where 16-byte quad u of a row is kept while its columns change lanes: without bank conflicts from either side.
__device__ __forceinline__ uint32_t quad_place(uint32_t u) { return u ^ ((u >> 3) & 1u) ^ (((u >> 4) & 3u) << 1); }
// Levels of the transform whose bit of the column is a bit of the register index, for the bits in LEVELS.  Two butterflies at a time (the
// difference as fma(b, -1, a), the same number): half the instructions, which is what these phases are bound by.
__device__ __forceinline__ uint64_t pair_of(float a, float b) { return (uint64_t)__float_as_uint(a) | ((uint64_t)__float_as_uint(b) << 32); }
template <int LEVELS>
__device__ __forceinline__ void rotate_registers(float (&v)[32]) {
    if (LEVELS & 1) {
#pragma unroll
        for (int k = 0; k < 32; k += 2) {
            const float a = v[k], b = v[k + 1];
            v[k] = a + b;
            v[k + 1] = a - b;
        }
    }
    const uint64_t minus_one = pair_of(-1.0f, -1.0f);
    uint64_t x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = pair_of(v[2 * k], v[2 * k + 1]);
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        if (!(LEVELS & (2 * d))) continue;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            if (k & d) continue;
            const uint64_t a = x[k], b = x[k | d];
            asm("add.rn.f32x2 %0, %1, %2;" : "=l"(x[k]) : "l"(a), "l"(b));
            asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(x[k | d]) : "l"(b), "l"(minus_one), "l"(a));
        }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        v[2 * k] = __uint_as_float((uint32_t)x[k]);
        v[2 * k + 1] = __uint_as_float((uint32_t)(x[k] >> 32));
    }
}
__device__ __forceinline__ void quads_store(uint32_t row, int j, const float (&v)[32]) {      // from chunks
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        sts128(row + (quad_place((uint32_t)(2 * (j + 8 * (k >> 1)) + (k & 1))) << 4), __float_as_uint(v[4 * k]), __float_as_uint(v[4 * k + 1]),
               __float_as_uint(v[4 * k + 2]), __float_as_uint(v[4 * k + 3]));
    }
}
__device__ __forceinline__ void lds128f(uint32_t addr, float& a, float& b, float& c, float& d) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "r"(addr));
}
__device__ __forceinline__ uint32_t quad_of(int l, int j) { return (uint32_t)(2 * (j + 8 * (l >> 1)) + (l & 1)); }
// Where 16-byte chunk c of a query row is staged: conflict-free for a thread per row and for the lanes of a rotated group.
template <bool ROT>
__device__ __forceinline__ uint32_t q_chunk_place(uint32_t c, uint32_t row) { return ROT ? (c & ~7u) | ((c ^ row ^ (2u * (c >> 3))) & 7u) : c ^ (row & 31u); }
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
// The sign diagonal's bits of a lane's four chunks, a byte each (from immediates: the constant bank serves one address at a time).
__device__ __forceinline__ uint32_t chunk_signs(int j) {
    constexpr uint32_t kMask[8] = W34_TQ4_SIGN_MASK;
    uint32_t bits = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) bits |= ((((j & 4) ? kMask[2 * i + 1] : kMask[2 * i]) >> (8 * (j & 3))) & 0xffu) << (8 * i);
    asm volatile("" : "+r"(bits));      // (kept as one word: expanded into 32 selects it makes the kernel spill)
    return bits;
}

// Accumulator of one row (columns [8 lane, + 8)) and its mass -> output row.
template <bool ROT>
__device__ __forceinline__ void prefill_finish_row(const PrefillPairParams& p, float (&v)[8], float l, size_t row_base, int lane) {
    const float inv = (l > 0.0f) ? 1.0f / (ROT ? l * (kPpLutScale * 16.0f) : l) : 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] *= inv;
    if (ROT) {
        butterfly8<5>(v, lane);
        sign8(v, lane);
    }
    uint32_t gate[4];
    load_gate8(p.og, row_base, lane, gate);
    apply_output_gate8(v, p.og, gate, lane, p.io_bf16);
    store8(p.attn_out, row_base, lane, p.io_bf16, v);
}

// One query row over its keys in [lo, hi] in fp32 by one warp, as the attention kernel leaves it (columns [8 lane, + 8) of the accumulator,
// mass, maximum): for tiles whose rows differ so much in magnitude that those the exponents were chosen by are not the others' kind.
template <int FMT>
__device__ __forceinline__ void prefill_row_fp32(const PrefillPairParams& p, int req, int q_off, int q_head, int lo, int hi, float (&acc)[8], float& l,
                                                 float& m) {
    constexpr bool ROT = PpFormat<FMT>::kRotated;
    const int lane = threadIdx.x & 31, kv_head = q_head / p.gqa;
    const ReqGeom g = load_req(p.batch, req);
    const int32_t* blocks = p.batch.block_tables + (size_t)req * p.batch.max_blocks_per_req;
    const uint8_t* k_head_base = (const uint8_t*)(uintptr_t)p.layout.k_base + (size_t)kv_head * p.layout.k_head_stride_bytes;
    const uint8_t* v_head_base = (const uint8_t*)(uintptr_t)p.layout.v_base + (size_t)kv_head * p.layout.v_head_stride_bytes;
    lo = max(lo, row_min_kv(p.batch, g, q_off));
    hi = min(hi, row_max_kv(p.batch, g, q_off));
    float q[8];
    load8(p.q_in, ((size_t)(g.q_start + q_off) * p.num_q_heads + q_head) * kHeadDim, lane, p.io_bf16, q);
    if (ROT) {
        sign8(q, lane);
        butterfly8<5>(q, lane);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        q[i] *= ROT ? p.q_scale * (0.0625f * kPpLutScale) : p.q_scale;
        acc[i] = 0.0f;
    }
    auto elements = [&](const uint8_t* row, float (&x)[8]) {
        if (FMT == WARP34_KV_FORMAT_TQ4) {
            const uint8_t* half = row + kTq4BlockBytes * (lane >> 4);
            const uint16_t* codes = reinterpret_cast<const uint16_t*>(half + 2 + 4 * (lane & 15));
            const float d = __half2float(*reinterpret_cast<const __half*>(half));
            const uint32_t w = (uint32_t)codes[0] | ((uint32_t)codes[1] << 16);
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = d * tq4_centroid((int)((w >> (4 * i)) & 15u));
        } else {
            constexpr bool FP8 = FMT == WARP34_KV_FORMAT_FP8_E4M3;
            const uint32_t* codes = reinterpret_cast<const uint32_t*>(row + (FP8 ? 8 * lane : 68 * (lane >> 3) + 4 + 8 * (lane & 7)));
            const float d = *reinterpret_cast<const float*>(row + (FP8 ? kHeadDim + 4 * (lane >> 4) : 68 * (lane >> 3)));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t a, b;
                kv8x4_to_f16x4<FMT>(codes[i], a, b);
                const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&a)), fb = __half22float2(*reinterpret_cast<const __half2*>(&b));
                x[4 * i] = d * fa.x; x[4 * i + 1] = d * fa.y; x[4 * i + 2] = d * fb.x; x[4 * i + 3] = d * fb.y;
            }
        }
    };
    l = 0.0f;
    m = -1e30f;
#pragma unroll 1
    for (int pos = lo; pos <= hi; ++pos) {
        const int32_t page = block_table_page(blocks, pos >> 4, p.batch.max_blocks_per_req, ROT ? kInPrefillExact : kInKv8);
        const size_t row = (size_t)(pos & 15) * PpFormat<FMT>::kRow;
        float x[8], s = 0.0f;
        elements(k_head_base + (size_t)page * p.layout.k_page_stride_bytes + row, x);
#pragma unroll
        for (int i = 0; i < 8; ++i) s += q[i] * x[i];
        s = warp_sum(s) * p.score_scale;
        const float m_new = fmaxf(m, s), alpha = ex2(m - m_new), w = ex2(s - m_new);
        l = l * alpha + w;
        m = m_new;
        elements(v_head_base + (size_t)page * p.layout.v_page_stride_bytes + row, x);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = acc[i] * alpha + w * (ROT ? x[i] * kPpLutScale : x[i]);
    }
}

// Combines the splits of every row that takes part: one warp per (token, q head).
template <bool ROT>
__global__ void __launch_bounds__(128) prefill_merge_kernel(const PrefillPairParams p) {
    grid_dependency_wait();
    grid_launch_dependents();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long rows = (long long)p.batch.total_tokens * p.num_q_heads, row = (long long)blockIdx.x * 4 + wid;
    if (row >= rows) return;
    const int tok = (int)(row / p.num_q_heads);
    // the same exits as the attention kernel: rows it skipped have no parts
    if (p.batch.valid_token_mask != nullptr && p.batch.valid_token_mask[tok] == 0) return;
    const int R = p.batch.num_reqs;
    if (tok < p.batch.query_start_loc[0] || tok >= p.batch.query_start_loc[R]) return;
    const int r = last_not_above(p.batch.query_start_loc, R, tok);
    if (p.skip_tokens != 0 && p.batch.query_start_loc[r + 1] - p.batch.query_start_loc[r] <= p.skip_tokens) return;
    if (p.batch.valid_req_mask != nullptr && p.batch.valid_req_mask[r] == 0) return;
    float2 ml = make_float2(-1e30f, 0.0f);
    if (lane < p.splits) ml = p.parts_ml[(size_t)lane * rows + row];
    const bool part = ROT ? !(ml.y <= 0.0f) : ml.y > 0.0f;      // PpFormat::has_keys
    float m_tot = part ? ml.x : -1e30f;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m_tot = fmaxf(m_tot, __shfl_xor_sync(0xffffffffu, m_tot, d));
    const float w = part ? ex2(ml.x - m_tot) : 0.0f;
    float l_tot = part ? ml.y * w : 0.0f;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) l_tot += __shfl_xor_sync(0xffffffffu, l_tot, d);
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int s = 0; s < p.splits; ++s) {
        const float ws = __shfl_sync(0xffffffffu, w, s);
        const float4* src = reinterpret_cast<const float4*>(p.parts + ((size_t)s * rows + row) * kHeadDim + 8 * lane);
        const float4 a = src[0], b = src[1];
        v[0] += ws * a.x; v[1] += ws * a.y; v[2] += ws * a.z; v[3] += ws * a.w;
        v[4] += ws * b.x; v[5] += ws * b.y; v[6] += ws * b.z; v[7] += ws * b.w;
    }
    prefill_finish_row<ROT>(p, v, l_tot, (size_t)row * kHeadDim, lane);
}

template <int FMT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPpThreads, 1) attention_prefill_pair_kernel(const PrefillPairParams p) {
    using S = PpSmem<FMT>;
    constexpr bool ROT = PpFormat<FMT>::kRotated;
    constexpr uint32_t ROW = PpFormat<FMT>::kRow;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t rank = cluster_rank();
    const uint32_t base = smem_u32(smem_raw);
    uint8_t* gen = smem_raw;

    const uint32_t k_t = base + S::kOffK, v_t = base + S::kOffV, qlo_t = base + S::kOffQLo;
    const uint32_t raw = base + S::kOffRaw, lut = base + S::kOffLut, bars = base + S::kOffBars;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + S::kOffBars + 240);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(gen + S::kOffBars + 244);
    uint32_t* row_max = reinterpret_cast<uint32_t*>(gen + S::kOffBars + 224);                      // largest scale of the tile's K, V rows
    volatile int* exponents = reinterpret_cast<volatile int*>(gen + S::kOffBars + 232);            // of K, of V
    // request, first block, first token, rows, first token of the request: for the epilogue, which reads them again so that they take no
    // registers from the consumers
    volatile int* place = reinterpret_cast<volatile int*>(gen + S::kOffBars + 256);
    auto bar = [&](int which) { return bars + 8u * (uint32_t)which; };
    // Waits and abort checks are warp-uniform: no lane leaves a loop alone.
    auto wait_all = [&](uint32_t b, uint32_t parity) {
        const bool ok = mbar_wait(b, parity);
        return __all_sync(0xffffffffu, ok) != 0;
    };
    auto aborted_any = [&]() { return __any_sync(0xffffffffu, *abort_flag != 0u) != 0; };

    if ((base & 1023u) != 0u) {      // the swizzled tiles need a 1024-byte-aligned window (the kernel has no static shared memory)
        grid_dependency_wait();
        if (tid == 0 && p.status != nullptr) *p.status = 2;
        return;
    }
    // ---- one-time setup -------------------------------------------------------------------------
    if (ROT) {
        for (int i = tid; i < 256 * 16; i += kPpThreads) {
            const int byte = i >> 4, copy = i & 15;
            const float c0 = kPpLutScale * tq4_centroid(byte & 15), c1 = kPpLutScale * tq4_centroid(byte >> 4);
            const uint32_t hi = pack_half2(c0, c1);
            const float2 hf = __half22float2(*reinterpret_cast<const __half2*>(&hi));
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(lut + (uint32_t)(byte * 128 + copy * 8)), "r"(hi),
                         "r"(pack_half2(c0 - hf.x, c1 - hf.y)) : "memory");
        }
    }
    if (tid == 0) {
        for (int s = 0; s < kPpStages; ++s) {
            mbar_init(bar(kPpFullK + s), 8u);      // four producer warps of each CTA
            mbar_init(bar(kPpFullV + s), 8u);
            mbar_init(bar(kPpEmptyK + s), 1u);
            mbar_init(bar(kPpEmptyV + s), 1u);
        }
        mbar_init(bar(kPpS), 1u);
        mbar_init(bar(kPpS + 1), 1u);
        mbar_init(bar(kPpPv), 1u);
        mbar_init(bar(kPpPv + 1), 1u);
        mbar_init(bar(kPpPReady), 8u);             // four consumer warps of each CTA
        mbar_init(bar(kPpPReady + 1), 8u);
        mbar_init(bar(kPpDrain), 1u);
        for (int s = 0; s < kPpRawStages; ++s) {
            mbar_init(bar(kPpRawKFull + s), 1u);
            mbar_init(bar(kPpRawKFree + s), 4u);
            mbar_init(bar(kPpRawVFull + s), 1u);
            mbar_init(bar(kPpRawVFree + s), 4u);
        }
        *abort_flag = 0u;
        row_max[0] = row_max[1] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    grid_dependency_wait();          // nothing above touches global memory
    grid_launch_dependents();
    if (tid == 0 && (blockIdx.x | blockIdx.y | blockIdx.z) == 0 && p.status != nullptr) *p.status = 0;

    // ---- which (request, token tile) is this pair?  Both CTAs agree on every exit here. -------------
    const int tpt = p.tok_per_tile;
    const int kv_head = blockIdx.y;
    int req = -1, tile_in_req = 0;
    {
        int t = (int)(blockIdx.x >> 1);
        if (p.batch.num_reqs <= 8) {
            for (int r = 0; r < p.batch.num_reqs; ++r) {
                const int ql = p.batch.query_start_loc[r + 1] - p.batch.query_start_loc[r];
                const int nt = min((ql + tpt - 1) / tpt, ql > p.skip_tokens ? 0x7fffffff : 0);
                if (t < nt) { req = r; tile_in_req = nt - 1 - t; break; }    // the tiles with the most keys first
                t -= nt;
            }
        } else {
            // a lane per request: one round trip to memory, where the loop above makes one for every few requests ahead of the pair's own
            // (64 requests of 16 tokens 112.0 -> 92.4 us; with two requests the shuffles cost 0.3 us, with eight or fewer the loop stays)
            for (int base_r = 0; base_r < p.batch.num_reqs && req < 0; base_r += 32) {
                const int r = base_r + lane;
                int nt = 0;
                if (r < p.batch.num_reqs) {
                    const int ql = p.batch.query_start_loc[r + 1] - p.batch.query_start_loc[r];
                    nt = max(min((ql + tpt - 1) / tpt, ql > p.skip_tokens ? 0x7fffffff : 0), 0);
                }
                int upto = nt;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int x = __shfl_up_sync(0xffffffffu, upto, d);
                    if (lane >= d) upto += x;
                }
                const uint32_t hit = __ballot_sync(0xffffffffu, t < upto);
                if (hit != 0u) {
                    const int src = __ffs((int)hit) - 1;
                    req = base_r + src;
                    tile_in_req = __shfl_sync(0xffffffffu, upto, src) - 1 - t;
                } else {
                    t -= __shfl_sync(0xffffffffu, upto, 31);
                }
            }
        }
    }
    if (req < 0) return;
    const ReqGeom g = load_req(p.batch, req);
    if (!g.valid) return;
    const int tok0 = tile_in_req * tpt;
    const int ntok = min(tpt, g.q_len - tok0);
    const int rows_used = ntok * p.gqa;
    const int row0 = (int)rank * kPpCtaRows;      // first row of this CTA in the tile
    // keys any row of the pair can see (both limits grow with the token)
    const int kv_lo = row_min_kv(p.batch, g, tok0);
    const int kv_hi = row_max_kv(p.batch, g, tok0 + ntok - 1);
    const bool any_keys = kv_hi >= kv_lo;
    const int pg_lo = any_keys ? (kv_lo >> 4) : 0, pg_hi = any_keys ? (kv_hi >> 4) : -1;
    const int all_lo = any_keys ? (kv_lo >> 6) : 0, all = any_keys ? ((kv_hi >> 6) - all_lo + 1) : 0;
    const int kb_lo = all_lo + (int)((long long)all * blockIdx.z / p.splits);     // this split's key blocks
    const int nblocks = all_lo + (int)((long long)all * (blockIdx.z + 1) / p.splits) - kb_lo;

    __syncwarp();
    if (wid == 0) {
        tc2_alloc(base + S::kOffBars + 240, 512);
        tc2_relinquish();
    }
    __syncthreads();                 // this CTA's barriers exist

    // ---- raw (page, head) runs of a block; the first blocks are on their way before the query is prepared ----------
    const int32_t* blocks = p.batch.block_tables + (size_t)req * p.batch.max_blocks_per_req;
    const uint8_t* k_head_base = (const uint8_t*)(uintptr_t)p.layout.k_base + (size_t)kv_head * p.layout.k_head_stride_bytes;
    const uint8_t* v_head_base = (const uint8_t*)(uintptr_t)p.layout.v_base + (size_t)kv_head * p.layout.v_head_stride_bytes;
    auto page_id = [&](int j) -> int32_t {      // lane pp < 4: page pp of block j, -1 outside the visible range
        const int pg = 4 * (kb_lo + j) + (lane & 3);
        return (j < nblocks && pg >= pg_lo && pg <= pg_hi)
                   ? block_table_page(blocks, pg, p.batch.max_blocks_per_req, ROT ? kInPrefillExact : kInKv8) : -1;
    };
    auto copy_k = [&](int j, int32_t id) {      // this CTA's two pages
        const int s = j % kPpRawStages;
        const uint32_t mask = (__ballot_sync(0xffffffffu, id >= 0) >> (2 * rank)) & 3u;
        if (lane == 0) mbar_expect_tx(bar(kPpRawKFull + s), (uint32_t)__popc(mask) * S::kRun);
        __syncwarp();
        if (lane < 4 && (lane >> 1) == (int)rank && id >= 0) {
            bulk_g2s(raw + (uint32_t)s * S::kRaw + (uint32_t)(lane & 1) * S::kRun, k_head_base + (size_t)id * p.layout.k_page_stride_bytes,
                     S::kRun, bar(kPpRawKFull + s));
        }
    };
    auto copy_v = [&](int j, int32_t id) {      // all four
        const int s = j % kPpRawStages;
        const uint32_t mask = __ballot_sync(0xffffffffu, id >= 0) & 15u;
        if (lane == 0) mbar_expect_tx(bar(kPpRawVFull + s), (uint32_t)__popc(mask) * S::kRun);
        __syncwarp();
        if (lane < 4 && id >= 0) {
            bulk_g2s(raw + (uint32_t)s * S::kRaw + S::kRawK + (uint32_t)lane * S::kRun, v_head_base + (size_t)id * p.layout.v_page_stride_bytes,
                     S::kRun, bar(kPpRawVFull + s));
        }
    };
    int32_t next_id = -1;
    if (wid == 13) {
        for (int j = 0; j < kPpRawStages && j < nblocks; ++j) {
            const int32_t id = page_id(j);
            copy_k(j, id);
            copy_v(j, id);
        }
        next_id = page_id(kPpRawStages);
    }
    // The sample that exponents are chosen by: the first scales of the first block's rows, the same in both CTAs.  Requested here,
    // looked at behind the query's rows.
    uint32_t sample_k[2] = {0u, 0u}, sample_v[2] = {0u, 0u};
    if (wid == 12) {
        const int32_t id = page_id(0);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int pos = (kb_lo << 6) + lane + 32 * x;
            const int32_t page = __shfl_sync(0xffffffffu, id, 2 * x + (lane >> 4));
            if (page >= 0 && pos >= kv_lo && pos <= kv_hi) {
                const size_t row = (size_t)(lane & 15) * ROW;
                sample_k[x] = PpScales<FMT>::first(k_head_base + (size_t)page * p.layout.k_page_stride_bytes + row);
                sample_v[x] = PpScales<FMT>::first(v_head_base + (size_t)page * p.layout.v_page_stride_bytes + row);
            }
        }
    }

    // ---- Q rows of this CTA: four rows a warp, eight lanes each.  TQ4: rotated, scaled, split into value (staging) and
    //      residual (swizzled A tile); 8-bit: the fp16 row as it is ------------------------------------
    const uint32_t q_stage = k_t;     // 128 rows x 512 B over the tile stages
    {
        const int r4 = lane >> 3, j = lane & 7;
        const uint32_t signs = ROT ? chunk_signs(j) : 0u;
        uint32_t raw_q[4][4];
        auto load_group = [&](int grp) {
            const int trow = row0 + 4 * grp + r4;
            const int q_off = tok0 + trow / p.gqa;
            const int q_head = kv_head * p.gqa + trow % p.gqa;
            const bool ok = 4 * grp < kPpCtaRows && trow < rows_used &&
                            (p.batch.valid_token_mask == nullptr || p.batch.valid_token_mask[g.q_start + q_off] != 0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                raw_q[i][0] = raw_q[i][1] = raw_q[i][2] = raw_q[i][3] = 0u;
                if (ok) load8_raw(p.q_in, ((size_t)(g.q_start + q_off) * p.num_q_heads + q_head) * kHeadDim, j + 8 * i, raw_q[i]);
            }
        };
#pragma unroll 1
        for (int grp = wid; 4 * grp < kPpCtaRows; grp += kPpWarps) {
            const int row = 4 * grp + r4;
            load_group(grp);
            if (!ROT) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float x[8];
                    widen8(raw_q[i], p.io_bf16, x);
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] *= p.q_scale;
                    sts128(q_stage + (uint32_t)row * 512u + (q_chunk_place<ROT>((uint32_t)(j + 8 * i), (uint32_t)row) << 4), pack_half2(x[0], x[1]),
                           pack_half2(x[2], x[3]), pack_half2(x[4], x[5]), pack_half2(x[6], x[7]));
                }
                continue;
            }
            float v[32];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float x[8];
                widen8(raw_q[i], p.io_bf16, x);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[8 * i + e] = __uint_as_float(__float_as_uint(x[e]) ^ (((signs >> (8 * i + e)) & 1u) << 31));
            }
            rotate_registers<31>(v);
            // two of the four rows change lanes where the group's values will lie, two in this warp's part of the space behind the staging rows
            const uint32_t turn = q_stage + (uint32_t)(r4 & 1) * 1024u + 2048u * (uint32_t)(r4 < 2 ? grp : kPpCtaRows / 4 + wid);
            quads_store(turn, j, v);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 8; ++k) lds128f(turn + (quad_place(quad_of(j, k)) << 4), v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            __syncwarp();
            rotate_registers<4 + 8 + 16>(v);
#pragma unroll
            for (int k = 0; k < 8; ++k) {      // chunk k + 8 (j / 2), its half j % 2
                uint32_t hi[2], lo[2];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float y0 = v[4 * k + 2 * x] * (p.q_scale * 0.0625f), y1 = v[4 * k + 2 * x + 1] * (p.q_scale * 0.0625f);
                    const __half2 h = __floats2half2_rn(y0, y1);
                    const float2 hf = __half22float2(h);
                    hi[x] = *reinterpret_cast<const uint32_t*>(&h);
                    lo[x] = pack_half2(y0 - hf.x, y1 - hf.y);
                }
                const uint32_t half = 8u * (uint32_t)(j & 1);
                sts64(q_stage + (uint32_t)row * 512u + (q_chunk_place<ROT>((uint32_t)(k + 8 * (j >> 1)), (uint32_t)row) << 4) + half, hi[0], hi[1]);
                sts64(qlo_t + (uint32_t)(j >> 1) * (kPpCtaRows * 128u) + (uint32_t)row * 128u + (uint32_t)((k ^ (row & 7)) << 4) + half, lo[0], lo[1]);
            }
        }
    }
    if (wid == 12) {
        const int ek = PpScales<FMT>::exponent(__reduce_max_sync(0xffffffffu, max(sample_k[0], sample_k[1])));
        const int ev = PpScales<FMT>::exponent(__reduce_max_sync(0xffffffffu, max(sample_v[0], sample_v[1])));
        if (lane == 0) { exponents[0] = ek; exponents[1] = ev; place[0] = req; place[1] = kb_lo; place[2] = tok0; place[3] = rows_used; place[4] = g.q_start; }
    }
    if (ROT) fence_proxy_async();     // the residual tile is read by the tensor core
    tc_fence_before();
    __syncthreads();                  // staging is written
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (wid < 4) {
        const uint32_t t_q = tmem + ((uint32_t)(32 * wid) << 16) + kPpColQ;
#pragma unroll 1
        for (int c4 = 0; c4 < 4; ++c4) {
            uint32_t r[32];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint32_t chunk = (uint32_t)(8 * c4 + c);
                const uint32_t addr = q_stage + (uint32_t)tid * 512u + (q_chunk_place<ROT>(chunk, (uint32_t)tid) << 4);
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(r[4 * c]), "=r"(r[4 * c + 1]), "=r"(r[4 * c + 2]), "=r"(r[4 * c + 3]) : "r"(addr));
            }
            tc_st32(t_q + 32u * c4, r);
        }
        tc_wait_st();
    }
    tc_fence_before();
    cluster_sync_all();               // both CTAs: barriers, TMEM and Q' are in place, the staging area becomes the tile stages
    tc_fence_after();

    float l_run = 0.0f, m_ref = -1e30f;     // consumers: of this thread's row
    const int ek = exponents[0], ev = exponents[1];

    if (wid == 12) {
        // ======================= MMA issue: lane 0 of CTA 0 feeds both tensor cores ====================
        // Order in the pipe: QK(0), QK(1), PV(0), QK(2), PV(1), ...  QK(j) overwrites the buffer of P(j - 2),
        // which PV(j - 2), issued before it, has read.
        if (rank == 0 && elect_one()) {
            constexpr uint32_t kIdescQk = tc_idesc(kPpRows, kPpKeys, 0);
            constexpr uint32_t kIdescPv = tc_idesc(kPpRows, kHeadDim, 1);
            const uint64_t desc_k = tc_smem_desc(k_t, 16u, 1024u);
            const uint64_t desc_v = tc_smem_desc(v_t, 4096u, 1024u);
            const uint64_t desc_q = tc_smem_desc(qlo_t, 16u, 1024u);
            uint32_t kst = 0, kph = 0, vst = 0, vph = 0;
            bool ok = true;
#pragma unroll 1
            for (int j = 0; j <= nblocks && ok && *abort_flag == 0u; ++j) {
                if (j < nblocks) {
                    const uint32_t d = tmem + kPpColS + 64u * (uint32_t)(j & 1);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        ok = ok && mbar_wait(bar(kPpFullK + (int)kst), kph);
                        if (!ok) break;
                        tc_fence_after();
                        const uint64_t b0 = desc_k + (uint64_t)(kst * (kPpStage / 16));
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks) {
                            const uint64_t b = b0 + (uint64_t)((ks >> 2) * (4096 / 16) + 2 * (ks & 3));
                            const uint32_t a = tmem + kPpColQ + 64u * (uint32_t)h + 8u * (uint32_t)ks;
                            tc2_mma_f16_ts(d, a, b, kIdescQk, (h || ks) ? 1u : 0u);
                            tc2_mma_f16_ts(d, a, b + kPpPart / 16, kIdescQk, 1u);
                            if (ROT) {
                                tc2_mma_f16(d, desc_q + (uint64_t)((2 * h + (ks >> 2)) * (kPpCtaRows * 128 / 16) + 2 * (ks & 3)), b,
                                            kIdescQk, 1u);
                            }
                        }
                        tc2_commit_both(bar(kPpEmptyK + (int)kst));
                        if (h == 1) tc2_commit_both(bar(kPpS + (j & 1)));
                        if (++kst == kPpStages) { kst = 0; kph ^= 1u; }
                    }
                }
                if (j > 0 && ok) {
                    const int i = j - 1;
                    ok = mbar_wait(bar(kPpPReady + (i & 1)), (uint32_t)((i >> 1) & 1));
                    const uint32_t a0 = tmem + kPpColS + 64u * (uint32_t)(i & 1);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        ok = ok && mbar_wait(bar(kPpFullV + (int)vst), vph);
                        if (!ok) break;
                        tc_fence_after();
                        const uint64_t b0 = desc_v + (uint64_t)(vst * (kPpStage / 16));
#pragma unroll
                        for (int ks = 0; ks < 2; ++ks) {
                            const uint64_t b = b0 + (uint64_t)((2048 / 16) * ks);
                            const uint32_t a = a0 + 32u * (uint32_t)h + 8u * (uint32_t)ks;
                            tc2_mma_f16_ts(tmem + kPpColO, a, b, kIdescPv, (i > 0 || h > 0 || ks > 0) ? 1u : 0u);
                            tc2_mma_f16_ts(tmem + kPpColO, a + 16u, b, kIdescPv, 1u);
                            tc2_mma_f16_ts(tmem + kPpColO, a, b + kPpPart / 16, kIdescPv, 1u);
                        }
                        tc2_commit_both(bar(kPpEmptyV + (int)vst));
                        if (h == 1) tc2_commit_both(bar(kPpPv + (i & 1)));
                        if (++vst == kPpStages) { vst = 0; vph ^= 1u; }
                    }
                }
            }
            if (!ok) *abort_flag = 1u;
            // nothing may be in flight when the CTAs leave (after an abort as well)
            tc2_commit_both(bar(kPpDrain));
        }
        __syncwarp();
        if (!wait_all(bar(kPpDrain), 0u)) *abort_flag = 1u;
    } else if (wid == 13) {
        // ======================= copy issue: raw (page, head) runs of a block ===========================
        int issued = 2 * min(nblocks, kPpRawStages);
#pragma unroll 1
        for (int j = kPpRawStages; j < nblocks; ++j) {
            if (aborted_any()) break;
            const int s = j % kPpRawStages;
            const int32_t id = next_id;
            next_id = page_id(j + 1);
            if (!wait_all(bar(kPpRawKFree + s), (uint32_t)((j / kPpRawStages - 1) & 1))) { *abort_flag = 1u; break; }
            copy_k(j, id);
            issued = 2 * j + 1;
            if (!wait_all(bar(kPpRawVFree + s), (uint32_t)((j / kPpRawStages - 1) & 1))) { *abort_flag = 1u; break; }
            copy_v(j, id);
            issued = 2 * j + 2;
        }
        // copies in flight must land before the CTA leaves
        const int kn = (issued + 1) / 2, vn = issued / 2;
        for (int j = max(0, kn - kPpRawStages); j < kn; ++j) (void)wait_all(bar(kPpRawKFull + j % kPpRawStages), (uint32_t)((j / kPpRawStages) & 1));
        for (int j = max(0, vn - kPpRawStages); j < vn; ++j) (void)wait_all(bar(kPpRawVFull + j % kPpRawStages), (uint32_t)((j / kPpRawStages) & 1));
    } else if (wid >= 4) {
        // ======================= producers: lane = key, this warp's 32 channels of the stage's 128 ========
        const bool is_v = wid >= 8;
        const int quarter = wid & 3;
        const int raw_full = is_v ? kPpRawVFull : kPpRawKFull, raw_free = is_v ? kPpRawVFree : kPpRawKFree;
        const int full = is_v ? kPpFullV : kPpFullK, empty = is_v ? kPpEmptyV : kPpEmptyK;
        const uint32_t tiles = is_v ? v_t : k_t;
        // chunk c (8 channels) of key `lane`: [block of 64 channels][key][16-byte chunk XOR (key & 7)]
        const uint32_t dst0 = (uint32_t)(quarter >> 1) * 4096u + (uint32_t)lane * 128u;
        const uint32_t lut_lane = lut + 8u * (uint32_t)(lane & 15);
        const uint32_t leader_full = map_to_rank(bar(full), 0u);
        const int exponent = is_v ? ev : ek;
        const float down = power_of_two(-exponent);
        uint32_t most = 0u;           // largest scale seen, where that matters
        uint32_t st = 0, ph = 1;      // parity 1: the first pass over the ring does not wait
#pragma unroll 1
        for (int j = 0; j < nblocks; ++j) {
            if (aborted_any()) break;
            const int rs = j % kPpRawStages;
            if (!wait_all(bar(raw_full + rs), (uint32_t)((j / kPpRawStages) & 1))) { *abort_flag = 1u; break; }
            const uint32_t run = raw + (uint32_t)rs * S::kRaw + (is_v ? S::kRawK : 0u);
            bool ok = true;
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                // K: channels [128 h, + 128) of this CTA's 32 keys.  V: channels [128 rank, + 128) of keys 32 h + lane.
                const int key = is_v ? 32 * h + lane : lane;
                const int half = is_v ? (int)rank : h;
                const int pos = ((kb_lo + j) << 6) + (is_v ? key : 32 * (int)rank + lane);
                const bool key_ok = pos >= kv_lo && pos <= kv_hi;     // others may hold never-written bytes
                const uint32_t rowp = run + (uint32_t)key * ROW;
                uint32_t w[FMT == WARP34_KV_FORMAT_TQ4 ? 4 : 8];
                float d = 0.0f;
                uint32_t dbits = 0;
                if (FMT == WARP34_KV_FORMAT_TQ4) {
                    if (half == 0) {       // codes of half 0 start at byte 2
                        uint32_t x[5];
#pragma unroll
                        for (int i = 0; i < 5; ++i) x[i] = lds32(rowp + 16u * quarter + 4u * i);
                        dbits = lds_u16(rowp);
#pragma unroll
                        for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(x[i], x[i + 1], 16);
                    } else {
                        dbits = lds_u16(rowp + 66u);
#pragma unroll
                        for (int i = 0; i < 4; ++i) w[i] = lds32(rowp + 68u + 16u * quarter + 4u * i);
                    }
                    if (!key_ok) dbits = 0u;
                    if (exponent != 0) {
                        most = max(most, dbits & 0x7fffu);
                        dbits = __half_as_ushort(__float2half_rn(__half2float(__ushort_as_half((unsigned short)dbits)) * down));
                    }
                } else if (FMT == WARP34_KV_FORMAT_FP8_E4M3) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i] = lds32(rowp + 128u * half + 32u * quarter + 4u * i);
                    d = __uint_as_float(lds32(rowp + kHeadDim + 4u * half));
                } else {
                    const uint32_t blk = rowp + 68u * (uint32_t)(2 * half + (quarter >> 1));
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i] = lds32(blk + 4u + 32u * (quarter & 1) + 4u * i);
                    d = __uint_as_float(lds32(blk));
                }
                if (FMT != WARP34_KV_FORMAT_TQ4 && !key_ok) {
                    d = 0.0f;
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i] = 0u;      // e4m3 codes of unwritten rows can be NaN patterns
                }
                if (FMT != WARP34_KV_FORMAT_TQ4 && exponent != 0) {
                    most = max(most, __float_as_uint(d) & 0x7fffffffu);
                    d *= down;
                }
                __syncwarp();
                if (h == 1 && lane == 0) mbar_arrive(bar(raw_free + rs));     // the runs are in registers
                ok = wait_all(bar(empty + (int)st), ph);
                if (!ok) break;
                const uint32_t dst = tiles + st * kPpStage + dst0;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t hi[4], lo[4];
                    if (FMT == WARP34_KV_FORMAT_TQ4) {
                        const __half2 d2 = __half2half2(__ushort_as_half((unsigned short)dbits));
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t off = (k == 0 ? (w[c] << 7) : (w[c] >> (8 * k - 7))) & 0x7f80u;
                            const uint2 e = lds64_lut(lut_lane + off);
                            const __half2 ch = *reinterpret_cast<const __half2*>(&e.x), cl = *reinterpret_cast<const __half2*>(&e.y);
                            const __half2 vh = __hmul2(d2, ch);
                            const __half2 vl = __hfma2(d2, cl, __hfma2(d2, ch, __hneg2(vh)));     // the inner fma is exact
                            hi[k] = *reinterpret_cast<const uint32_t*>(&vh);
                            lo[k] = *reinterpret_cast<const uint32_t*>(&vl);
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            uint32_t c01, c23;
                            kv8x4_to_f16x4<FMT>(w[2 * c + k], c01, c23);
#pragma unroll
                            for (int x = 0; x < 2; ++x) {
                                const uint32_t cc = x ? c23 : c01;
                                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&cc));
                                const __half2 vh = __floats2half2_rn(d * f.x, d * f.y);
                                const float2 hf = __half22float2(vh);
                                const __half2 vl = __floats2half2_rn(__fmaf_rn(d, f.x, -hf.x), __fmaf_rn(d, f.y, -hf.y));
                                hi[2 * k + x] = *reinterpret_cast<const uint32_t*>(&vh);
                                lo[2 * k + x] = *reinterpret_cast<const uint32_t*>(&vl);
                            }
                        }
                    }
                    const uint32_t a = dst + (uint32_t)(((4 * (quarter & 1) + c) ^ (lane & 7)) << 4);
                    sts128(a, hi[0], hi[1], hi[2], hi[3]);
                    sts128(a + kPpPart, lo[0], lo[1], lo[2], lo[3]);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(leader_full + 8u * st);
                if (++st == kPpStages) { st = 0; ph ^= 1u; }
            }
            if (!ok) { *abort_flag = 1u; break; }
        }
        if (exponent != 0) {
            most = __reduce_max_sync(0xffffffffu, most);
            if (lane == 0) {
#pragma unroll
                for (uint32_t r = 0; r < 2; ++r) {
                    asm volatile("red.relaxed.cluster.shared::cluster.max.u32 [%0], %1;" ::"r"(map_to_rank(smem_u32(row_max + (is_v ? 1 : 0)), r)), "r"(most) : "memory");
                }
            }
        }
    } else {
        // ======================= consumers: softmax, P, rescale =========================================
        const int trow = row0 + tid;
        const int q_off = tok0 + trow / p.gqa;
        const bool row_ok = trow < rows_used &&
                            (p.batch.valid_token_mask == nullptr || p.batch.valid_token_mask[g.q_start + q_off] != 0);
        const int rmax = row_ok ? row_max_kv(p.batch, g, q_off) : -1;
        const int rmin = row_ok ? row_min_kv(p.batch, g, q_off) : 0x7fffffff;
        const uint32_t lane_base = (uint32_t)(32 * wid) << 16;
        const uint32_t t_o = tmem + lane_base + kPpColO, t_s = tmem + lane_base + kPpColS;
        const uint32_t leader_pready = map_to_rank(bar(kPpPReady), 0u);
        const float factor = ROT ? power_of_two(ek) : 1.0f;
#pragma unroll 1
        for (int j = 0; j < nblocks; ++j) {
            if (aborted_any()) break;
            if (!wait_all(bar(kPpS + (j & 1)), (uint32_t)((j >> 1) & 1))) { *abort_flag = 1u; break; }
            // PV(j - 2) precedes QK(j) in the pipe.  Every phase is waited for: the next one of the same barrier, PV(j), needs this
            // block's weights, so that no delay of this warp lets two go by.  (One barrier for all blocks would have: PV(j - 1) needs
            // nothing more from here, and once it had completed the parity meant PV(j).)
            if (j >= 2 && !wait_all(bar(kPpPv + (j & 1)), (uint32_t)(((j - 2) >> 1) & 1))) { *abort_flag = 1u; break; }
            tc_fence_after();
            const uint32_t t_sj = t_s + 64u * (uint32_t)(j & 1);
            const int kbase = (kb_lo + j) << 6;
            const bool all_seen = kbase >= rmin && kbase + 63 <= rmax;
            // Scores of keys [32 c, + 32) of the block, masked.  TQ4: `factor`, the exponent's power of two, is still to be applied.  8-bit:
            // p.score_scale is, a constant operand (in one register with the power of two it made these builds spill, and a stack
            // frame costs this kernel several us a launch).
            auto scores = [&](int c, float (&sv)[32]) {
                uint32_t r[32];
                tc_ld32(r, t_sj + 32u * (uint32_t)c);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) sv[i] = __uint_as_float(r[i]);
                if (!ROT && ek != 0) {
                    const float up = power_of_two(exponents[0]);
#pragma unroll
                    for (int i = 0; i < 32; ++i) sv[i] *= up;
                }
                if (!all_seen) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int pos = kbase + 32 * c + i;
                        if (!(pos >= rmin && pos <= rmax)) sv[i] = -INFINITY;
                    }
                }
            };
            // TQ4 reads them twice (maximum, then weights): holding all 64 spills there (92 bytes a thread, five ragged
            // prompts 270 us instead of 245), while the 8-bit builds have room and the second read costs them 10 %.
            float sv[2][32];
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};     // four independent chains
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                scores(c, sv[ROT ? 0 : c]);
#pragma unroll
                for (int i = 0; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], sv[ROT ? 0 : c][i]);
            }
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * (ROT ? factor : p.score_scale);
            // the reference maximum moves only when the true maximum ran ahead by more than the threshold
            const bool need = mx > m_ref + kPpRescaleThreshold;
            float alpha = 1.0f;
            if (need) {
                alpha = ex2(m_ref - mx);      // 0 when nothing was visible before
                m_ref = mx;
            }
            if (j > 0 && __any_sync(0xffffffffu, need)) {
                // O is at rest once the previous output product has completed (the next one waits for this block's P)
                if (!wait_all(bar(kPpPv + ((j - 1) & 1)), (uint32_t)(((j - 1) >> 1) & 1))) { *abort_flag = 1u; break; }
                tc_fence_after();
#pragma unroll 1
                for (int c = 0; c < 16; ++c) {
                    uint32_t o[16];
                    tc_ld16(o, t_o + 16u * c);
                    tc_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                    tc_st16(t_o + 16u * c, o);
                }
            }
            float ls4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const float m_use = ((m_ref < -1e29f) ? 0.0f : m_ref) - kPpShift;     // nothing visible yet: every P is 0
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t hi[16], lo[16];
                if (ROT) scores(c, sv[0]);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    // masked scores are -infinity: ex2 gives exactly 0 against any finite reference
                    const float sa = sv[ROT ? 0 : c][2 * i], sb = sv[ROT ? 0 : c][2 * i + 1];
                    const float pa = ex2(__fmaf_rn(sa, ROT ? factor : p.score_scale, -m_use)), pb = ex2(__fmaf_rn(sb, ROT ? factor : p.score_scale, -m_use));
                    ls4[i & 3] += pa + pb;
                    const __half2 h = __floats2half2_rn(pa, pb);
                    const float2 hf = __half22float2(h);
                    hi[i] = *reinterpret_cast<const uint32_t*>(&h);
                    lo[i] = pack_half2(pa - hf.x, pb - hf.y);
                }
                // P takes the place of the scores it came from: value in columns 32 c .. + 15, residual in the next 16
                tc_st16(t_sj + 32u * c, hi);
                tc_st16(t_sj + 32u * c + 16u, lo);
            }
            tc_wait_st();
            l_run = l_run * alpha + ((ls4[0] + ls4[1]) + (ls4[2] + ls4[3]));
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader_pready + 8u * (uint32_t)(j & 1));
        }
        // the last output product
        if (nblocks > 0 && !aborted_any()) {
            if (nblocks > 1 && !wait_all(bar(kPpPv + (nblocks & 1)), (uint32_t)(((nblocks - 2) >> 1) & 1))) *abort_flag = 1u;
            if (!wait_all(bar(kPpPv + ((nblocks - 1) & 1)), (uint32_t)(((nblocks - 1) >> 1) & 1))) *abort_flag = 1u;
        }
        tc_fence_after();
    }

    // ---- epilogue: O / l -> staging -> inverse rotation -> global ---------------------------------
    // (staging aliases the tiles: every MMA of the pair that read them has completed, see kPpDrain)
    __syncthreads();
    const int k_exp = exponents[0], v_exp = exponents[1];      // (read again: in registers throughout, they would make the kernel spill)
    bool fits = true;
    if ((k_exp | v_exp) != 0) {      // does every row of the tile fit the sample's exponents?  (K rows are spread over both CTAs.)
        cluster_sync_all();
        fits = PpScales<FMT>::fits(row_max[0], k_exp) && PpScales<FMT>::fits(row_max[1], v_exp);
    }
    const bool aborted = *abort_flag != 0u;
    float* stage = reinterpret_cast<float*>(gen);
    if (wid < 4 && !aborted) {
        float* mine = stage + tid * kPpOutStride;
        if (nblocks > 0) {
            const uint32_t t_o = tmem + ((uint32_t)(32 * wid) << 16) + kPpColO;
#pragma unroll 1
            for (int c = 0; c < 8; ++c) {
                uint32_t o[32];
                tc_ld32(o, t_o + 32u * c);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    *reinterpret_cast<uint4*>(mine + 4u * (ROT ? quad_place((uint32_t)(8 * c + i)) : (uint32_t)(8 * c + i))) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                }
            }
        }
        mine[256] = l_run;
        mine[257] = m_ref;
    }
    tc_fence_before();
    __syncthreads();
    if (!aborted) {
        const int first_token = place[2], rows = place[3], q_start = place[4];
        const bool by_rows = !fits || p.splits > 1;      // (tiles that are computed in fp32, and parts of a tile's keys, which are not rotated here)
        if (by_rows) {
            for (int row = wid; row < kPpCtaRows; row += kPpWarps) {
                const int trow = (int)cluster_rank() * kPpCtaRows + row;
                if (trow >= rows) break;
                const int q_off = first_token + trow / p.gqa;
                const int q_head = kv_head * p.gqa + trow % p.gqa;
                if (p.batch.valid_token_mask != nullptr && p.batch.valid_token_mask[q_start + q_off] == 0) continue;
                const float* src = stage + row * kPpOutStride;
                float l = src[256], m = src[257];
                float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                if (!fits) {
                    prefill_row_fp32<FMT>(p, place[0], q_off, q_head, place[1] << 6, ((place[1] + nblocks) << 6) - 1, v, l, m);
                } else if (PpFormat<FMT>::has_keys(l)) {
                    const uint32_t qa = ROT ? quad_place(2u * lane) : 2u * lane;      // (the next quad is its neighbour)
                    const float4 a = *reinterpret_cast<const float4*>(src + 4u * qa), b = *reinterpret_cast<const float4*>(src + 4u * (qa ^ 1u));
                    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
                    if (v_exp != 0) {
                        const float up = power_of_two(v_exp);
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[i] *= up;
                    }
                }
                const size_t out_row = (size_t)(q_start + q_off) * p.num_q_heads + q_head;
                if (p.splits > 1) {
                    const size_t part_row = (size_t)blockIdx.z * p.batch.total_tokens * p.num_q_heads + out_row;
                    float4* dst = reinterpret_cast<float4*>(p.parts + part_row * kHeadDim + 8 * lane);
                    dst[0] = make_float4(v[0], v[1], v[2], v[3]);
                    dst[1] = make_float4(v[4], v[5], v[6], v[7]);
                    if (lane == 0) p.parts_ml[part_row] = make_float2(m, l);
                    continue;
                }
                prefill_finish_row<ROT>(p, v, l, out_row * kHeadDim, lane);
            }
        } else {
            const int r4 = lane >> 3, j = lane & 7;
#pragma unroll 1
            for (int grp = wid; 4 * grp < kPpCtaRows; grp += kPpWarps) {
                const int row = 4 * grp + r4, trow = (int)cluster_rank() * kPpCtaRows + row;
                if ((int)cluster_rank() * kPpCtaRows + 4 * grp >= rows) break;      // warp-uniform
                const int q_off = first_token + trow / p.gqa;
                const size_t out_base = ((size_t)(q_start + q_off) * p.num_q_heads + kv_head * p.gqa + trow % p.gqa) * kHeadDim;
                const bool ok = trow < rows && (p.batch.valid_token_mask == nullptr || p.batch.valid_token_mask[q_start + q_off] != 0);
                const bool gated = ok && p.og.mode != 0 && p.og.gate != nullptr;
                const uint32_t at = smem_u32(smem_raw) + (uint32_t)row * (4u * kPpOutStride);
                const float l = __uint_as_float(lds32(at + 1024u));
                float inv = l > 0.0f ? 1.0f / (ROT ? l * (kPpLutScale * 16.0f) : l) : 0.0f;
                const bool keys = PpFormat<FMT>::has_keys(l);
                if (v_exp != 0) inv *= power_of_two(v_exp);
                float v[32];
                const auto chunk_quad = [&](int k) { return (uint32_t)(2 * (j + 8 * (k >> 1)) + (k & 1)); };
#pragma unroll
                for (int k = 0; k < 8; ++k) lds128f(at + ((ROT ? quad_place(quad_of(j, k)) : chunk_quad(k)) << 4), v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
#pragma unroll
                for (int k = 0; k < 32; ++k) v[k] = keys ? v[k] * inv : 0.0f;
                if (ROT) {
                    rotate_registers<31>(v);
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < 8; ++k) sts128(at + (quad_place(quad_of(j, k)) << 4), __float_as_uint(v[4 * k]), __float_as_uint(v[4 * k + 1]), __float_as_uint(v[4 * k + 2]), __float_as_uint(v[4 * k + 3]));
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < 8; ++k) lds128f(at + (quad_place(chunk_quad(k)) << 4), v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                }
                uint32_t gate[2][4] = {{0u, 0u, 0u, 0u}, {0u, 0u, 0u, 0u}};      // two ahead: a store would hold a load behind it back
                if (gated) {
                    load8_raw(p.og.gate, out_base, j, gate[0]);
                    load8_raw(p.og.gate, out_base, j + 8, gate[1]);
                }
                if (ROT) rotate_registers<4 + 8 + 16>(v);
                const uint32_t signs = ROT ? chunk_signs(j) : 0u;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float x[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] = ROT ? __uint_as_float(__float_as_uint(v[8 * i + e]) ^ (((signs >> (8 * i + e)) & 1u) << 31)) : v[8 * i + e];
                    apply_output_gate8(x, p.og, gate[i & 1], lane, p.io_bf16);
                    if (i < 2 && gated) load8_raw(p.og.gate, out_base, j + 8 * (i + 2), gate[i & 1]);
                    if (ok) store8(p.attn_out, out_base, j + 8 * i, p.io_bf16, x);
                }
            }
        }
    } else if (tid == 0 && p.status != nullptr) {
        atomicOr(p.status, 1);
    }
    // neither CTA leaves (or frees tensor memory) while the other may still signal it
    cluster_sync_all();
    if (wid == 0) {
        tc_fence_after();
        tc2_dealloc(tmem, 512);
    }
}

}  // namespace w34

namespace w34 {
// Tiles and key ranges of a launch, and an estimate of its time in units of one 64-key block (about 1.8 us).  A CTA pair costs its
// blocks and about 7 more for its start, query and output; pairs run in waves of sm_count / 2; a split adds a merge launch (3) and
// its rows, written and read (1e-4 each).  Measured on chunks of 16 to 2048 tokens after 0 to 30 000: within 10 % of the best split.
// A split needs workspace for its rows.
struct PrefillPairPlan {
    long long tiles;
    int splits;
    float cost;
};
// Workspace of a launch that cuts its keys into `splits` ranges: the status word's line, then rows and their (m, l).
static size_t prefill_pair_parts_bytes(const warp34_attention_batch* batch, int num_q_heads, int splits) {
    return splits > 1 ? 256 + (size_t)splits * (size_t)batch->total_tokens * (size_t)num_q_heads * (kHeadDim + 2) * sizeof(float) : 0;
}
// Requests of the longest one's length that leave one token for each of the others.
static long long likely_longs(const warp34_attention_batch* batch) {
    if (batch->max_q_len < 2) return batch->num_reqs;
    const long long n = ((long long)batch->total_tokens - batch->num_reqs + batch->max_q_len - 2) / (batch->max_q_len - 1);
    return n < 1 ? 1 : n > batch->num_reqs ? batch->num_reqs : n;
}
static PrefillPairPlan prefill_pair_plan(const warp34_exec* ex, const warp34_kv_layer_layout* layout, const warp34_attention_batch* batch, int num_q_heads,
                                         int sm_count, int skip_rows) {
    const int gqa = num_q_heads / layout->local_kv_heads, tok_per_tile = kPpRows / gqa;
    long long reqs = batch->num_reqs;      // with tiles: those that are not skipped have more tokens than skip_rows / gqa
    if (skip_rows != 0 && batch->total_tokens / (skip_rows / gqa + 1) < reqs) reqs = batch->total_tokens / (skip_rows / gqa + 1);
    PrefillPairPlan plan;
    plan.tiles = (long long)batch->total_tokens / tok_per_tile + reqs;
    long long likely = plan.tiles;      // that have work
    if (skip_rows != 0) {
        const long long longs = likely_longs(batch);
        if (longs < reqs) { likely -= reqs - longs; reqs = longs; }
    }
    plan.splits = 1;
    plan.cost = 0.0f;
    const long long rows = (long long)batch->total_tokens * num_q_heads;
    const long long blocks = batch->max_seq_len > 0 ? (batch->max_seq_len + kPpKeys - 1) / kPpKeys : 0;
    const long long by_longest = reqs * ((batch->max_q_len + tok_per_tile - 1) / tok_per_tile);
    const long long pairs = (by_longest > 0 && by_longest < likely ? by_longest : likely) * layout->local_kv_heads, at_once = sm_count / 2 > 0 ? sm_count / 2 : 1;
    long long fit = 1;
    if (ex->scratch_ptr != 0 && (ex->scratch_ptr & 15u) == 0 && ex->scratch_size > 256 && rows > 0) {
        fit = kPpMaxSplits;
        while (fit > 1 && prefill_pair_parts_bytes(batch, num_q_heads, (int)fit) > ex->scratch_size) --fit;
    }
    const float mean = (float)blocks - 0.5f * (float)batch->max_q_len / kPpKeys;      // a causal chunk's tiles differ
    for (int n = 1; n <= fit && (n == 1 || n <= blocks); ++n) {
        const float waves = (float)((pairs * n + at_once - 1) / at_once);
        float cost = waves * (mean / (float)n + 7.0f);
        if (cost < (float)blocks / (float)n + 7.0f) cost = (float)blocks / (float)n + 7.0f;
        if (n > 1) cost += 3.0f + 1e-4f * (float)n * (float)rows;
        if (n == 1 || cost < plan.cost) { plan.cost = cost; plan.splits = n; }
    }
    return plan;
}

// The pair kernel for one layer's chunk.  Workspace: a status word, and room for the parts when it splits.
template <int FMT>
static int launch_prefill_pair(const warp34_exec* ex, const warp34_kv_layer_layout* layout, const warp34_attention_batch* batch,
                               const void* q_in, void* attn_out, int num_q_heads, int io_bf16, const OutputGate& og, int sm_count, int skip_rows = 0) {
    int32_t* status = nullptr;      // the first word of the workspace, when there is one
    if (ex->scratch_ptr != 0 && (ex->scratch_ptr & 3u) == 0 && ex->scratch_size >= sizeof(PlanHeader)) {
        status = reinterpret_cast<int32_t*>((uintptr_t)ex->scratch_ptr);   // PlanHeader::status
    }
    if (layout->local_kv_heads > 65535) return (int)cudaErrorInvalidValue;
    PrefillPairParams pp;
    pp.layout = *layout;
    pp.batch = *batch;
    pp.q_in = q_in;
    pp.attn_out = attn_out;
    pp.io_bf16 = io_bf16;
    pp.num_q_heads = num_q_heads;
    pp.gqa = num_q_heads / layout->local_kv_heads;
    pp.tok_per_tile = kPpRows / pp.gqa;
    pp.q_scale = batch->sm_scale * 1.4426950408889634f;
    pp.score_scale = 1.0f;
    if (PpFormat<FMT>::kRotated) {
        pp.q_scale /= kPpLutScale;
    } else if (pp.q_scale != 0.0f) {
        pp.score_scale = fmaxf(fabsf(pp.q_scale), 1.2e-38f);      // (never 0: masked scores are -infinity)
        pp.q_scale = pp.q_scale < 0.0f ? -1.0f : 1.0f;
    }
    pp.status = status;
    pp.og = og;
    pp.skip_tokens = skip_rows / pp.gqa;
    const PrefillPairPlan plan = prefill_pair_plan(ex, layout, batch, num_q_heads, sm_count, skip_rows);
    const long long tiles = plan.tiles;
    if (tiles > 0x3fffffffll) return (int)cudaErrorInvalidValue;
    if (tiles == 0) return 0;
    const long long rows = (long long)batch->total_tokens * num_q_heads;
    pp.splits = plan.splits;
    pp.parts = nullptr;
    pp.parts_ml = nullptr;
    if (pp.splits > 1) {
        pp.parts = reinterpret_cast<float*>((uintptr_t)ex->scratch_ptr + 256);
        pp.parts_ml = reinterpret_cast<float2*>(pp.parts + (size_t)pp.splits * rows * kHeadDim);
    }
    cudaStream_t st = (cudaStream_t)ex->stream;
    const dim3 grid(2u * (unsigned)tiles, (unsigned)layout->local_kv_heads, (unsigned)pp.splits);
    int rc = launch_behind(attention_prefill_pair_kernel<FMT>, grid, kPpThreads, PpSmem<FMT>::kBytes, st, pp);
    if (rc == 0 && pp.splits > 1) {
        rc = launch_behind(prefill_merge_kernel<PpFormat<FMT>::kRotated>, dim3((unsigned)((rows + 3) / 4)), 128, 0, st, pp);
    }
    return rc;
}
}  // namespace w34
