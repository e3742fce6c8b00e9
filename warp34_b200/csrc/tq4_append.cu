// TQ4 quantize-and-append for sm_100a.
//
// Replaces kv_cache_write_kernel / write_kv_row of the reference
// (crates/warp34-kernels/csrc/ops/op_kv_cache.cu:152-218, :325-368) for
// head_dim 256, TQ4 storage and the sign-diagonal + WHT-256 rotation.
//
// Per (token, kv head) and per K / V row:
//   v = sign * x  ->  WHT-256  ->  per 128-half: s = sum v^2,
//   inv = 0.70710678 * rsqrt(s)  ->  code = #{i : v*inv > boundary_i}
//   ->  d = sum(v * c[code]) / sum(c[code]^2)  ->  fp16(d) + 64 packed bytes.
//
// The packed bytes and scales are bit-identical to the reference because every
// fp32 operation is issued in the same association order:
//   * the WHT is the same butterfly network (stage order 1..128);
//   * each of the 24 sums is the reference's 32-lane xor butterfly (levels over
//     column bits 4,3,2,1,0) followed by a sequential sum over the four
//     32-column groups of a half.
// The thread layout is different: 8 lanes hold one row, lane `sub` the 32-column group [32 sub, + 32).  A row is four
// 16-byte loads per lane, the reference's 32-lane butterfly sums are register-only, five of the eight WHT stages as well,
// and a lane's codes are four packed words in place.  A warp encodes 4 rows at once.  (Columns interleaved over the lanes
// instead needed 2-byte loads, a halving exchange per sum and a nibble transpose: 449 instructions a row, 158 us for
// 32 768 tokens x 4 kv heads.)  Bound by issue: parity fixes the order of the operations, so that what is left is to do two columns at
// a time (packed fp32 arithmetic) and to find a code in fewer instructions: 112.8 -> 92.5 us, with the K producer 140.7 -> 122.0.
//
// This translation unit is compiled with -use_fast_math like the reference
// build (crates/warp34-kernels/build.rs:56-59), so rsqrtf() and '/' lower to the
// same approximate instructions and denormals flush the same way.
#include "tq4_common.cuh"

#include <cuda_bf16.h>

namespace w34 {

// The reference computes warp_reduce_sum(a * b): the product is rounded, then summed by the
// butterfly, and nvcc does not contract the butterfly's first add with the product into an fma
// (all eight contracted / uncontracted combinations of the three sums were compared with the
// reference kernels built for sm_100a: only "none contracted" is bit-identical).  Products and adds
// below are therefore explicit __fmul_rn / __fadd_rn.

constexpr float kBinScale = 58.75f;
constexpr int kBins = 128;

// code = #{i : rv > boundary_i} for the 15 ascending boundaries.  rv falls into one of kBins equal bins around 0 (kBinScale a unit,
// chosen so that no bin holds two boundaries and none lies within a fifth of a bin of an edge; |rv| is at most 0.7072, 42 bins); the
// bin's entry {boundary inside it or infinity, boundaries below it} settles the code with one comparison.  `bins`: shared-memory
// address of the table, a multiple of its size.  NaN ends in the last entry, which no number reaches, and gives 0 as the
// comparison chain does; zeros of either sign give 7.  (With the magnitude's bins and the sign handled apart a code took eleven
// instructions instead of seven.)
__device__ __forceinline__ int tq4_bucket(float rv, uint32_t bins) {
    const uint32_t bin = __float_as_uint(__fmaf_rn(rv, kBinScale, 12582912.0f + (float)(kBins / 2)));
    float boundary;
    uint32_t below;
    asm("ld.shared.v2.b32 {%0, %1}, [%2];" : "=f"(boundary), "=r"(below) : "r"(((bin << 3) & (8u * kBins - 8u)) | bins));
    return (int)below + (rv > boundary ? 1 : 0);
}

// The rest of a group's butterfly, column bits 2, 1, 0, after its levels over bits 4 and 3.
__device__ __forceinline__ float group_total(const float (&t)[8]) {
    return __fadd_rn(__fadd_rn(__fadd_rn(t[0], t[4]), __fadd_rn(t[2], t[6])), __fadd_rn(__fadd_rn(t[1], t[5]), __fadd_rn(t[3], t[7])));
}

// Sequential sum (((0 + t0) + t1) + t2) + t3 of the group totals held by four lanes.
__device__ __forceinline__ float half_sum(float t, int lane0) {
    // The reference starts from 0.0f (0 + (-0) = +0 matters for all-zero rows).
    float s = __fadd_rn(0.0f, __shfl_sync(0xffffffffu, t, lane0));
    s = __fadd_rn(s, __shfl_sync(0xffffffffu, t, lane0 + 1));
    s = __fadd_rn(s, __shfl_sync(0xffffffffu, t, lane0 + 2));
    return __fadd_rn(s, __shfl_sync(0xffffffffu, t, lane0 + 3));
}

// ---- two columns at a time ------------------------------------------------------------------------------
// The packed forms round each half as the scalar instruction does (subnormals flushed, as everywhere in this unit), at half the
// instructions, which is what the kernel is bound by.  a - b is fma(b, -1, a): the same number, signed zeros included.
typedef unsigned long long Pair;
__device__ __forceinline__ Pair pair_of(float a, float b) { return (Pair)__float_as_uint(a) | ((Pair)__float_as_uint(b) << 32); }
__device__ __forceinline__ float first(Pair p) { return __uint_as_float((uint32_t)p); }
__device__ __forceinline__ float second(Pair p) { return __uint_as_float((uint32_t)(p >> 32)); }
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
    Pair r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
    Pair r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
    Pair r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

struct AppendParams {
    warp34_kv_layer_layout layout;
    warp34_attention_batch batch;
    const uint16_t* k_in;   // fp16 or bf16 bits, see the kernel's template argument
    const uint16_t* v_in;
    int k_row_stride;
    int v_row_stride;
    int total_rows;  // total_tokens * local_kv_heads * 2
    // producer fused in front of the K rows (PRODUCER builds only)
    const uint16_t* k_norm_w;   // fp16 [256]
    const int32_t* positions;   // [planes][pos_plane_stride]
    int pos_plane_stride;
    int rotary_dim;
    int mrope_s1, mrope_s2;
    float rope_theta;
    float rms_eps;
};

// Accurate libdevice routines, by name, as the reference's producer calls them
// (op_norms_rope_act.cu:14-16): -use_fast_math must not swap them for the approximate ones.
extern "C" __device__ float __nv_sinf(float);
extern "C" __device__ float __nv_cosf(float);
extern "C" __device__ float __nv_powf(float, float);

constexpr int kAppendBlocksPerSm = 7;
constexpr int kProducerBlocksPerSm = 5;

struct ProducerShared {
    float w1[8 * 36];                     // 1 + w of columns 32 s + c at 36 s + c
    float inv_freq[kHeadDim / 2];
    float sin_t[4][4][kHeadDim / 2], cos_t[4][4][kHeadDim / 2];      // per warp and row
    __align__(16) uint16_t rows[4][4][kHeadDim + 8];
};
template <bool PRODUCER> struct AppendShared { };
template <> struct AppendShared<true> { ProducerShared s; };

// The producer of the reference's layer, K half: per-head Gemma RMS norm (weight 1 + w) and partial
// interleaved 3-D mRoPE (fused_qk_rmsnorm_rope_gate_f16_kernel, op_norms_rope_act.cu:524-680), on the fp16 row a
// lane group holds (lane `sub`: columns 32 sub .. + 31 as 16 packed pairs), in place: the values that kernel would have
// written to k_out, so that the packed bytes are the same as those of the two-kernel sequence.  Arithmetic order is the
// reference's:
//  * sum of squares: its thread t adds the squares of columns 8 t .. 8 t + 7 in order, as a chain of fused multiply-adds
//    from 0, then a 32-wide xor butterfly: here a lane runs the four chains t = 4 sub + j;
//  * x * inv_rms, then * (1 + w), each rounded, then to fp16;
//  * angle = position * (1 / powf(theta, 2 i / rotary_dim)), sine and cosine rounded to fp16.
// The rotated columns (at most the first rotary_dim) go through shared memory, eight lanes a row.  Every lane of the warp
// takes part.
__device__ __forceinline__ void k_producer(uint32_t (&raw)[16], int sub, int row, int tok, const AppendParams& p, ProducerShared& sh) {
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float part[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float acc = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&raw[4 * j + i]));
            acc = __fmaf_rn(f.x, f.x, acc);
            acc = __fmaf_rn(f.y, f.y, acc);
        }
        part[j] = acc;
    }
    // its 32-wide xor butterfly 16, 8, 4, 2, 1: thread bits 4..2 are sub, bits 1 and 0 are j
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j) part[j] = __fadd_rn(part[j], __shfl_xor_sync(0xffffffffu, part[j], h));
    }
    const float sum_sq = __fadd_rn(__fadd_rn(part[0], part[2]), __fadd_rn(part[1], part[3]));
    const float inv_rms = rsqrtf(sum_sq / (float)kHeadDim + p.rms_eps);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float4 w = *reinterpret_cast<const float4*>(&sh.w1[36 * sub + 4 * i]);
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw[2 * i]));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&raw[2 * i + 1]));
        const __half2 ha = __floats2half2_rn(__fmul_rn(__fmul_rn(a.x, inv_rms), w.x), __fmul_rn(__fmul_rn(a.y, inv_rms), w.y));
        const __half2 hb = __floats2half2_rn(__fmul_rn(__fmul_rn(b.x, inv_rms), w.z), __fmul_rn(__fmul_rn(b.y, inv_rms), w.w));
        raw[2 * i] = *reinterpret_cast<const uint32_t*>(&ha);
        raw[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&hb);
    }
    const int half_rot = p.rotary_dim >> 1;
    if (half_rot == 0) return;
    // sines and cosines: the four rows of a warp are usually the kv heads of one token, whose angles are then computed once
    const bool one_token = __all_sync(0xffffffffu, tok == __shfl_sync(0xffffffffu, tok, 0));
    const int trow = one_token ? 0 : row;
    for (int i = one_token ? lane : sub; i < half_rot; i += one_token ? 32 : 8) {
        int plane = 0;
        if ((i % 3) == 1 && i < p.mrope_s1 * 3) {
            plane = 1;
        } else if ((i % 3) == 2 && i < p.mrope_s2 * 3) {
            plane = 2;
        }
        const float pos = (float)p.positions[(size_t)plane * p.pos_plane_stride + tok];
        const float angle = pos * sh.inv_freq[i];
        sh.sin_t[wid][trow][i] = __half2float(__float2half_rn(__nv_sinf(angle)));
        sh.cos_t[wid][trow][i] = __half2float(__float2half_rn(__nv_cosf(angle)));
    }
    uint16_t* line = sh.rows[wid][row];
    uint4* mine = reinterpret_cast<uint4*>(line + 32 * sub);
    const bool rotates = 32 * sub < p.rotary_dim;
    if (rotates) {
#pragma unroll
        for (int i = 0; i < 4; ++i) mine[i] = make_uint4(raw[4 * i], raw[4 * i + 1], raw[4 * i + 2], raw[4 * i + 3]);
    }
    __syncwarp();
    for (int i = sub; i < half_rot; i += 8) {
        const float sin_a = sh.sin_t[wid][trow][i], cos_a = sh.cos_t[wid][trow][i];
        const float x1 = __half2float(__ushort_as_half(line[i]));
        const float x2 = __half2float(__ushort_as_half(line[i + half_rot]));
        line[i] = __half_as_ushort(__float2half(x1 * cos_a - x2 * sin_a));
        line[i + half_rot] = __half_as_ushort(__float2half(x2 * cos_a + x1 * sin_a));
    }
    __syncwarp();
    if (rotates) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 q = mine[i];
            raw[4 * i] = q.x; raw[4 * i + 1] = q.y; raw[4 * i + 2] = q.z; raw[4 * i + 3] = q.w;
        }
    }
    __syncwarp();   // the line and the angles are rewritten by the warp's next group
}

// IN_BF16: activations are bf16 instead of fp16.  Values that both types can hold encode to the
// same bytes; bf16 values beyond the fp16 range are simply larger fp32 inputs.
// PRODUCER: K rows go through k_producer() first (fp16 activations only).
template <bool IN_BF16, bool PRODUCER>
__global__ void __launch_bounds__(128, PRODUCER ? kProducerBlocksPerSm : kAppendBlocksPerSm) tq4_append_kernel(const AppendParams p) {
    __shared__ float s_centroid[16];
    __shared__ __align__(8 * kBins) uint2 s_bin[kBins];
    __shared__ AppendShared<PRODUCER> s_prod;
    if (threadIdx.x < 16) s_centroid[threadIdx.x] = tq4_centroid(threadIdx.x);
    static_assert(kBins == 128, "one entry per thread");
    {
        uint2 e = make_uint2(0x7f800000u, 0u);
        for (int k = 0; k < 15; ++k) {
            const int bin = kBins / 2 + (int)rintf(tq4_boundary(k) * kBinScale);
            if (bin < (int)threadIdx.x) ++e.y;
            if (bin == (int)threadIdx.x) e.x = c_boundary_bits[k];
        }
        if (threadIdx.x == kBins - 1) e.y = 0u;
        s_bin[threadIdx.x] = e;
    }
    const int lane = threadIdx.x & 31;
    const int sub = lane & 7;
    uint32_t sign[16];        // of the lane's columns, as the sign bits of packed 16-bit pairs
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const uint32_t m = c_sign_mask[sub] >> (2 * i);
        sign[i] = ((m & 1u) << 15) | ((m & 2u) << 30);
    }
    const uint32_t bins = (uint32_t)__cvta_generic_to_shared(s_bin);
    // butterfly direction of the three cross-lane WHT stages: upper lanes compute o - v
    const float one_f = __uint_as_float(0x3f800000u | (uint32_t)(p.layout.head_dim - kHeadDim));      // 1, see quarter_sums
    const Pair one = pair_of(one_f, one_f);
    const float dir1 = (sub & 1) ? -1.0f : 1.0f, dir2 = (sub & 2) ? -1.0f : 1.0f, dir4 = (sub & 4) ? -1.0f : 1.0f;
    // This kernel may start while the last blocks of the one before it finish (nothing above touches global memory), and an
    // attention kernel launched behind it may set itself up meanwhile.
    grid_dependency_wait();
    grid_launch_dependents();
    if constexpr (PRODUCER) {
        for (int i = threadIdx.x; i < kHeadDim; i += blockDim.x) {
            s_prod.s.w1[36 * (i >> 5) + (i & 31)] = 1.0f + __half2float(__ushort_as_half(p.k_norm_w[i]));
        }
        for (int i = threadIdx.x; i < (p.rotary_dim >> 1); i += blockDim.x) {
            s_prod.s.inv_freq[i] = __fdiv_rn(1.0f, __nv_powf(p.rope_theta, (float)(2 * i) / (float)p.rotary_dim));
        }
    }
    __syncthreads();

    const int heads = p.layout.local_kv_heads;
    const int warps_total = gridDim.x * 4;
    // A warp takes four rows at a time.  Plain append: rows 4 q .. 4 q + 3 of the list (token, head, K | V).
    // With the producer in front, a group holds four K rows or four V rows (groups alternate), so that the
    // norm and the rotation run for K groups only and not for the V rows that would share a warp with them.
    const int pairs = p.total_rows >> 1;                      // (token, head) pairs
    const int quads = PRODUCER ? 2 * ((pairs + 3) >> 2) : (p.total_rows + 3) >> 2;
#pragma unroll 1
    for (int quad = blockIdx.x * 4 + (threadIdx.x >> 5); quad < quads; quad += warps_total) {
        // ---- resolve the row: (token, head, K or V), masks, destination ------------------
        const int row_id = quad * 4 + (lane >> 3);
        const int which = PRODUCER ? (quad & 1) : (row_id & 1);
        const int th = PRODUCER ? ((quad >> 1) * 4 + (lane >> 3)) : (row_id >> 1);
        bool active = PRODUCER ? (th < pairs) : (row_id < p.total_rows);
        const int tok = active ? th / heads : 0;
        const int head = th - tok * heads;
        int slot = -1;
        if (active) {
            if (p.batch.valid_token_mask != nullptr && p.batch.valid_token_mask[tok] == 0) active = false;
        }
        if (active && p.batch.valid_req_mask != nullptr && p.batch.query_start_loc != nullptr &&
            p.batch.num_reqs > 0) {
            const int req = find_request(p.batch.query_start_loc, p.batch.num_reqs, tok);
            if (req < 0 || p.batch.valid_req_mask[req] == 0) active = false;
        }
        if (active) {
            slot = p.batch.write_slot_mapping[tok];
            if (slot < 0 || !write_slot_ok(slot, kInAppend)) active = false;
        }
        // All 8 lanes of a row agree on `active`; rows of a warp may differ, and every lane
        // still takes part in the shuffles below.
        // ---- load: 32 columns as packed pairs ----------------------------------------------
        uint32_t raw[16];
        {
            const uint16_t* src = (which == 0 ? p.k_in + (size_t)tok * p.k_row_stride : p.v_in + (size_t)tok * p.v_row_stride) +
                                  head * kHeadDim + 32 * sub;
            if (active && ((uintptr_t)src & 15u) == 0u) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 q = reinterpret_cast<const uint4*>(src)[i];
                    raw[4 * i] = q.x; raw[4 * i + 1] = q.y; raw[4 * i + 2] = q.z; raw[4 * i + 3] = q.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) raw[i] = active ? (uint32_t)src[2 * i] | ((uint32_t)src[2 * i + 1] << 16) : 0u;
            }
        }
        if constexpr (PRODUCER) {
            if (which == 0) k_producer(raw, sub, lane >> 3, tok, p, s_prod.s);   // warp-uniform: a group is all K or all V
        }
        Pair v[16];      // columns 2 i, 2 i + 1
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint32_t w = raw[i] ^ sign[i];
            const float2 f = IN_BF16 ? make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u))
                                     : __half22float2(*reinterpret_cast<const __half2*>(&w));
            v[i] = pair_of(__fadd_rn(f.x, f.y), __fsub_rn(f.x, f.y));      // stage 1 of the transform
        }

        // ---- WHT-256: stages 1 .. 16 in registers, 32, 64, 128 across lanes --------------------------
        const Pair minus_one = pair_of(-1.0f, -1.0f);
#pragma unroll
        for (int s = 1; s < 16; s <<= 1) {
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                if ((r & s) == 0) {
                    const Pair a = v[r], b = v[r | s];
                    v[r] = add2(a, b);
                    v[r | s] = fma2(b, minus_one, a);
                }
            }
        }
        // lower lane: v + o, upper lane: o - v; fma(+-1, v, o) is the same single rounding.
        auto across = [&](float dir, int d) {
            const Pair dir2 = pair_of(dir, dir);
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const Pair o = pair_of(__shfl_xor_sync(0xffffffffu, first(v[r]), d), __shfl_xor_sync(0xffffffffu, second(v[r]), d));
                v[r] = fma2(dir2, v[r], o);
            }
        };
        across(dir1, 1);
        across(dir2, 2);
        across(dir4, 4);
        // The transform's factor 1/16.  Sums of fp16 values are multiples of 2^-24 far below the overflow threshold, so
        // that a power of two commutes with every rounding that follows: it is left out and put back into the scale.
        constexpr float kSq = IN_BF16 ? 1.0f : 256.0f, kBack = IN_BF16 ? 1.0f : 0.0625f;
        if (IN_BF16) {
            const Pair sixteenth = pair_of(0.0625f, 0.0625f);
#pragma unroll
            for (int r = 0; r < 16; ++r) v[r] = mul2(v[r], sixteenth);
        }

        // ---- scale of the lane's half, codes, centroids, least-squares sums ----------------------------------
        // (a b of columns c + c of 16 further) + (those 8 and 24 further), for columns 2 r, 2 r + 1.  A sum of products is written
        // fma(x, one, y): the assembler makes one rounding of a packed product and the add behind it, .rn or not, unless the add is
        // itself a product that it cannot know (22 of a million scales then differ; tests/test_gpu_append_edges.py holds rows that show it).
        auto quarter_sums = [&](const Pair (&x)[16], const Pair (&y)[16], float (&t)[8]) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const Pair near = fma2(mul2(x[r], y[r]), one, mul2(x[r + 8], y[r + 8]));
                const Pair far = fma2(mul2(x[r + 4], y[r + 4]), one, mul2(x[r + 12], y[r + 12]));
                const Pair q = add2(near, far);
                t[2 * r] = first(q);
                t[2 * r + 1] = second(q);
            }
        };
        const int half_lane = lane & ~3;
        float inv;
        {
            float t[8];
            quarter_sums(v, v, t);
            const float s = half_sum(group_total(t), half_lane);
            inv = (s > 1e-20f * kSq) ? (0.7071067811865475f * rsqrtf(s)) : 0.0f;
        }
        uint32_t nib[4] = {0u, 0u, 0u, 0u};
        Pair c[16];
        const Pair inv2 = pair_of(inv, inv);
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const Pair x = mul2(v[r], inv2);
            const int qa = tq4_bucket(first(x), bins), qb = tq4_bucket(second(x), bins);
            nib[r >> 2] += (uint32_t)qa * (1u << (8 * (r & 3))) + (uint32_t)qb * (1u << (8 * (r & 3) + 4));   // disjoint nibbles: add == or
            c[r] = pair_of(s_centroid[qa], s_centroid[qb]);
        }
        float vct[8], cct[8];
        quarter_sums(v, c, vct);
        quarter_sums(c, c, cct);
        const float vc = half_sum(group_total(vct), half_lane);
        const float cc = half_sum(group_total(cct), half_lane);
        const float d = (cc > 1e-10f) ? (vc / cc) * kBack : 0.0f;
        const uint32_t dh = __half_as_ushort(__float2half_rn(d));      // of the lane's half

        // ---- the row as 33 aligned 32-bit words: W0 = d0 | word 0 << 16, Wk = hi16(word k - 1) | lo16(word k) << 16
        //      (k = 1..15), W16 = hi16(word 15) | d1 << 16, W(17 + k) = word 16 + k; this lane holds words 4 sub .. + 3 ----
        const uint32_t before = __shfl_up_sync(0xffffffffu, nib[3], 1);
        if (active) {
            uint8_t* dst = which == 0 ? (uint8_t*)(uintptr_t)p.layout.k_base + (size_t)(slot >> 4) * p.layout.k_page_stride_bytes +
                                            (size_t)head * p.layout.k_head_stride_bytes + (size_t)(slot & 15) * p.layout.k_token_stride_bytes
                                      : (uint8_t*)(uintptr_t)p.layout.v_base + (size_t)(slot >> 4) * p.layout.v_page_stride_bytes +
                                            (size_t)head * p.layout.v_head_stride_bytes + (size_t)(slot & 15) * p.layout.v_token_stride_bytes;
            if ((((uintptr_t)dst) & 3u) == 0u) {
                uint32_t* w = reinterpret_cast<uint32_t*>(dst) + 4 * sub;
                if (sub < 4) {
                    w[0] = __funnelshift_l(sub == 0 ? dh << 16 : before, nib[0], 16);
                    w[1] = __funnelshift_l(nib[0], nib[1], 16);
                    w[2] = __funnelshift_l(nib[1], nib[2], 16);
                    w[3] = __funnelshift_l(nib[2], nib[3], 16);
                } else {
                    if (sub == 4) w[0] = (before >> 16) | (dh << 16);
                    w[1] = nib[0];
                    w[2] = nib[1];
                    w[3] = nib[2];
                    w[4] = nib[3];
                }
            } else {
                // Row base not 4-byte aligned: 16-bit stores (rows are always 2-byte aligned).
                uint16_t* h = reinterpret_cast<uint16_t*>(dst) + 33 * (sub >> 2);
                if ((sub & 3) == 0) h[0] = (uint16_t)dh;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    h[1 + 8 * (sub & 3) + 2 * i] = (uint16_t)nib[i];
                    h[2 + 8 * (sub & 3) + 2 * i] = (uint16_t)(nib[i] >> 16);
                }
            }
        }
    }
}

W34_BOUNDS_HOST_HOOKS(append)

}  // namespace w34

#include "kv8_append.cuh"

namespace w34 {
// Unrotated 8-bit layers: one warp per row.
static int launch_append_kv8(const warp34_exec* ex, const warp34_kv_layer_layout* layout,
                             const warp34_attention_batch* batch, const void* k_in, const void* v_in,
                             int k_row_stride, int v_row_stride) {
    const int min_stride = layout->local_kv_heads * layout->head_dim;
    if (k_row_stride < min_stride || v_row_stride < min_stride) return (int)cudaErrorInvalidValue;
    if (batch->write_slot_mapping == nullptr || layout->k_base == 0 || layout->v_base == 0) {
        return (int)cudaErrorInvalidValue;
    }
    // Scales are fp32 and the codes are stored as 32-bit words: every row must be 4-byte aligned
    // (the reference's row structs have the same alignment).
    if ((layout->k_base | layout->v_base | layout->k_page_stride_bytes | layout->k_head_stride_bytes |
         layout->k_token_stride_bytes | layout->v_page_stride_bytes | layout->v_head_stride_bytes |
         layout->v_token_stride_bytes) & 3u) {
        return (int)cudaErrorInvalidValue;
    }
    AppendParams p;
    p.layout = *layout;
    p.batch = *batch;
    p.k_in = static_cast<const uint16_t*>(k_in);
    p.v_in = static_cast<const uint16_t*>(v_in);
    p.k_row_stride = k_row_stride;
    p.v_row_stride = v_row_stride;
    const long long rows = 2ll * batch->total_tokens * layout->local_kv_heads;
    if (rows > 0x7fffffffll) return (int)cudaErrorInvalidValue;
    p.total_rows = (int)rows;
    const bool aligned = ((((uintptr_t)k_in | (uintptr_t)v_in) & 15u) == 0u) && (k_row_stride & 7) == 0 && (v_row_stride & 7) == 0;
    const unsigned blocks8 = (unsigned)((rows / 2 + 3) / 4);   // a warp per (token, head)
    return launch_behind(aligned ? kv8_append_kernel<true> : kv8_append_kernel<false>, dim3(blocks8), 128, 0, (cudaStream_t)ex->stream, p);
}

struct KProducer {
    const void* k_norm_w;
    const int32_t* positions;
    int pos_plane_stride, rotary_dim, mrope_s1, mrope_s2;
    float rope_theta, rms_eps;
};

static int launch_append(const warp34_exec* ex, const warp34_kv_layer_layout* layout,
                         const warp34_attention_batch* batch, const void* k_in, const void* v_in,
                         int k_row_stride, int v_row_stride, bool in_bf16, const KProducer* producer = nullptr) {
    if (ex == nullptr || layout == nullptr || batch == nullptr || k_in == nullptr || v_in == nullptr) {
        return (int)cudaErrorInvalidValue;
    }
    if (producer != nullptr) {
        if (producer->k_norm_w == nullptr || producer->positions == nullptr) return (int)cudaErrorInvalidValue;
        // both elements of a rotated pair must sit in one lane: rotary_dim / 2 a multiple of 8
        if (producer->rotary_dim < 0 || producer->rotary_dim > kHeadDim || (producer->rotary_dim & 15) != 0) {
            return (int)cudaErrorNotSupported;
        }
    }
    if (batch->total_tokens <= 0 || layout->local_kv_heads <= 0) return 0;
    if (kv8_layout_ok(layout)) {
        if (in_bf16 || producer != nullptr) return (int)cudaErrorNotSupported;
        return launch_append_kv8(ex, layout, batch, k_in, v_in, k_row_stride, v_row_stride);
    }
    if (layout->head_dim != kHeadDim || layout->block_size != kPageTokens ||
        layout->k_format != WARP34_KV_FORMAT_TQ4 || layout->v_format != WARP34_KV_FORMAT_TQ4 ||
        layout->k_transform != WARP34_KV_TRANSFORM_RADEMACHER_WHT256 ||
        layout->v_transform != WARP34_KV_TRANSFORM_RADEMACHER_WHT256) {
        return (int)cudaErrorNotSupported;
    }
    const int min_stride = layout->local_kv_heads * layout->head_dim;
    if (k_row_stride < min_stride || v_row_stride < min_stride) return (int)cudaErrorInvalidValue;
    if (batch->write_slot_mapping == nullptr || layout->k_base == 0 || layout->v_base == 0) {
        return (int)cudaErrorInvalidValue;
    }
    // Scales are stored with 16-bit accesses: every row must be 2-byte aligned.
    if ((layout->k_base | layout->v_base | layout->k_page_stride_bytes | layout->k_head_stride_bytes |
         layout->k_token_stride_bytes | layout->v_page_stride_bytes | layout->v_head_stride_bytes |
         layout->v_token_stride_bytes) & 1u) {
        return (int)cudaErrorInvalidValue;
    }
    AppendParams p;
    p.layout = *layout;
    p.batch = *batch;
    p.k_in = static_cast<const uint16_t*>(k_in);
    p.v_in = static_cast<const uint16_t*>(v_in);
    p.k_row_stride = k_row_stride;
    p.v_row_stride = v_row_stride;
    const long long rows = 2ll * batch->total_tokens * layout->local_kv_heads;
    if (rows > 0x7fffffffll) return (int)cudaErrorInvalidValue;
    p.total_rows = (int)rows;
    // 4 warps x 4 rows per block and pass; each warp then strides over the remaining row groups,
    // so per-thread constants are set up once.  The grid is what the GPU can hold at once.
    const long long blocks_needed = (rows + 15) / 16;
    static int sm_count_cache[64];
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
        if (sm_count_cache[dev] == 0) {
            int n = 0;
            if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0) {
                sm_count_cache[dev] = n;
            }
        }
        if (sm_count_cache[dev] > 0) sms = sm_count_cache[dev];
    }
    const long long resident = (long long)sms * (producer != nullptr ? kProducerBlocksPerSm : kAppendBlocksPerSm);
    const unsigned blocks = (unsigned)(blocks_needed < resident ? blocks_needed : resident);
    p.k_norm_w = nullptr;
    p.positions = nullptr;
    p.pos_plane_stride = p.rotary_dim = p.mrope_s1 = p.mrope_s2 = 0;
    p.rope_theta = p.rms_eps = 0.0f;
    if (producer != nullptr) {
        if (in_bf16) return (int)cudaErrorNotSupported;
        p.k_norm_w = static_cast<const uint16_t*>(producer->k_norm_w);
        p.positions = producer->positions;
        p.pos_plane_stride = producer->pos_plane_stride;
        p.rotary_dim = producer->rotary_dim;
        p.mrope_s1 = producer->mrope_s1;
        p.mrope_s2 = producer->mrope_s2;
        p.rope_theta = producer->rope_theta;
        p.rms_eps = producer->rms_eps;
        return launch_behind(tq4_append_kernel<false, true>, dim3(blocks), 128, 0, (cudaStream_t)ex->stream, p);
    }
    if (in_bf16) return launch_behind(tq4_append_kernel<true, false>, dim3(blocks), 128, 0, (cudaStream_t)ex->stream, p);
    return launch_behind(tq4_append_kernel<false, false>, dim3(blocks), 128, 0, (cudaStream_t)ex->stream, p);
}
}  // namespace w34

extern "C" int warp34_kv_cache_write_strided(const warp34_exec* ex, const warp34_kv_layer_layout* layout,
                                             const warp34_attention_batch* batch, const void* k_in,
                                             const void* v_in, int k_row_stride, int v_row_stride) {
    return w34::launch_append(ex, layout, batch, k_in, v_in, k_row_stride, v_row_stride, false);
}

// K-norm + RoPE + rotate / quantise / pack in one kernel: the K half of the reference's
// warp34_fused_qk_rmsnorm_rope_gate_strided_f16 followed by its warp34_kv_cache_write_strided
// (crates/warp34-host/src/model/forward.rs:1109-1149), without the fp16 K rows going through HBM.
extern "C" int warp34_fused_k_rmsnorm_rope_kv_cache_write_f16(
    const warp34_exec* ex, const warp34_kv_layer_layout* layout, const warp34_attention_batch* batch,
    const void* k_in, const void* v_in, const void* k_norm_w, const int32_t* positions, int pos_plane_stride,
    int rotary_dim, int mrope_s0, int mrope_s1, int mrope_s2, int k_row_stride, int v_row_stride, float rope_theta,
    float rms_eps) {
    (void)mrope_s0;   // the first section needs no bound: plane 0 is the default (op_norms_rope_act.cu:640-646)
    w34::KProducer pr;
    pr.k_norm_w = k_norm_w;
    pr.positions = positions;
    pr.pos_plane_stride = pos_plane_stride;
    pr.rotary_dim = rotary_dim;
    pr.mrope_s1 = mrope_s1;
    pr.mrope_s2 = mrope_s2;
    pr.rope_theta = rope_theta;
    pr.rms_eps = rms_eps;
    return w34::launch_append(ex, layout, batch, k_in, v_in, k_row_stride, v_row_stride, false, &pr);
}

extern "C" int warp34_kv_cache_write(const warp34_exec* ex, const warp34_kv_layer_layout* layout,
                                     const warp34_attention_batch* batch, const void* k_in,
                                     const void* v_in) {
    if (layout == nullptr) return (int)cudaErrorInvalidValue;
    const int stride = layout->local_kv_heads * layout->head_dim;
    return w34::launch_append(ex, layout, batch, k_in, v_in, stride, stride, false);
}

extern "C" int warp34_tq4_kv_cache_write_strided_bf16(const warp34_exec* ex, const warp34_kv_layer_layout* layout,
                                                      const warp34_attention_batch* batch, const void* k_in,
                                                      const void* v_in, int k_row_stride, int v_row_stride) {
    return w34::launch_append(ex, layout, batch, k_in, v_in, k_row_stride, v_row_stride, true);
}
