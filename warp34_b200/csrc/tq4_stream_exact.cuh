// Decode, verify and query-sparse attention over TQ4 pages with value + residual operands: the default streaming kernel.
// Included by tq4_attention.cu (shares the plan, the PTX wrappers, the stage layout and the partial format with the
// single-operand build).
//
// A worker is one warp: it streams its share of (request, kv head, 8-row group, page) units through a private ring of
// shared-memory slots, two pages (32 keys) at a time, and computes S^T = K Q'^T and O^T += V^T (P d_v)^T with mma.sync
// m16n8k16 (fp32 accumulators).
//
// The score product puts value and residual of the SAME keys into one A fragment: rows 0-7 of the MMA are the centroids
// of eight keys, rows 8-15 their fp16 rounding residuals.  One 8-byte table look-up returns (value pair, residual pair)
// into two neighbouring registers, two look-ups fill the four registers of the fragment in place, and the sum of both
// products is c0 + c2, c1 + c3 of a lane's accumulators.  (With values of sixteen keys in one fragment and residuals in
// another, every fragment had to be gathered with register moves: about 220 of 965 instructions per unit.)  The query's
// rounding residual, fp16 as well, meets values only: one MMA takes those of both fragments' keys (its four operands are moved next to
// each other), 80 MMAs a page instead of 96 with the residuals' half of each fragment along: 64 sequences of 8192 to 32768 on 24 / 4
// heads 495 -> 473 us.  What falls away, query residual by centroid residual, is at most 9.3e-8 of sum |q k| (the centroids lie within 9.5e-5 of
// fp16 values, the residual is below 2^-10 of q), a twentieth of what the residual's own step of 1/255 leaves; the scores' error against
// float64 over normal, outlier, sparse and large queries is 1 to 14 % lower than with all three products in one accumulator (2.08e-6 of the
// scores instead of 2.10e-6 on the benchmark's values), and the same to three digits with the product added to the separate one.
// Items of at most four rows keep it, at no cost (see x_share).
#pragma once

namespace w34 {

constexpr int kXThreads = kExactWarps * 32;
constexpr uint32_t kXSlot = 2u * (uint32_t)kStageStride;     // two pages; two slots per warp

__device__ __forceinline__ uint32_t lds32_lut_residual(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1+4];" : "=r"(v) : "r"(addr));
    return v;
}

// One warp's place in the kernel: its ring, the lane's part in the fragments, the state of its copies.
struct XWarp {
    uint32_t ring, bars;          // two slots of two pages; one mbarrier per slot
    uint32_t lut_lane, lutk_lane; // V values; K (and V) value + residual.  Byte 1 is zero: the code byte goes there
    int lane, gid, tig;
    int key_a;                    // score fragments: MMA row gid <-> token key_a of the page (first fragment), key_a + 4 (second)
    int kv0;                      // output fragments: thread tig owns tokens kv0 + {0, 1, 4, 5} (k positions 2 tig, + 1, + 8, + 9)
    uint32_t vwb;
    uint32_t phase_bits, pending; // bit s: parity to wait for on slot s; a copy into slot s not yet awaited
    bool failed;
};

__device__ __forceinline__ void x_init(XWarp& x, uint32_t lut_addr, uint32_t ring, uint32_t bars) {
    x.lane = threadIdx.x & 31;
    x.gid = x.lane >> 2;
    x.tig = x.lane & 3;
    x.key_a = (x.gid & 3) + 8 * (x.gid >> 2);
    x.kv0 = 2 * (x.tig & 1) + 8 * (x.tig >> 1);
    x.vwb = 4u * (uint32_t)(x.gid >> 1) + (uint32_t)(x.gid & 1);
    x.lut_lane = lut_addr + 128u + 4u * (uint32_t)x.lane;
    x.lutk_lane = lut_addr + 8u * (uint32_t)(x.lane & 15);
    x.ring = ring;
    x.bars = bars;
    x.phase_bits = x.pending = 0u;
    x.failed = false;
    if (x.lane == 0) {
        for (int s = 0; s < 2; ++s) mbar_init(bars + 8u * s, 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// Byte-pair tables: (value pair, residual pair) in 16 copies of 8 bytes for K, value pair in 32 copies of 4 bytes for V in the
// upper half of the same 256-byte entry; conflict-free for any data.  Lane k of a warp makes the words of entry
// k * warps + warp, the warp then spreads them one entry at a time (a quarter of the instructions of making them per copy).
__device__ __forceinline__ void x_build_tables(uint32_t lut_addr) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    static_assert(32 * kExactWarps == 256, "one entry per thread");
    const int mine = lane * kExactWarps + wid;
    const float c0 = kLutScale * tq4_centroid(mine & 15), c1 = kLutScale * tq4_centroid(mine >> 4);
    const uint32_t hi = pack_half2(c0, c1);
    const float2 hf = __half22float2(*reinterpret_cast<const __half2*>(&hi));
    const uint32_t lo = pack_half2((c0 - hf.x) * kResidualScale, (c1 - hf.y) * kResidualScale);
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
        const uint32_t h = __shfl_sync(0xffffffffu, hi, k), l = __shfl_sync(0xffffffffu, lo, k);
        const uint32_t entry = lut_addr + (uint32_t)(k * kExactWarps + wid) * 256u;
        sts32(entry + 4u * (uint32_t)lane, (lane & 1) ? l : h);
        sts32(entry + 128u + 4u * (uint32_t)lane, h);
    }
}

// Query fragments of one work item as qprep_block() lays them out: value, and residual as bytes in units of the row's step,
// widened here once per item.  `word(i)` reads word i of this lane.
// FOUR: `word` reads the words of row gid % 4, and the lanes of rows 4-7 keep its residual in place of a value.
template <bool FOUR, class Word>
__device__ __forceinline__ void x_load_query(Word word, uint32_t (&qb)[16][2], uint32_t (&ql)[FOUR ? 1 : 16][2]) {
    const float step = __uint_as_float(word(48));
    const bool low = FOUR && (threadIdx.x & 16) != 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        qb[i][0] = word(2 * i);
        qb[i][1] = word(2 * i + 1);
        const uint32_t b = word(32 + i);
        const uint32_t l0 = pack_half2((float)(b & 0xffu) * step, (float)((b >> 8) & 0xffu) * step);
        const uint32_t l1 = pack_half2((float)((b >> 16) & 0xffu) * step, (float)(b >> 24) * step);
        if (FOUR) {
            qb[i][0] = low ? l0 : qb[i][0];
            qb[i][1] = low ? l1 : qb[i][1];
        } else {
            ql[FOUR ? 0 : i][0] = l0;
            ql[FOUR ? 0 : i][1] = l1;
        }
    }
}

// The un-normalised output of one work item, [8 rows][256] in natural column order, into this warp's idle ring.
// FOUR: columns 4-7 hold the products of the weights' residuals; their sum with columns 0-3 is rows 0-3.
template <bool FOUR>
__device__ __forceinline__ void x_stage_output(const XWarp& x, float* stage_o, float (&o)[16][4]) {
    const int gid = x.gid, tig = x.tig;
    if (FOUR) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
#pragma unroll
            for (int c = 0; c < 4; ++c) o[i][c] += __shfl_xor_sync(0xffffffffu, o[i][c], 2);
        }
        if (tig >= 2) return;      // rows 4-7 do not exist (their mass is 0)
    }
#pragma unroll
    for (int i4 = 0; i4 < 4; ++i4) {
        const int half = i4 >> 1, vw = 4 * (gid >> 1) + (gid & 1) + 2 * (i4 & 1);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int ca = vword_col(half, vw, 2 * t), cb = vword_col(half, vw, 2 * t + 1);
            stage_o[(2 * tig) * kHeadDim + ca] = o[4 * i4 + t][0];
            stage_o[(2 * tig + 1) * kHeadDim + ca] = o[4 * i4 + t][1];
            stage_o[(2 * tig) * kHeadDim + cb] = o[4 * i4 + t][2];
            stage_o[(2 * tig + 1) * kHeadDim + cb] = o[4 * i4 + t][3];
        }
    }
}

// Streams units [pg0, pg0 + n_here) of one work item.  `load_query(qb, ql)` runs once, after the first copies are on their way.
// Leaves the accumulators, running maxima and row masses of this lane's rows (2 tig, 2 tig + 1); x.failed when a wait gave up.
template <bool SPARSE, bool FOUR, class LoadQuery>
__device__ __forceinline__ void x_stream(const StreamParams& p, XWarp& x, int r, const ReqGeom& g, int kv_head, int group, int pg0,
                                         int n_here, LoadQuery load_query, float (&o)[16][4], float (&m_run)[2], float (&l_row)[2]) {
    const int lane = x.lane, gid = x.gid, tig = x.tig, key_a = x.key_a, kv0 = x.kv0;
    const uint32_t ring = x.ring, bars = x.bars, lut_lane = x.lut_lane, lutk_lane = x.lutk_lane, vwb = x.vwb;
    const int rows_in_req = g.q_len * p.gqa;
#define W34_LDS(addr) lds32_dep(addr, ptok)
#define W34_LUT(word, k) lds32_lut(__byte_perm((word), lut_lane, 0x7604 + ((k) << 4)))
#define W34_LUTK(word, k) lds64_lut(__byte_perm((word), lutk_lane, 0x7604 + ((k) << 4)))
#define W34_LUTR(word, k) lds32_lut_residual(__byte_perm((word), lutk_lane, 0x7604 + ((k) << 4)))
    // ---- page pipeline ---------------------------------------------------------------
    const int32_t* blocks = p.batch.block_tables + (size_t)r * p.batch.max_blocks_per_req;
    const uint8_t* k_head_base = (const uint8_t*)(uintptr_t)p.layout.k_base + (size_t)kv_head * p.layout.k_head_stride_bytes;
    const uint8_t* v_head_base = (const uint8_t*)(uintptr_t)p.layout.v_base + (size_t)kv_head * p.layout.v_head_stride_bytes;
    auto page_of = [&](int idx) { return (idx < n_here) ? block_table_page(blocks, pg0 + idx, p.batch.max_blocks_per_req, kInStream) : 0; };
    int32_t my_page = 0, next_page = 0;     // page ids of units [64 c, 64 c + 32) and [64 c + 32, 64 c + 64)
    if (!SPARSE) {
        my_page = page_of(lane);
        next_page = page_of(32 + lane);
    }
    // query-sparse: the token's selected list and its length
    const int32_t* sel_phys = SPARSE ? p.sel_phys + (size_t)r * p.select_k : nullptr;
    const int32_t* sel_logical = SPARSE ? p.sel_logical + (size_t)r * p.select_k : nullptr;
    const int n_sel = SPARSE ? min(p.num_selected[r], p.select_k) : 0;
    fence_proxy_async();  // generic-proxy writes to the ring precede the copies
    const bool copies_v = (lane & 2) != 0;
    const uint8_t* lane_base = (copies_v ? v_head_base : k_head_base) + (lane & 1) * kHalfBytes;
    const uint64_t lane_page_stride = copies_v ? p.layout.v_page_stride_bytes : p.layout.k_page_stride_bytes;
    const uint32_t lane_dst = (uint32_t)((lane >> 2) & 1) * kStageStride + (copies_v ? (uint32_t)kRunStride : 0u) + (uint32_t)(lane & 1) * kHalfStride;
    auto issue = [&](int st) {  // units 2 st and 2 st + 1 into slot st & 1; called by all lanes
        const uint32_t bar = bars + 8u * (uint32_t)(st & 1), dst = ring + (uint32_t)(st & 1) * kXSlot;
        const int n = min(2, n_here - 2 * st);
        x.pending |= 1u << (st & 1);
        if (SPARSE) {
            // A unit is four entries of the list.  Lane j < 8 takes entry j: a group of four rows (528 bytes of K, 528 of
            // V) lands at rows 4 (j & 3) .. of stage j >> 2; a skipped entry (negative id, past the list's end, or wholly
            // after the token's position) copies nothing and is masked through the position word left in the padding.
            const int gi = 4 * (pg0 + 2 * st) + lane;
            int ph = -1, first_pos = 0x3fffffff;
            if (lane < 4 * n && gi < n_sel) {
                ph = sel_phys[gi];
                const int lg = sel_logical[gi];
                if (ph >= 0 && 4 * lg <= g.ctx_before) first_pos = 4 * lg; else ph = -1;
            }
            const int n_valid = __popc(__ballot_sync(0xffffffffu, ph >= 0));
            if (lane == 0) mbar_expect_tx(bar, (uint32_t)n_valid * 8u * kTq4RowBytes);
            __syncwarp();
            if (lane < 8) {
                const uint32_t stage = dst + (uint32_t)(lane >> 2) * kStageStride;
                sts32(stage + kHalfBytes + 4u * (lane & 3), (uint32_t)first_pos);
                if (ph >= 0) {
                    const int page = pool_page(ph >> 2, kInStream);
                    const uint32_t row_off = (uint32_t)(ph & 3) * 4u * kTq4RowBytes;
                    bulk_g2s(stage + token_offset(4 * (lane & 3)), k_head_base + (size_t)page * p.layout.k_page_stride_bytes + row_off,
                             4u * kTq4RowBytes, bar);
                    bulk_g2s(stage + kRunStride + token_offset(4 * (lane & 3)),
                             v_head_base + (size_t)page * p.layout.v_page_stride_bytes + row_off, 4u * kTq4RowBytes, bar);
                }
            }
            return;
        }
        // lanes 0-7: page lane >> 2, K or V run (lane >> 1) & 1, 8-row half lane & 1
        const int32_t page = __shfl_sync(0xffffffffu, (2 * st & 32) ? next_page : my_page, (2 * st + (lane >> 2)) & 31);
        if (lane == 0) mbar_expect_tx(bar, (uint32_t)n * 4u * kHalfBytes);
        __syncwarp();
        if (lane < 4 * n) {
            const uint8_t* src = lane_base + (size_t)page * lane_page_stride;
            bulk_g2s(dst + lane_dst, src, kHalfBytes, bar);
        }
    };
    if (n_here > 0) issue(0);

    // limits of this lane's two query rows (2 tig, 2 tig + 1)
    int rmax[2], rmin[2];
    bool rvalid[2];
#pragma unroll
    for (int y = 0; y < 2; ++y) {
        const int row = group * kRowsPerGroup + 2 * (FOUR ? tig & 1 : tig) + y;
        const int q_off = row / p.gqa;
        rvalid[y] = row < rows_in_req &&
                    (p.batch.valid_token_mask == nullptr || p.batch.valid_token_mask[g.q_start + q_off] != 0);
        rmax[y] = rvalid[y] ? row_max_kv(p.batch, g, q_off) : -1;
        rmin[y] = rvalid[y] ? row_min_kv(p.batch, g, q_off) : 0x7fffffff;
    }
    // keys in [safe_lo, safe_hi] are visible to every valid row of the group
    int safe_hi = min(rvalid[0] ? rmax[0] : 0x7fffffff, rvalid[1] ? rmax[1] : 0x7fffffff);
    int safe_lo = max(rvalid[0] ? rmin[0] : 0, rvalid[1] ? rmin[1] : 0);
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
        safe_hi = min(safe_hi, __shfl_xor_sync(0xffffffffu, safe_hi, d));
        safe_lo = max(safe_lo, __shfl_xor_sync(0xffffffffu, safe_lo, d));
    }
    uint32_t qb[16][2], ql[FOUR ? 1 : 16][2];
    load_query(qb, ql);
#pragma unroll
    for (int i = 0; i < 16; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f; }
    m_run[0] = m_run[1] = -1e30f;
    // row mass: complete up to the last reduction, and this lane's share since then
    float l_tot[2] = {0.0f, 0.0f}, l_part[2] = {0.0f, 0.0f};

#pragma unroll 1
    for (int st = 0; 2 * st < n_here; ++st) {
        // refill page-id registers every 32 units, one window ahead
        if (!SPARSE && (st & 15) == 0 && st > 0) {
            const int32_t fresh = page_of(2 * st + 32 + lane);
            if (st & 16) my_page = fresh; else next_page = fresh;
        }
        if (2 * (st + 1) < n_here) issue(st + 1);
        const uint32_t sb = (uint32_t)(st & 1);
        if (!mbar_wait(bars + 8u * sb, (x.phase_bits >> sb) & 1u)) { x.failed = true; break; }
        x.phase_bits ^= 1u << sb;
        x.pending &= ~(1u << sb);
        if (SPARSE) __syncwarp();   // the position words written by lanes 0-7 are read by all lanes
        const uint32_t slot_base = ring + sb * kXSlot;
        // A step whose second page does not exist computes on whatever that stage holds, all of it masked.
        const bool two = 2 * st + 1 < n_here;
        const uint32_t ptok = page_token(st);
        float pr[2][4];     // scores, then weights: [page][token key_a rows 2 tig, 2 tig + 1; token key_a + 4 likewise]
        bool full[2];
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const uint32_t kst = slot_base + (uint32_t)y * kStageStride;
            // per 128-half, two fragments (tokens key_a, key_a + 4), value and residual rows in each
            float sh[2][2][4];
            float sl[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};      // eight rows: per half, values by the query's residuals
            const uint32_t krow_a = kst + token_offset(key_a);
            const uint32_t krow_b = krow_a + 4u * kTq4RowBytes;
            const uint32_t ka0 = W34_LDS(krow_a), ka16 = W34_LDS(krow_a + 64);
            const uint32_t kb0 = W34_LDS(krow_b), kb16 = W34_LDS(krow_b + 64);
#pragma unroll
            for (int t8 = 0; t8 < 8; ++t8) {     // halves alternate: four independent accumulator chains
                const int half = t8 & 1, s8 = 4 * half + (t8 >> 1);
                const uint32_t off = 4u * ((half ? 17u : 0u) + 4u * tig + (s8 & 3));
                uint32_t wa = W34_LDS(krow_a + off), wb = W34_LDS(krow_b + off);
                if (s8 == 0 && tig == 0) {     // virtual word 0 of half 0: splice (W0 >> 16) | (W16 << 16)
                    wa = (ka0 >> 16) | (ka16 << 16);
                    wb = (kb0 >> 16) | (kb16 << 16);
                }
#pragma unroll
                for (int hk = 0; hk < 2; ++hk) {
                    const int ks = 2 * s8 + hk;
                    const uint2 a0 = W34_LUTK(wa, 2 * hk), a1 = W34_LUTK(wa, 2 * hk + 1);
                    const uint2 b0 = W34_LUTK(wb, 2 * hk), b1 = W34_LUTK(wb, 2 * hk + 1);
                    if ((s8 & 3) == 0 && hk == 0) {
                        mma16816_zero(sh[half][0], a0.x, a0.y, a1.x, a1.y, qb[ks][0], qb[ks][1]);
                        mma16816_zero(sh[half][1], b0.x, b0.y, b1.x, b1.y, qb[ks][0], qb[ks][1]);
                    } else {
                        mma16816(sh[half][0], a0.x, a0.y, a1.x, a1.y, qb[ks][0], qb[ks][1]);
                        mma16816(sh[half][1], b0.x, b0.y, b1.x, b1.y, qb[ks][0], qb[ks][1]);
                    }
                    if (!FOUR) {      // the query's residuals by the values of both tokens
                        if ((s8 & 3) == 0 && hk == 0) mma16816_zero(sl[half], a0.x, b0.x, a1.x, b1.x, ql[FOUR ? 0 : ks][0], ql[FOUR ? 0 : ks][1]);
                        else mma16816(sl[half], a0.x, b0.x, a1.x, b1.x, ql[FOUR ? 0 : ks][0], ql[FOUR ? 0 : ks][1]);
                    }
                }
            }
            const float dka0 = __half2float(__ushort_as_half((unsigned short)(ka0 & 0xffffu)));
            const float dkb0 = __half2float(__ushort_as_half((unsigned short)(kb0 & 0xffffu)));
            const float dka1 = __half2float(__ushort_as_half((unsigned short)(ka16 >> 16)));
            const float dkb1 = __half2float(__ushort_as_half((unsigned short)(kb16 >> 16)));
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                pr[y][c] = dka0 * (sh[0][0][c] + sh[0][0][c + 2] * (1.0f / kResidualScale) + sl[0][c]) +
                           dka1 * (sh[1][0][c] + sh[1][0][c + 2] * (1.0f / kResidualScale) + sl[1][c]);
                pr[y][2 + c] = dkb0 * (sh[0][1][c] + sh[0][1][c + 2] * (1.0f / kResidualScale) + sl[0][2 + c]) +
                               dkb1 * (sh[1][1][c] + sh[1][1][c + 2] * (1.0f / kResidualScale) + sl[1][2 + c]);
            }
            if (FOUR) {      // value and residual of the query
#pragma unroll
                for (int c = 0; c < 4; ++c) pr[y][c] += __shfl_xor_sync(0xffffffffu, pr[y][c], 2);
            }
            const int kv_base = (pg0 + 2 * st + y) << 4;
            int pos_a = kv_base + key_a, pos_b = pos_a + 4;
            if (SPARSE) {     // position of the first row of the two groups this lane's keys sit in
                const uint32_t pw = kst + kHalfBytes;
                const int f0 = (int)W34_LDS(pw), f1 = (int)W34_LDS(pw + 4), f2 = (int)W34_LDS(pw + 8), f3 = (int)W34_LDS(pw + 12);
                full[y] = max(max(f0, f1), max(f2, f3)) + 3 <= safe_hi;
                pos_a = ((key_a >> 3) ? f2 : f0) + (key_a & 3);
                pos_b = ((key_a >> 3) ? f3 : f1) + (key_a & 3);
            } else {
                full[y] = (kv_base >= safe_lo) && (kv_base + 15 <= safe_hi);
            }
            if (y == 1 && !two) { full[y] = false; pos_a = pos_b = 0x3fffffff; }
            if (!full[y]) {
                if (!(pos_a >= rmin[0] && pos_a <= rmax[0])) pr[y][0] = -1e30f;
                if (!(pos_a >= rmin[1] && pos_a <= rmax[1])) pr[y][1] = -1e30f;
                if (!(pos_b >= rmin[0] && pos_b <= rmax[0])) pr[y][2] = -1e30f;
                if (!(pos_b >= rmin[1] && pos_b <= rmax[1])) pr[y][3] = -1e30f;
            }
        }
        // ---- online softmax over the 32 keys, per query row -----------------------------
        float mx0 = fmaxf(fmaxf(pr[0][0], pr[0][2]), fmaxf(pr[1][0], pr[1][2]));
        float mx1 = fmaxf(fmaxf(pr[0][1], pr[0][3]), fmaxf(pr[1][1], pr[1][3]));
#pragma unroll
        for (int d = 4; d < 32; d <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, d));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, d));
        }
        const float mn0 = fmaxf(m_run[0], mx0), mn1 = fmaxf(m_run[1], mx1);
        if (__any_sync(0xffffffffu, mn0 > m_run[0] || mn1 > m_run[1])) {
            const float al0 = ex2(m_run[0] - mn0), al1 = ex2(m_run[1] - mn1);
            l_tot[0] *= al0;
            l_tot[1] *= al1;
            l_part[0] *= al0;
            l_part[1] *= al1;
#pragma unroll
            for (int t = 0; t < 16; ++t) { o[t][0] *= al0; o[t][1] *= al1; o[t][2] *= al0; o[t][3] *= al1; }
            m_run[0] = mn0;
            m_run[1] = mn1;
        }
        float top[2][2];     // largest weight of a page, per row
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            float w[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) w[c] = ex2(pr[y][c] - ((c & 1) ? mn1 : mn0));
            if (!full[y]) {     // a row that has seen nothing yet: its masked scores equal its maximum
#pragma unroll
                for (int c = 0; c < 4; ++c) if (pr[y][c] <= -1e30f) w[c] = 0.0f;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) pr[y][c] = w[c];
            top[y][0] = fmaxf(w[0], w[2]);
            top[y][1] = fmaxf(w[1], w[3]);
        }
        l_part[0] += ((pr[0][0] + pr[0][2]) + (pr[1][0] + pr[1][2]));
        l_part[1] += ((pr[0][1] + pr[0][3]) + (pr[1][1] + pr[1][3]));
        if (st < 2 || (st & 1)) {
#pragma unroll
            for (int d = 4; d < 32; d <<= 1) {
                l_part[0] += __shfl_xor_sync(0xffffffffu, l_part[0], d);
                l_part[1] += __shfl_xor_sync(0xffffffffu, l_part[1], d);
            }
            l_tot[0] += l_part[0];
            l_tot[1] += l_part[1];
            l_part[0] = l_part[1] = 0.0f;
        }
        // A page is peaked when a key holds more than kPeakedWeight of a row's mass so far; the mass known here
        // is a lower bound of it.  (Rows that do not exist score 0 and must not count.)
        const float cut0 = kPeakedWeight * (l_tot[0] + l_part[0]), cut1 = kPeakedWeight * (l_tot[1] + l_part[1]);
        const bool pk0 = (rvalid[0] && top[0][0] > cut0) || (rvalid[1] && top[0][1] > cut1);
        const bool pk1 = (rvalid[0] && top[1][0] > cut0) || (rvalid[1] && top[1][1] > cut1);
        const uint32_t both = (uint32_t)__any_sync(0xffffffffu, pk0) | ((uint32_t)__any_sync(0xffffffffu, pk1) << 1);
        // P x d_v per 128-half, laid out as B fragments (k = key, n = query row).  A key no row can see may hold
        // never-written bytes: its scale must not meet a zero weight.
        auto weighted = [&](int y, float (&pd)[2][4]) {
            const uint32_t vrow_a = slot_base + (uint32_t)y * kStageStride + kRunStride + token_offset(key_a);
            const uint32_t va0 = W34_LDS(vrow_a), va16 = W34_LDS(vrow_a + 64);
            const uint32_t vb0 = W34_LDS(vrow_a + 4u * kTq4RowBytes), vb16 = W34_LDS(vrow_a + 4u * kTq4RowBytes + 64);
            const bool za = pr[y][0] == 0.0f && pr[y][1] == 0.0f, zb = pr[y][2] == 0.0f && pr[y][3] == 0.0f;
            const float da0 = za ? 0.0f : __half2float(__ushort_as_half((unsigned short)(va0 & 0xffffu)));
            const float da1 = za ? 0.0f : __half2float(__ushort_as_half((unsigned short)(va16 >> 16)));
            const float db0 = zb ? 0.0f : __half2float(__ushort_as_half((unsigned short)(vb0 & 0xffffu)));
            const float db1 = zb ? 0.0f : __half2float(__ushort_as_half((unsigned short)(vb16 >> 16)));
            pd[0][0] = pr[y][0] * da0; pd[0][1] = pr[y][1] * da0; pd[0][2] = pr[y][2] * db0; pd[0][3] = pr[y][3] * db0;
            pd[1][0] = pr[y][0] * da1; pd[1][1] = pr[y][1] * da1; pd[1][2] = pr[y][2] * db1; pd[1][3] = pr[y][3] * db1;
        };
        // code bytes of step i4: byte t of ab[0] -> (V[ka][e = 2 t], V[kb][e = 2 t]), of ab[1] -> e = 2 t + 1
        auto code_pairs = [&](uint32_t vr, int i4, uint32_t (&ab)[2], uint32_t (&cd)[2]) {
            const uint32_t off = 4u * (((i4 >> 1) ? 17u : 0u) + vwb + 2u * (i4 & 1));
            uint32_t w[4] = {W34_LDS(vr + off), W34_LDS(vr + kTq4RowBytes + off), W34_LDS(vr + 4u * kTq4RowBytes + off),
                             W34_LDS(vr + 5u * kTq4RowBytes + off)};
            if (i4 == 0 && gid == 0) {  // virtual word 0 of half 0
                w[0] = (w[0] >> 16) | (W34_LDS(vr + 64) << 16);
                w[1] = (w[1] >> 16) | (W34_LDS(vr + kTq4RowBytes + 64) << 16);
                w[2] = (w[2] >> 16) | (W34_LDS(vr + 4u * kTq4RowBytes + 64) << 16);
                w[3] = (w[3] >> 16) | (W34_LDS(vr + 5u * kTq4RowBytes + 64) << 16);
            }
            ab[0] = (w[0] & 0x0f0f0f0fu) | ((w[1] << 4) & 0xf0f0f0f0u);
            ab[1] = ((w[0] >> 4) & 0x0f0f0f0fu) | (w[1] & 0xf0f0f0f0u);
            cd[0] = (w[2] & 0x0f0f0f0fu) | ((w[3] << 4) & 0xf0f0f0f0u);
            cd[1] = ((w[2] >> 4) & 0x0f0f0f0fu) | (w[3] & 0xf0f0f0f0u);
        };
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            float pd[2][4];
            weighted(y, pd);
            uint32_t pb[2][2], pl[2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const __half2 hi = __floats2half2_rn(pd[h][2 * z], pd[h][2 * z + 1]);
                    const float2 hf = __half22float2(hi);
                    const __half2 lo = __floats2half2_rn(pd[h][2 * z] - hf.x, pd[h][2 * z + 1] - hf.y);
                    if (FOUR) {
                        pb[h][z] = movmatrix_trans(tig < 2 ? *reinterpret_cast<const uint32_t*>(&hi) : *reinterpret_cast<const uint32_t*>(&lo));
                    } else {
                        pb[h][z] = movmatrix_trans(*reinterpret_cast<const uint32_t*>(&hi));
                        pl[h][z] = movmatrix_trans(*reinterpret_cast<const uint32_t*>(&lo));
                    }
                }
            }
            // ---- O^T += V^T P^T.  Step i4: half i4 >> 1, virtual word 4 (gid >> 1) + (gid & 1) + 2 (i4 & 1) -----
            const uint32_t vr = slot_base + (uint32_t)y * kStageStride + kRunStride + token_offset(kv0);
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) {
                uint32_t ab[2], cd[2];
                code_pairs(vr, i4, ab, cd);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const uint32_t a0 = W34_LUT(ab[0], t), a1 = W34_LUT(ab[1], t), a2 = W34_LUT(cd[0], t), a3 = W34_LUT(cd[1], t);
                    mma16816(o[4 * i4 + t], a0, a1, a2, a3, pb[i4 >> 1][0], pb[i4 >> 1][1]);
                    if (!FOUR) mma16816(o[4 * i4 + t], a0, a1, a2, a3, pl[i4 >> 1][0], pl[i4 >> 1][1]);
                }
            }
        }
        // A peaked page adds V_residual (P d_v): a branch of its own, so that the common pass stays one basic block.
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            if (((both >> y) & 1u) == 0u) continue;
            const uint32_t vr = slot_base + (uint32_t)y * kStageStride + kRunStride + token_offset(kv0);
            float pd[2][4];
            weighted(y, pd);
            uint32_t ps[2][2];      // P d_v / kResidualScale, the partner of the scaled centroid residuals
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const __half2 s2 = __floats2half2_rn(pd[h][2 * z] * (1.0f / kResidualScale), pd[h][2 * z + 1] * (1.0f / kResidualScale));
                    ps[h][z] = movmatrix_trans(FOUR && tig >= 2 ? 0u : *reinterpret_cast<const uint32_t*>(&s2));
                }
            }
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) {
                uint32_t ab[2], cd[2];
                code_pairs(vr, i4, ab, cd);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    mma16816(o[4 * i4 + t], W34_LUTR(ab[0], t), W34_LUTR(ab[1], t), W34_LUTR(cd[0], t), W34_LUTR(cd[1], t),
                             ps[i4 >> 1][0], ps[i4 >> 1][1]);
                }
            }
        }
        __syncwarp();  // every lane is done with this slot before it is refilled
    }
#pragma unroll
    for (int d = 4; d < 32; d <<= 1) {
        l_part[0] += __shfl_xor_sync(0xffffffffu, l_part[0], d);
        l_part[1] += __shfl_xor_sync(0xffffffffu, l_part[1], d);
    }
    l_row[0] = l_tot[0] + l_part[0];
    l_row[1] = l_tot[1] + l_part[1];
#undef W34_LDS
#undef W34_LUT
#undef W34_LUTK
#undef W34_LUTR
}

// wait, bounded, for copies already issued so the CTA does not exit under them
__device__ __forceinline__ void x_drain(XWarp& x) {
    for (int s = 0; s < 2; ++s) {
        if (x.pending & (1u << s)) (void)mbar_wait(x.bars + 8u * s, (x.phase_bits >> s) & 1u);
    }
}

// What the workers of a CTA leave for each other at the end.
struct XHeld {
    float m[kExactWarps][kRowsPerGroup], l[kExactWarps][kRowsPerGroup];
    int item[kExactWarps];
    uint32_t ring[kExactWarps];
};

// One worker's share: units [u, u_end) of the step's list.  Writes the partial of every item but, where neighbours are merged, the last,
// which stays in the worker's ring: returns it (its place among the slots, less the worker's), or -1.
// FOUR: items of at most four query rows.  The N = 8 columns of an MMA hold their values and, beside them, their rounding residuals (of the
// query for the scores, of the weights for the output), so that one MMA does what takes two with eight rows: 48 a page instead of 80,
// with the tensor pipe at 45 % and its issue among the stalls.
template <bool SPARSE, bool FOUR>
__device__ __forceinline__ int x_share(const StreamParams& p, XWarp& x, PlanHeader* hdr, int u, int u_end, int w_global, bool neighbours,
                                       float* ring_gen, XHeld& held_by) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int R = p.batch.num_reqs;
    const int32_t* unit_prefix = plan_array(p.scratch, 0, R);
    const int32_t* item_prefix = plan_array(p.scratch, 1, R);
    const int32_t* page_lo_a = plan_array(p.scratch, 2, R);
    const int32_t* npages_a = plan_array(p.scratch, 3, R);
    const int32_t* ngroups_a = plan_array(p.scratch, 4, R);
    float* partials = reinterpret_cast<float*>(p.scratch + plan_bytes(R));

    int r = u < u_end ? last_not_above(unit_prefix, R, u) : 0;
    int held = -1;      // item whose state this warp still holds when its share is done
#pragma unroll 1
    while (u < u_end) {
        while (unit_prefix[r + 1] <= u) ++r;  // skips requests without units
        const int npages = npages_a[r];
        const int ngroups = ngroups_a[r];
        const int in_req = u - unit_prefix[r];
        const int item = in_req / npages;
        const int page_in_item = in_req - item * npages;
        const int n_here = min(u_end - u, npages - page_in_item);
        const int kv_head = item / ngroups;
        const int group = item - kv_head * ngroups;
        const int pg0 = page_lo_a[r] + page_in_item;   // first logical page (sparse: first unit of four entries)
        const int slot = w_global + item_prefix[r] + item;
        const ReqGeom g = stream_req(p, r);
        float o[16][4], m_run[2], l_row[2];
        const uint32_t* qf = p.qfrag + ((size_t)(r * p.layout.local_kv_heads + kv_head) * p.q_groups_max + group) * (kQFragWords * 32) + (FOUR ? lane & 15 : lane);
        x_stream<SPARSE, FOUR>(p, x, r, g, kv_head, group, pg0, n_here,
                         // (not __ldg: the plan kernel was still writing these words when this one started)
                         [&](uint32_t (&qb)[16][2], uint32_t (&ql)[FOUR ? 1 : 16][2]) { x_load_query<FOUR>([&](int i) { return qf[i * 32]; }, qb, ql); },
                         o, m_run, l_row);
        if (x.failed) {
            x_drain(x);
            if (lane == 0) atomicOr(&hdr->status, 1);
            break;
        }
        x_stage_output<FOUR>(x, ring_gen, o);
        if (FOUR && x.tig >= 2) {
            m_run[0] = m_run[1] = -1e30f;
            l_row[0] = l_row[1] = 0.0f;
        }
        u += n_here;
        if (u >= u_end && neighbours) {      // the last segment: merged with the neighbours' below
            held = slot - w_global;
            if (x.gid == 0) {
                held_by.m[wid][2 * x.tig] = m_run[0];
                held_by.m[wid][2 * x.tig + 1] = m_run[1];
                held_by.l[wid][2 * x.tig] = l_row[0];
                held_by.l[wid][2 * x.tig + 1] = l_row[1];
            }
            break;
        }
        // ---- write the partial ----------------------------------------------------------------
        __syncwarp();
        if (slot < p.max_slots) {
            const float4* src4 = reinterpret_cast<const float4*>(ring_gen);
            float4* dst4 = reinterpret_cast<float4*>(partials + (size_t)slot * kPartialFloats);
#pragma unroll
            for (int k = 0; k < (kRowsPerGroup * kHeadDim / 4) / 32; ++k) dst4[k * 32 + lane] = src4[k * 32 + lane];
            if (x.gid == 0) {
                float* ml = partials + (size_t)slot * kPartialFloats + kRowsPerGroup * kHeadDim;
                ml[2 * x.tig] = m_run[0];
                ml[2 * x.tig + 1] = m_run[1];
                ml[kRowsPerGroup + 2 * x.tig] = l_row[0];
                ml[kRowsPerGroup + 2 * x.tig + 1] = l_row[1];
            }
        }
        __syncwarp();
    }
    return held;
}

// Rows per item: eight, four, or four where the plan found that no request has more (kRowsByPlan: a batch that declares up to four, but a
// request may hold more than its batch declares, and an item of eight still takes all of its rows then).
enum ItemRows { kEightRows, kFourRows, kRowsByPlan };
template <bool SPARSE, ItemRows ROWS>
__global__ void __launch_bounds__(kXThreads, 1) tq4_attention_stream_exact_kernel(const StreamParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // The lookup table sits at the first 64 KB-aligned SHARED address inside the dynamic window, so that
    // (table address | code byte << 8 | lane offset) is one PRMT.  Warp rings fill the space below and above it; the
    // mbarriers follow the last ring.
    const uint32_t win_lo = smem_u32(smem);
    const uint32_t win_hi = win_lo + p.smem_bytes;
    const uint32_t lut_addr = (win_lo + 0xffffu) & ~0xffffu;
    constexpr uint32_t kRingBytes = 2u * kXSlot;
    const uint32_t warps_below = (lut_addr - win_lo) / kRingBytes;
    const uint32_t ring = ((uint32_t)wid < warps_below) ? (win_lo + (uint32_t)wid * kRingBytes)
                                                         : (lut_addr + kLutBytes + ((uint32_t)wid - warps_below) * kRingBytes);
    const uint32_t above = (uint32_t)kExactWarps > warps_below ? (uint32_t)kExactWarps - warps_below : 0u;
    const uint32_t bars_base = lut_addr + kLutBytes + above * kRingBytes;
    const uint32_t bars = bars_base + (uint32_t)wid * 16u;
    PlanHeader* hdr = reinterpret_cast<PlanHeader*>(p.scratch);
    if (lut_addr + kLutBytes > win_hi || bars_base + (uint32_t)kExactWarps * 16u + (uint32_t)sizeof(XHeld) > win_hi) {
        grid_dependency_wait();
        if (threadIdx.x == 0) atomicOr(&hdr->status, 2);  // shared-memory window cannot hold the layout
        return;
    }
    XHeld& held_by = *reinterpret_cast<XHeld*>(smem + (bars_base + (uint32_t)kExactWarps * 16u - win_lo));
    float* ring_gen = reinterpret_cast<float*>(smem + (ring - win_lo));

    XWarp x;
    x_init(x, lut_addr, ring, bars);
    x_build_tables(lut_addr);
    grid_dependency_wait();      // nothing above touches global memory
    grid_launch_dependents();
    __syncthreads();

    const int R = p.batch.num_reqs;
    const int per = hdr->units_per_warp;
    const int total_units = hdr->total_units;
    // A step with work for every worker: the eight workers of a CTA take neighbouring shares, so that what they hold of one
    // item can be merged before it is written.  A smaller one: consecutive shares sit on different SMs.
    const bool neighbours = per > kMinUnitsPerWarp;
    const int w_global = neighbours ? (int)blockIdx.x * kExactWarps + wid : wid * (int)gridDim.x + (int)blockIdx.x;
    const long long u_ll = (long long)w_global * per;
    const int u = (int)min(u_ll, (long long)total_units);
    const int u_end = min(u + per, total_units);
    int held;
    if constexpr (ROWS == kRowsByPlan) {
        held = plan_array(p.scratch, 2, R)[R] == 0 ? x_share<SPARSE, true>(p, x, hdr, u, u_end, w_global, neighbours, ring_gen, held_by)
                                                   : x_share<SPARSE, false>(p, x, hdr, u, u_end, w_global, neighbours, ring_gen, held_by);
    } else {
        held = x_share<SPARSE, ROWS == kFourRows>(p, x, hdr, u, u_end, w_global, neighbours, ring_gen, held_by);
    }
    if (!neighbours) return;
    float* partials = reinterpret_cast<float*>(p.scratch + plan_bytes(R));

    // ---- merge what the CTA's workers hold of one item: warp w does row w of every run of workers with the same item, the
    //      run's first slot takes the result, the others are left empty (l = 0) ------------------------------------
    if (lane == 0) {
        held_by.item[wid] = held;
        held_by.ring[wid] = ring - win_lo;
    }
    __syncthreads();
    for (int first = 0; first < kExactWarps;) {
        const int item = held_by.item[first];
        int end = first + 1;
        while (end < kExactWarps && held_by.item[end] == item) ++end;
        const int slot = (int)blockIdx.x * kExactWarps + first + item;
        if (item >= 0 && slot + (end - first) <= p.max_slots) {
            float m_tot = -1e30f, l_tot = 0.0f, v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int w = first; w < end; ++w) if (held_by.l[w][wid] > 0.0f) m_tot = fmaxf(m_tot, held_by.m[w][wid]);
            for (int w = first; w < end; ++w) {
                const float l = held_by.l[w][wid], wgt = l > 0.0f ? ex2(held_by.m[w][wid] - m_tot) : 0.0f;
                l_tot += l * wgt;
                const float4* src = reinterpret_cast<const float4*>(smem + held_by.ring[w] + (wid * kHeadDim + 8 * lane) * 4);
                const float4 a = src[0], b = src[1];
                v[0] += wgt * a.x; v[1] += wgt * a.y; v[2] += wgt * a.z; v[3] += wgt * a.w;
                v[4] += wgt * b.x; v[5] += wgt * b.y; v[6] += wgt * b.z; v[7] += wgt * b.w;
            }
            float* dst = partials + (size_t)slot * kPartialFloats;
            float4* dst4 = reinterpret_cast<float4*>(dst + wid * kHeadDim + 8 * lane);
            dst4[0] = make_float4(v[0], v[1], v[2], v[3]);
            dst4[1] = make_float4(v[4], v[5], v[6], v[7]);
            if (lane < end - first) {
                float* ml = dst + (size_t)lane * kPartialFloats + kRowsPerGroup * kHeadDim + wid;
                ml[0] = lane == 0 ? m_tot : -1e30f;
                ml[kRowsPerGroup] = lane == 0 ? l_tot : 0.0f;
            }
        }
        first = end;
    }
}

}  // namespace w34
