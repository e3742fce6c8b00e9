// Decode and verify attention over TQ4 pages on the 5th-generation tensor cores, with value + residual operands.  Included by
// tq4_attention.cu (shares the plan, the table, the PTX wrappers and the merge with the other streaming kernels).
//
// One CTA per SM is one worker: it takes an equal contiguous share of the step's (request, kv head, group of R query rows,
// page) units and walks it in blocks of 128 keys.  The cached keys are the M dimension of both products, so that every code
// is dequantised once for up to 24 query rows, and straight into tensor memory, where it is the MMAs' A operand:
//   S^T[128 keys x 2R]      per 128-half = Khi [Q'hi | Q'lo]^T + Klo [Q'hi | Q'lo]^T        lane = key
//   O^T[128 channels x 2R]  per 128-half += (Vhi + Vlo)^T [(P d_v)hi | (P d_v)lo]^T          lane = channel
// (the centroids' residuals on every block: leaving them out where no key has a large weight takes one more vote of the softmax
// warps a block, then 921 us against 914, and an error several times as large).  Scales stay outside the operands: a thread holds a key's
// scores of both halves and applies its K scales there, and P is multiplied by the V scale of its key and half.
//
//   softmax: four warps per eight rows, thread = key.  P goes to shared memory as the B operand; the running maximum is a
//            reference that moves only when it is exceeded by 2^3, so a block usually needs no reduction over its keys.  P d_v is held
//            times a power of two that moves with it and brings the block's largest V scale to [2^11, 2^12): two fp16 numbers then
//            hold 22 bits of the weights of small V rows as well (without it 7.9 % of the outputs over V of magnitude 2^-10 were not the
//            nearest fp16 value, 4.1 % with three 8-row items of the one-warp kernel)
//   V:       eight warps, thread = fragment position (16x256b stores put channel pairs of four keys in place), half x quadrant;
//            64 keys at a time, values and residuals (one look-up for both) into neighbouring columns of one granule
//   K:       eight warps, thread = key, 32 channels at a time into a ring of four TMEM granules; values and residuals lie next
//            to each other as the table returns them, and the query operand repeats each pair of columns to match
//   one warp copies raw pages and query rows, one issues the score products, one the output products
//
// Measured on 128 requests of 2048 to 16384 keys, four query tokens, 24 / 4 heads (1.26 GB of pages): attention call 800 us against 1458
// with three 8-row items of the one-warp kernel (tq4_stream_exact.cuh), which looks every code up three times.  A block of 128 keys takes
// about 5000 cycles: the V warps' look-ups and stores (3500) and the chain from one block's output product over the next one's weights
// to its own, which share the issue slots.  (With a look-up each for value and residual the V warps were busy for 5700 of 6170
// cycles, and with one barrier for all keys the weights waited for the whole product before: 895 us.)  Taking the weights before the
// vote on the reference (one barrier a block fewer) put them behind the wait for the previous output product: 1008 us.  Weights as
// fragments of four keys by two rows a thread, stored 8 bytes at a time: 830, but 25 us instead of 26.5 on one short request.
#pragma once

namespace w34 {

constexpr int kXtKeys = 128, kXtPages = kXtKeys / kPageTokens;
// four softmax warps per eight rows, 8 V warps, 8 K warps, copies, two MMA warps, one idle
__host__ __device__ constexpr int xt_threads(int rows) { return (rows / 2 + 20) * 32; }
constexpr int kXtStages = 2;                                  // blocks of raw K and V in shared memory
constexpr uint32_t kXtRun = (uint32_t)kXtPages * kTq4PageHeadBytes;       // 16896: K or V of a block
constexpr uint32_t kXtColK = 0, kXtColV = 128, kXtColS = 256, kXtColO = 384;
constexpr int kXtKRing = 4;                                   // granules of 32 channels: a column of values, one of residuals in turn
constexpr float kXtLag = 3.0f;                                // log2 units the reference maximum may lag; P is carried times 2^-3

__host__ __device__ constexpr uint32_t xt_query_bytes(int rows) { return 2u * (uint32_t)rows * 1024u; }

struct XtShared {
    float2 k_scale[2][kXtKeys];
    __align__(16) float m_ref[24], alpha[24], mass[24];
    float red[4][24];                // [warp of the part][row]
    float red_v[4][3];               // [warp of the part][part]
    int row_min[24], row_max[24];
    uint32_t tmem;
    uint32_t aborted;
    uint64_t bars[48];
};
enum { kXtRawKFull = 0, kXtRawKFree = 4, kXtRawVFull = 8, kXtRawVFree = 12, kXtKFull = 16, kXtKEmpty = 20, kXtVFull = 24, kXtVEmpty,
       kXtQFull, kXtQFree, kXtSReady, kXtSFree, kXtPReady, kXtPvDone = kXtPReady + 2, kXtKScale = kXtPvDone + 2,
       kXtDrain = kXtKScale + 2, kXtBarCount };
static_assert(kXtBarCount <= 48, "barrier slots");

__device__ __forceinline__ void tc_ld4(uint32_t (&r)[4], uint32_t taddr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_st4(uint32_t taddr, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
                 :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
// 16 lanes x 256 bits, twice: registers 4 i + {0, 1} go to lane t / 4, columns 8 i + 2 (t % 4) + {0, 1}; 4 i + {2, 3} eight
// lanes further (t: thread of the warp).
__device__ __forceinline__ void tc_st_16x256b_x2(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// D (+)= A B with A in tensor memory, all output lanes.
template <bool ACC>
__device__ __forceinline__ void xt_mma(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 :: "r"(d), "r"(a), "l"(b_desc), "r"(idesc), "n"(ACC ? 1 : 0) : "memory");
}
// Barrier of the four warps of a softmax part.
__device__ __forceinline__ void xt_sync(int part) { asm volatile("bar.sync %0, 128;" :: "r"(1 + part) : "memory"); }
__device__ __forceinline__ bool xt_any(bool x, int part) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((uint32_t)x), "r"(1 + part) : "memory");
    return r != 0;
}

// Query rows of item idx = (request * kv heads + kv head) * q_groups_max + group as the B operand: 2R rows (R values, then R
// residuals) of the 256 rotated columns, every pair of columns twice in a row (K's table entries hold a pair's values and, next to
// them, its residuals, and go to tensor memory as they are): eight blocks of 32 columns, 16-byte chunks swizzled by the row.
// Eight warps.
__device__ void xt_prepare_query(const StreamParams& p, int idx) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, R = p.rows_per_group;
    const int hkv = p.layout.local_kv_heads;
    const int group = idx % p.q_groups_max, kv_head = (idx / p.q_groups_max) % hkv, r = idx / (p.q_groups_max * hkv);
    if (r >= p.batch.num_reqs) return;
    const ReqGeom g = load_req(p.batch, r);
    const int rows_in_req = g.q_len * p.gqa;
    if (!g.valid || group * R >= rows_in_req) return;
    uint8_t* dst = reinterpret_cast<uint8_t*>(p.qfrag) + (size_t)idx * xt_query_bytes(R);
    for (int i = wid; i < R; i += kRowsPerGroup) {
        const int row = group * R + i;
        const int q_off = row / p.gqa, q_head = kv_head * p.gqa + (row - q_off * p.gqa);
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (row < rows_in_req && (p.batch.valid_token_mask == nullptr || p.batch.valid_token_mask[g.q_start + q_off] != 0)) {
            load8(p.q_in, ((size_t)(g.q_start + q_off) * p.num_q_heads + q_head) * kHeadDim, lane, p.io_bf16, v);
            sign8(v, lane);
            butterfly8<5>(v, lane);
        }
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float a = v[2 * k] * (p.q_scale * 0.0625f), b = v[2 * k + 1] * (p.q_scale * 0.0625f);
            const __half2 h = __floats2half2_rn(a, b);
            const float2 hf = __half22float2(h);
            hi[k] = *reinterpret_cast<const uint32_t*>(&h);
            lo[k] = pack_half2(a - hf.x, b - hf.y);
        }
        // (i and i + R share their low three bits: R is a multiple of 8)
        uint8_t* out = dst + (size_t)(lane >> 2) * (2 * R * 128) + (size_t)i * 128;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            uint4* at = reinterpret_cast<uint4*>(out + (((2 * (lane & 3) + k) ^ (i & 7)) << 4));
            at[0] = make_uint4(hi[2 * k], hi[2 * k], hi[2 * k + 1], hi[2 * k + 1]);
            at[R * 8] = make_uint4(lo[2 * k], lo[2 * k], lo[2 * k + 1], lo[2 * k + 1]);
        }
    }
}

// A worker's position in the step's unit list; every role warp advances its own.
struct XtWalk {
    int u, u_end, r;
};
struct XtSegment {
    int r, kv_head, group, pg0, pages, slot;
};
__device__ __forceinline__ bool xt_next(const StreamParams& p, XtWalk& w, XtSegment& s) {
    if (w.u >= w.u_end) return false;
    const int R = p.batch.num_reqs;
    const int32_t* unit_prefix = plan_array(p.scratch, 0, R);
    while (unit_prefix[w.r + 1] <= w.u) ++w.r;  // skips requests without units
    const int npages = plan_array(p.scratch, 3, R)[w.r], ngroups = plan_array(p.scratch, 4, R)[w.r];
    const int in_req = w.u - unit_prefix[w.r];
    const int item = in_req / npages, page = in_req - item * npages;
    s.r = w.r;
    s.kv_head = item / ngroups;
    s.group = item - s.kv_head * ngroups;
    s.pg0 = plan_array(p.scratch, 2, R)[w.r] + page;
    s.pages = min(w.u_end - w.u, npages - page);
    s.slot = (int)blockIdx.x + plan_array(p.scratch, 1, R)[w.r] + item;
    w.u += s.pages;
    return true;
}

template <int R>
__global__ void __launch_bounds__(xt_threads(R), 1) tq4_attention_stream_tc_kernel(const StreamParams p) {
    constexpr int N = 2 * R, STAGES = kXtStages, PARTS = R / 8, W0 = 4 * PARTS;      // W0: first V warp
    constexpr uint32_t kQueryBytes = xt_query_bytes(R), kPBytes = (uint32_t)N * 256u;      // P of one half: [2 x 64 keys][N][128 B]
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t win_lo = smem_u32(smem);
    const uint32_t lut_addr = (win_lo + 0xffffu) & ~0xffffu;
    PlanHeader* hdr = reinterpret_cast<PlanHeader*>(p.scratch);
    SmemCarver carve(win_lo, lut_addr, win_lo + p.smem_bytes);
    const uint32_t q_t = carve.take(kQueryBytes, 1024);
    const uint32_t p_t = carve.take(2u * kPBytes, 1024);
    uint32_t raw[2 * STAGES];
#pragma unroll
    for (int i = 0; i < 2 * STAGES; ++i) raw[i] = carve.take(kXtRun, 128);
    const uint32_t sh_addr = carve.take((uint32_t)sizeof(XtShared), 16);
    if (!carve.ok) {
        grid_dependency_wait();
        if (tid == 0) atomicOr(&hdr->status, 2);  // shared-memory window cannot hold the layout
        return;
    }
    XtShared& sh = *reinterpret_cast<XtShared*>(smem + (sh_addr - win_lo));
    auto raw_k = [&](int s) { return s == 0 ? raw[0] : raw[1]; };
    auto raw_v = [&](int s) { return s == 0 ? raw[2] : raw[3]; };
    const uint32_t bars = smem_u32(sh.bars);
    auto bar = [&](int which) { return bars + 8u * (uint32_t)which; };
    volatile uint32_t* aborted = &sh.aborted;
    // Waits are bounded and warp-uniform, the decision to give up included: a lane that left alone would leave the others in a vote
    // that never completes.  One that gives up ends every loop.
    auto wait_all = [&](uint32_t b, uint32_t parity) {
        if (__all_sync(0xffffffffu, mbar_try_wait(b, parity))) return true;
        const long long t0 = clock64();
        for (;;) {
            if (__all_sync(0xffffffffu, mbar_try_wait(b, parity))) return true;
            if (__any_sync(0xffffffffu, *aborted != 0u || clock64() - t0 >= kWaitCycleLimit)) break;
        }
        *aborted = 1u;
        return false;
    };

    for (int i = tid; i < 256 * 16; i += xt_threads(R)) {      // per byte: {values, residuals} x 16, 256 bytes apart (an address is one byte_perm; 128 are unused)
        const int byte = i >> 4, ln = i & 15;
        const float c0 = kLutScale * tq4_centroid(byte & 15), c1 = kLutScale * tq4_centroid(byte >> 4);
        const uint32_t hi = pack_half2(c0, c1);
        const float2 hf = __half22float2(*reinterpret_cast<const __half2*>(&hi));
        const uint32_t lo = pack_half2(c0 - hf.x, c1 - hf.y);
        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(lut_addr + (uint32_t)(byte * 256 + ln * 8)), "r"(hi), "r"(lo) : "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bar(kXtRawKFull + s), 1u);
            mbar_init(bar(kXtRawKFree + s), 8u);
            mbar_init(bar(kXtRawVFull + s), 1u);
            mbar_init(bar(kXtRawVFree + s), 8u + W0);
        }
        for (int s = 0; s < kXtKRing; ++s) { mbar_init(bar(kXtKFull + s), 4u); mbar_init(bar(kXtKEmpty + s), 1u); }
        for (int s = 0; s < 2; ++s) {
            mbar_init(bar(kXtKScale + s), 4u);
        }
        mbar_init(bar(kXtVFull), 8u);
        mbar_init(bar(kXtVEmpty), 1u);
        mbar_init(bar(kXtQFull), 1u);
        mbar_init(bar(kXtQFree), 1u);
        mbar_init(bar(kXtSReady), 1u);
        mbar_init(bar(kXtSFree), W0);
        for (int kk = 0; kk < 2; ++kk) {      // of each half of the keys
            mbar_init(bar(kXtPReady + kk), W0 / 2);
            mbar_init(bar(kXtPvDone + kk), 1u);
        }
        mbar_init(bar(kXtDrain), 2u);
        sh.aborted = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    grid_dependency_wait();      // nothing above touches global memory
    grid_launch_dependents();

    const int per = hdr->units_per_warp, total_units = hdr->total_units;
    XtWalk walk;
    {
        const long long u0 = (long long)blockIdx.x * per;
        walk.u = (int)min(u0, (long long)total_units);
        walk.u_end = min(walk.u + per, total_units);
    }
    if (walk.u >= walk.u_end) return;      // block-uniform
    walk.r = last_not_above(plan_array(p.scratch, 0, p.batch.num_reqs), p.batch.num_reqs, walk.u);
    __syncwarp();
    if (wid == 0) {
        tc_alloc(smem_u32(&sh.tmem), 512);
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&sh.tmem);
    const uint32_t quad = (uint32_t)(wid & 3) << 21;      // this warp's 32 TMEM lanes
    XtSegment sg;
    uint32_t c = 0;                                       // blocks so far

    if (wid == W0 + 16) {
        // ======================= raw pages and query rows ==========================================
        uint32_t seg = 0, k_issued = 0, v_issued = 0;
        bool ok = true;
        while (ok && xt_next(p, walk, sg)) {
            const int32_t* blocks = p.batch.block_tables + (size_t)sg.r * p.batch.max_blocks_per_req;
            const uint8_t* kb = (const uint8_t*)(uintptr_t)p.layout.k_base + (size_t)sg.kv_head * p.layout.k_head_stride_bytes;
            const uint8_t* vb = (const uint8_t*)(uintptr_t)p.layout.v_base + (size_t)sg.kv_head * p.layout.v_head_stride_bytes;
            auto page_id = [&](int b) -> int32_t {
                const int pg = kXtPages * b + lane;
                return (lane < kXtPages && pg < sg.pages) ? block_table_page(blocks, sg.pg0 + pg, p.batch.max_blocks_per_req, kInStream) : -1;
            };
            int32_t id = page_id(0);
            ok = wait_all(bar(kXtQFree), (seg & 1u) ^ 1u);
            if (!ok) break;
            if (lane == 0) {
                const size_t idx = (size_t)(sg.r * p.layout.local_kv_heads + sg.kv_head) * p.q_groups_max + sg.group;
                mbar_expect_tx(bar(kXtQFull), kQueryBytes);
                bulk_g2s(q_t, reinterpret_cast<const uint8_t*>(p.qfrag) + idx * kQueryBytes, kQueryBytes, bar(kXtQFull));
            }
            __syncwarp();
            ++seg;
            for (int b = 0; kXtPages * b < sg.pages; ++b, ++c) {
                const int s = (int)(c % STAGES);
                const uint32_t lap = (c / STAGES) & 1u, bytes = (uint32_t)min(kXtPages, sg.pages - kXtPages * b) * kTq4PageHeadBytes;
                const int32_t next = page_id(b + 1);
                if (!(ok = wait_all(bar(kXtRawKFree + s), lap ^ 1u))) break;
                if (lane == 0) mbar_expect_tx(bar(kXtRawKFull + s), bytes);
                __syncwarp();
                if (id >= 0) {
                    bulk_g2s(raw_k(s) + (uint32_t)lane * kTq4PageHeadBytes, kb + (size_t)id * p.layout.k_page_stride_bytes, kTq4PageHeadBytes,
                             bar(kXtRawKFull + s));
                }
                k_issued = c + 1;
                if (!(ok = wait_all(bar(kXtRawVFree + s), lap ^ 1u))) break;
                if (lane == 0) mbar_expect_tx(bar(kXtRawVFull + s), bytes);
                __syncwarp();
                if (id >= 0) {
                    bulk_g2s(raw_v(s) + (uint32_t)lane * kTq4PageHeadBytes, vb + (size_t)id * p.layout.v_page_stride_bytes, kTq4PageHeadBytes,
                             bar(kXtRawVFull + s));
                }
                v_issued = c + 1;
                id = next;
            }
        }
        // copies in flight must land before the CTA leaves
        for (uint32_t j = k_issued > STAGES ? k_issued - STAGES : 0; j < k_issued; ++j) (void)mbar_wait(bar(kXtRawKFull + (int)(j % STAGES)), (j / STAGES) & 1u);
        for (uint32_t j = v_issued > STAGES ? v_issued - STAGES : 0; j < v_issued; ++j) (void)mbar_wait(bar(kXtRawVFull + (int)(j % STAGES)), (j / STAGES) & 1u);
        if (seg > 0) (void)mbar_wait(bar(kXtQFull), (seg - 1) & 1u);
        __syncwarp();
    } else if (wid == W0 + 17) {
        // ======================= score products =====================================================
        // An MMA of this size takes the tensor cores some 40 cycles, so that operands are kept where an issue needs no more than a
        // few instructions: warp-uniform bases, everything else constant.
        constexpr uint32_t kIdesc = tc_idesc(kXtKeys, N, 0);
        const uint64_t desc_q = tc_smem_desc(q_t, 16u, 1024u);
        const uint32_t base = __shfl_sync(0xffffffffu, tmem, 0);
        uint32_t seg = 0;
        bool ok = true;
        while (ok && xt_next(p, walk, sg)) {
            ok = wait_all(bar(kXtQFull), seg & 1u);
            for (int b = 0; ok && kXtPages * b < sg.pages; ++b, ++c) {
                ok = wait_all(bar(kXtSFree), (c & 1u) ^ 1u);      // the scores of the block before are in registers
#pragma unroll
                for (int gr = 0; gr < 8; ++gr) {
                    ok = ok && wait_all(bar(kXtKFull + (gr & 3)), (uint32_t)(gr >> 2));      // fills 2 c + (gr >> 2)
                    if (ok && elect_one()) {
                        tc_fence_after();
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {      // eight channels each
                            const uint64_t bq = desc_q + (uint64_t)(gr * (N * 128 / 16) + 2 * ks);
                            const uint32_t d = base + kXtColS + (uint32_t)((gr >> 2) * N), a = base + kXtColK + (uint32_t)(32 * (gr & 3) + 8 * ks);
                            if ((gr & 3) || ks) xt_mma<true>(d, a, bq, kIdesc);
                            else xt_mma<false>(d, a, bq, kIdesc);
                        }
                        tc_commit(bar(kXtKEmpty + (gr & 3)));
                        if (gr == 7) tc_commit(bar(kXtSReady));
                    }
                    __syncwarp();
                }
            }
            if (ok && elect_one()) tc_commit(bar(kXtQFree));
            __syncwarp();
            ++seg;
        }
        if (!ok) *aborted = 1u;
        if (elect_one()) tc_commit(bar(kXtDrain));      // nothing may be in flight when the CTA leaves
        __syncwarp();
        (void)mbar_wait(bar(kXtDrain), 0u);
        __syncwarp();
    } else if (wid == W0 + 18) {
        // ======================= output products ====================================================
        constexpr uint32_t kIdesc = tc_idesc(128, N, 0);
        const uint64_t desc_p = tc_smem_desc(p_t, 16u, 1024u);
        const uint32_t base = __shfl_sync(0xffffffffu, tmem, 0);
        bool ok = true;
        while (ok && xt_next(p, walk, sg)) {
            for (int b = 0; ok && kXtPages * b < sg.pages; ++b, ++c) {
#pragma unroll
                for (int kk = 0; kk < 2; ++kk) {
                    ok = ok && wait_all(bar(kXtPReady + kk), c & 1u);
                    ok = ok && wait_all(bar(kXtVFull), (uint32_t)kk);      // fill 2 c + kk
                    if (ok && elect_one()) {
                        tc_fence_after();
#pragma unroll
                        for (int res = 0; res < 2; ++res) {      // the centroids' values, then their residuals
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
#pragma unroll
                                for (int ks = 0; ks < 4; ++ks) {
                                    const uint64_t bp = desc_p + (uint64_t)(h * (int)(kPBytes / 16) + kk * (N * 128 / 16) + 2 * ks);
                                    const uint32_t d = base + kXtColO + (uint32_t)(h * N), a = base + kXtColV + (uint32_t)(64 * h + 32 * res + 8 * ks);
                                    if ((kk | res | ks) || b != 0) xt_mma<true>(d, a, bp, kIdesc);
                                    else xt_mma<false>(d, a, bp, kIdesc);
                                }
                            }
                        }
                        tc_commit(bar(kXtVEmpty));
                        tc_commit(bar(kXtPvDone + kk));
                    }
                    __syncwarp();
                }
            }
        }
        if (!ok) *aborted = 1u;
        if (elect_one()) tc_commit(bar(kXtDrain));
        __syncwarp();
        (void)mbar_wait(bar(kXtDrain), 0u);
        __syncwarp();
    } else if (wid >= W0 && wid < W0 + 8) {
        // ======================= V: 32 channels of a half, fragments of four keys a thread ===============
        const int gid = lane >> 2, tig = lane & 3, half = (wid - W0) >> 2;
        const int vw = 4 * (wid & 3) + (gid >> 1);                           // this thread's code word of the half
        const uint32_t word_off = 4u * ((half ? 17u : 0u) + (uint32_t)vw);
        const bool splice_warp = half == 0 && (wid & 3) == 0;                // virtual word 0: (W0 >> 16) | (W16 << 16)
        const uint32_t lut_lane = lut_addr + 8u * (uint32_t)(lane & 15);
        // byte 2 (gid & 1) + T of the paired codes belongs to tile T
        const uint32_t sel[2] = {0x7604u + ((uint32_t)(2 * (gid & 1)) << 4), 0x7604u + ((uint32_t)(2 * (gid & 1) + 1) << 4)};
        bool ok = true;
        while (ok && xt_next(p, walk, sg)) {
            for (int b = 0; ok && kXtPages * b < sg.pages; ++b, ++c) {
                const int s = (int)(c % STAGES);
                if (!(ok = wait_all(bar(kXtRawVFull + s), (c / STAGES) & 1u))) break;
                const uint32_t run = raw_v(s);
                const uint32_t rows = run + (uint32_t)(4 * tig) * kTq4RowBytes;
#pragma unroll 1
                for (int kk = 0; kk < 2; ++kk) {
                    uint32_t x[4][4];
#pragma unroll
                    for (int pg = 0; pg < 4; ++pg) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) x[pg][k] = lds32(rows + (uint32_t)(4 * kk + pg) * kTq4PageHeadBytes + (uint32_t)k * kTq4RowBytes + word_off);
                    }
                    if (splice_warp) {
#pragma unroll
                        for (int pg = 0; pg < 4; ++pg) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const uint32_t y = lds32(rows + (uint32_t)(4 * kk + pg) * kTq4PageHeadBytes + (uint32_t)k * kTq4RowBytes + 64u);
                                if (vw == 0) x[pg][k] = (x[pg][k] >> 16) | (y << 16);
                            }
                        }
                    }
#pragma unroll
                    for (int pg = 0; pg < 4; ++pg) {
                        // byte t of x[0] -> keys 0 and 1 of channel 2 t, x[1]: of channel 2 t + 1; x[2], x[3]: keys 2 and 3
                        const uint32_t w0 = x[pg][0], w1 = x[pg][1], w2 = x[pg][2], w3 = x[pg][3];
                        x[pg][0] = (w0 & 0x0f0f0f0fu) | ((w1 << 4) & 0xf0f0f0f0u);
                        x[pg][1] = ((w0 >> 4) & 0x0f0f0f0fu) | (w1 & 0xf0f0f0f0u);
                        x[pg][2] = (w2 & 0x0f0f0f0fu) | ((w3 << 4) & 0xf0f0f0f0u);
                        x[pg][3] = ((w2 >> 4) & 0x0f0f0f0fu) | (w3 & 0xf0f0f0f0u);
                    }
                    const uint32_t dst = tmem + quad + kXtColV + 64u * (uint32_t)half;
#pragma unroll
                    for (int part = 0; part < 4; ++part) {      // tile, pair of pages
                        const int T = part & 1, pg0 = part & 2;
                        uint32_t a[8], r[8];      // values, residuals: one look-up for both
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int pg = pg0 + (i >> 1), o = i & 1;
                            const uint2 e01 = lds64_lut(__byte_perm(x[pg][o], lut_lane, sel[T])), e23 = lds64_lut(__byte_perm(x[pg][2 + o], lut_lane, sel[T]));
                            a[2 * i] = e01.x;
                            r[2 * i] = e01.y;
                            a[2 * i + 1] = e23.x;
                            r[2 * i + 1] = e23.y;
                        }
                        if (part == 0) {
                            if (!(ok = wait_all(bar(kXtVEmpty), (uint32_t)(kk ^ 1)))) break;
                            tc_fence_after();      // the MMAs that read the granule come before the stores over it
                        }
                        tc_st_16x256b_x2(dst + ((uint32_t)(16 * T) << 16) + 8u * (uint32_t)pg0, a);
                        tc_st_16x256b_x2(dst + ((uint32_t)(16 * T) << 16) + 8u * (uint32_t)pg0 + 32u, r);
                    }
                    if (!ok) break;
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(kXtVFull));
                }
                __syncwarp();
                if (ok && lane == 0) mbar_arrive(bar(kXtRawVFree + s));
            }
        }
    } else if (wid >= W0 + 8 && wid < W0 + 16) {
        // ======================= K: thread = key ===================================================
        const int part = (wid - W0 - 8) >> 2, key = tid & 127;          // part 0 takes the even granules, part 1 the odd ones
        const uint32_t lutk_lane = lut_addr + 8u * (uint32_t)(lane & 15);
        bool ok = true;
        while (ok && xt_next(p, walk, sg)) {
            for (int b = 0; ok && kXtPages * b < sg.pages; ++b, ++c) {
                const int s = (int)(c % STAGES);
                if (!(ok = wait_all(bar(kXtRawKFull + s), (c / STAGES) & 1u))) break;
                const uint32_t rowp = raw_k(s) + (uint32_t)key * kTq4RowBytes;
                if (part == 0) {
                    sh.k_scale[c & 1][key] = make_float2(__half2float(__ushort_as_half((unsigned short)(lds32(rowp) & 0xffffu))),
                                                         __half2float(__ushort_as_half((unsigned short)(lds32(rowp + 64) >> 16))));
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(kXtKScale + (int)(c & 1)));
                }
#pragma unroll 1
                for (int gr = part; gr < 8; gr += 2) {
                    const uint32_t slot = (uint32_t)gr & (kXtKRing - 1), lap = 2u * c + ((uint32_t)gr >> 2);
                    uint32_t x[5], w[4];
                    const uint32_t at = rowp + 16u * (uint32_t)(gr & 3) + (gr >= 4 ? 68u : 0u);
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[i] = lds32(at + 4u * i);
                    x[4] = lds32(at + (gr < 4 ? 16u : 12u));
                    const uint32_t shift = gr < 4 ? 16u : 0u;            // half 0 starts at byte 2
#pragma unroll
                    for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(x[i], x[i + 1], shift);
                    uint32_t e[32];      // values and residuals of 16 pairs of channels
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const uint2 v = lds64_lut(__byte_perm(w[i >> 2], lutk_lane, 0x7604 + ((i & 3) << 4)));
                        e[2 * i] = v.x;
                        e[2 * i + 1] = v.y;
                    }
                    if (!(ok = wait_all(bar(kXtKEmpty + (int)slot), (lap & 1u) ^ 1u))) break;
                    tc_fence_after();
                    tc_st32(tmem + quad + kXtColK + 32u * slot, e);
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(kXtKFull + (int)slot));
                }
                __syncwarp();
                if (ok && lane == 0) mbar_arrive(bar(kXtRawKFree + s));
            }
        }
    } else if (wid < W0) {
        // ======================= softmax: thread = key, a part = eight rows =============================================
        constexpr int P = 8;
        const int part = wid >> 2, row0 = part * P, key = tid & 127, khalf = (wid & 3) >> 1;
        const uint32_t t_s = tmem + quad + kXtColS + (uint32_t)row0, t_o = tmem + quad + kXtColO + (uint32_t)row0;
        float* m_ref = sh.m_ref + row0;      // this part's rows
        float* alpha = sh.alpha + row0;
        float* mass = sh.mass + row0;
        int *row_min = sh.row_min + row0, *row_max = sh.row_max + row0;
        float* red = &sh.red[0][row0];
        float* partials = reinterpret_cast<float*>(p.scratch + plan_bytes(p.batch.num_reqs));
        // The four warps share barriers, so that one whose wait gave up carries on (nothing it reads can be out of bounds) and
        // all leave together behind a vote at the end of a segment; no wait after the first that gave up takes any time.
        bool failed = false;
        while (xt_next(p, walk, sg)) {
            const ReqGeom g = load_req(p.batch, sg.r);
            if (key < P) {
                const int row = sg.group * R + row0 + key, q_off = row / p.gqa;
                const bool valid = row < g.q_len * p.gqa && (p.batch.valid_token_mask == nullptr || p.batch.valid_token_mask[g.q_start + q_off] != 0);
                row_max[key] = valid ? row_max_kv(p.batch, g, q_off) : -1;
                row_min[key] = valid ? row_min_kv(p.batch, g, q_off) : 0x7fffffff;
                m_ref[key] = -1e30f;
                mass[key] = 0.0f;
            }
            xt_sync(part);
            int safe_lo = 0, safe_hi = 0x7fffffff;      // keys every valid row can see
#pragma unroll
            for (int i = 0; i < P; ++i) {
                if (row_max[i] >= 0) {
                    safe_lo = max(safe_lo, row_min[i]);
                    safe_hi = min(safe_hi, row_max[i]);
                }
            }
            float v_up = 1.0f;         // power of two by which P d_v is multiplied
            float l[P], m_lag[P];      // this key's mass of every row; the reference maxima plus the lag
#pragma unroll
            for (int i = 0; i < P; ++i) {
                l[i] = 0.0f;
                m_lag[i] = -1e30f;
            }
            // mass of every row over all keys, into sh.mass
            auto reduce_mass = [&]() {
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    float t = l[i];
#pragma unroll
                    for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
                    if (lane == 0) red[(wid & 3) * 24 + i] = t;
                }
                xt_sync(part);
                if (key < P) mass[key] = (red[0 + key] + red[24 + key]) + (red[48 + key] + red[72 + key]);
                xt_sync(part);
            };
            const int nblocks = (sg.pages + kXtPages - 1) / kXtPages;
#pragma unroll 1
            for (int b = 0; b < nblocks; ++b, ++c) {
                bool bad = !wait_all(bar(kXtKScale + (int)(c & 1)), (c >> 1) & 1u);
                const float2 dk = sh.k_scale[c & 1][key];
                bad = bad || !wait_all(bar(kXtSReady), c & 1u);
                tc_fence_after();
                float sc[P];
#pragma unroll
                for (int i0 = 0; i0 < P; i0 += 4) {
                    uint32_t h0[4], l0[4], h1[4], l1[4];
                    tc_ld4(h0, t_s + (uint32_t)i0);
                    tc_ld4(l0, t_s + (uint32_t)(R + i0));
                    tc_ld4(h1, t_s + (uint32_t)(N + i0));
                    tc_ld4(l1, t_s + (uint32_t)(N + R + i0));
                    tc_wait_ld();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        sc[i0 + i] = dk.x * (__uint_as_float(h0[i]) + __uint_as_float(l0[i])) + dk.y * (__uint_as_float(h1[i]) + __uint_as_float(l1[i]));
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(kXtSFree));
                const int kv_base = (sg.pg0 + kXtPages * b) << 4;
                const int last = (min(kXtPages, sg.pages - kXtPages * b) << 4) - 1;       // keys past it are not in the block
                const bool full = kv_base >= safe_lo && kv_base + kXtKeys - 1 <= safe_hi && last == kXtKeys - 1;
                const int pos = kv_base + key;
                if (!full) {
#pragma unroll
                    for (int i = 0; i < P; ++i) {
                        if (key > last || pos < row_min[i] || pos > row_max[i]) sc[i] = -INFINITY;
                    }
                }
                bad = bad || !wait_all(bar(kXtRawVFull + (int)(c % STAGES)), (c / STAGES) & 1u);
                const uint32_t v_row = raw_v((int)(c % STAGES)) + (uint32_t)key * kTq4RowBytes;
                float2 dv = make_float2(__half2float(__ushort_as_half((unsigned short)(lds32(v_row) & 0xffffu))),
                                        __half2float(__ushort_as_half((unsigned short)(lds32(v_row + 64) >> 16))));
                if (!full) {      // a key no row can see may hold never-written bytes: its scale must not meet a zero weight
                    bool seen = false;
#pragma unroll
                    for (int i = 0; i < P; ++i) seen = seen || sc[i] > -INFINITY;
                    if (!seen) dv = make_float2(0.0f, 0.0f);
                }
                const float v_most = fmaxf(fabsf(dv.x), fabsf(dv.y));
                bool ahead = v_most * v_up > 32768.0f && v_most <= 65504.0f;      // (infinite scales have no power of two)
#pragma unroll
                for (int i = 0; i < P; ++i) ahead = ahead || sc[i] > m_lag[i];
                const bool moved = xt_any(ahead, part);
                float v_by = 1.0f;
                if (moved) {      // the reference maximum of some row moves, or V outgrows its power of two: take the block's maxima
                    {
                        float t = v_most <= 65504.0f ? v_most : 0.0f;
#pragma unroll
                        for (int d = 16; d > 0; d >>= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, d));
                        if (lane == 0) sh.red_v[wid & 3][part] = t;
                    }
#pragma unroll
                    for (int i = 0; i < P; ++i) {
                        float t = sc[i];
#pragma unroll
                        for (int d = 16; d > 0; d >>= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, d));
                        if (lane == 0) red[(wid & 3) * 24 + i] = t;
                    }
                    xt_sync(part);
                    if (key < P) {
                        const float old = m_ref[key];
                        const float now = fmaxf(fmaxf(fmaxf(red[0 + key], red[24 + key]), fmaxf(red[48 + key], red[72 + key])), old);
                        const float a = ex2(old - now);      // 0 when nothing was visible before
                        m_ref[key] = now;
                        alpha[key] = a;
                    }
                    xt_sync(part);
#pragma unroll
                    for (int i = 0; i < P; ++i) {
                        l[i] *= alpha[i];
                        m_lag[i] = m_ref[i] + kXtLag;
                    }
                    const float t = fmaxf(fmaxf(sh.red_v[0][part], sh.red_v[1][part]), fmaxf(sh.red_v[2][part], sh.red_v[3][part]));
                    if (t > 0.0f) {
                        v_by = 1.0f / v_up;      // (powers of two throughout)
                        v_up = __uint_as_float((uint32_t)(127 + 11 + 127 - (int)(__float_as_uint(t) >> 23)) << 23);
                        v_by *= v_up;
                    }
                }
                // This half of the keys' P is in use until its output product of the block before has completed, O until both have.  (The
                // halves follow each other: one's weights are written while the other is multiplied.)
                bad = bad || (c > 0 && !wait_all(bar(kXtPvDone + khalf), (c - 1) & 1u));
                if (moved && b > 0) {
                    // (The other half's barrier is not waited for in every block.  Its parity is enough all the same: products complete in
                    // order, so that its phase before this one is over by the wait above, and this block's cannot be, for the other
                    // half's weights come behind the barrier below.)
                    bad = bad || !wait_all(bar(kXtPvDone + (khalf ^ 1)), (c - 1) & 1u);
                    tc_fence_after();
#pragma unroll 1
                    for (int q = 0; q < 4; ++q) {      // value and residual columns of both halves
#pragma unroll
                        for (int i0 = 0; i0 < P; i0 += 4) {
                            uint32_t o[4];
                            tc_ld4(o, t_o + (uint32_t)(q * R + i0));
                            tc_wait_ld();
#pragma unroll
                            for (int i = 0; i < 4; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * (alpha[i0 + i] * v_by));
                            tc_st4(t_o + (uint32_t)(q * R + i0), o);
                        }
                    }
                    tc_wait_st();
                    tc_fence_before();
                    xt_sync(part);      // neither half's product starts before all four warps have rescaled their channels
                }
                dv.x *= v_up;
                dv.y *= v_up;
                const uint64_t dv2 = pair_of(dv.x, dv.y), minus_one = pair_of(-1.0f, -1.0f);
                // 16-byte chunk of the key's column, swizzled by the row
                const uint32_t at = p_t + (uint32_t)(key >> 6) * (uint32_t)(N * 128) + (uint32_t)row0 * 128u + 2u * (uint32_t)(key & 7) +
                                    (((uint32_t)(key & 63) >> 3) << 4);
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    const float w = ex2(sc[i] - m_lag[i]);
                    l[i] += w;
                    uint64_t x, rest;      // of both halves: w d_v, and what its fp16 values leave
                    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(x) : "l"(pair_of(w, w)), "l"(dv2));
                    const __half2 h = __floats2half2_rn(__uint_as_float((uint32_t)x), __uint_as_float((uint32_t)(x >> 32)));
                    const float2 hf = __half22float2(h);
                    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rest) : "l"(pair_of(hf.x, hf.y)), "l"(minus_one), "l"(x));
                    const uint32_t hi = *reinterpret_cast<const uint32_t*>(&h), lo = pack_half2(__uint_as_float((uint32_t)rest), __uint_as_float((uint32_t)(rest >> 32)));
                    const uint32_t a = (at ^ (uint32_t)(i << 4)) + (uint32_t)i * 128u;
                    sts16(a, hi);
                    sts16(a + (uint32_t)R * 128u, lo);
                    sts16(a + kPBytes, hi >> 16);
                    sts16(a + kPBytes + (uint32_t)R * 128u, lo >> 16);
                }
                if (bad) failed = true;
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(bar(kXtPReady + khalf));
                    mbar_arrive(bar(kXtRawVFree + (int)(c % STAGES)));
                }
            }
            // ---- the item's share is done: write the partial (lane = channel) ----------------------
            reduce_mass();
            if (failed || !wait_all(bar(kXtPvDone), (c - 1) & 1u) || !wait_all(bar(kXtPvDone + 1), (c - 1) & 1u)) failed = true;
            tc_fence_after();
            if (sg.slot < p.max_slots) {
                float* dst = partials + (size_t)sg.slot * (R * kHeadDim + 2 * R);
                // TMEM lane 32 q + 16 T + gid (+ 8): code word 4 q + gid / 2, channels 2 (2 (gid & 1) + T) (+ 1) of it
                const int T = lane >> 4, gid = lane & 7, odd = (lane >> 3) & 1;
                const float v_down = 1.0f / v_up;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int ch = vword_col(h, 4 * (wid & 3) + (gid >> 1), 2 * (2 * (gid & 1) + T) + odd);
#pragma unroll
                    for (int i0 = 0; i0 < P; i0 += 4) {
                        uint32_t a[4], b4[4];
                        tc_ld4(a, t_o + (uint32_t)(h * N + i0));
                        tc_ld4(b4, t_o + (uint32_t)(h * N + R + i0));
                        tc_wait_ld();
#pragma unroll
                        for (int i = 0; i < 4; ++i) dst[(row0 + i0 + i) * kHeadDim + ch] = (__uint_as_float(a[i]) + __uint_as_float(b4[i])) * v_down;
                    }
                }
                if (key < P) {
                    dst[R * kHeadDim + row0 + key] = m_ref[key] + kXtLag;
                    dst[R * kHeadDim + R + row0 + key] = mass[key];
                }
            }
            tc_fence_before();
            if (xt_any(failed, part)) break;
        }
    }

    __syncthreads();
    if (wid == 0) {
        tc_fence_after();
        tc_dealloc(tmem, 512);
    }
    if (*aborted != 0u && tid == 0) atomicOr(&hdr->status, 1);
}

}  // namespace w34
