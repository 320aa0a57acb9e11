// match.cu — brute-force descriptor matching: for every query descriptor the
// nearest and second-nearest train descriptor by Euclidean distance, the
// input of Lowe's ratio test. Not part of the reference crate; it consumes
// the 128-float descriptors that detect_and_compute returns.
//
// Squared distances are |q|^2 + |t|^2 - 2 q.t. The products q.t run on the
// 5th-generation tensor cores (tcgen05, TF32 operands, f32 accumulators in
// tensor memory) over TMA-staged 128-descriptor tiles; they only select
// candidates: the 4 best per query and quarter of the columns of a CTA's
// train tiles. A second kernel keeps those that TF32's error lets be among the
// best two and ranks them by exact f32 dot products. Ties go to the lower
// train index, so the result does not depend on how the tiles are split over
// the CTAs.
#include <cuda.h>

#include <algorithm>

#include "sift_internal.cuh"
#include "tma.cuh"

namespace sift {
namespace {

constexpr int kD = kDescLen;

struct Best2 {
    float d1, d2;
    int i1, i2;
};

__device__ __forceinline__ bool before(float d, int i, float e, int j) { return d < e || (d == e && i < j); }

__device__ __forceinline__ void push(Best2& b, float d, int i) {
    if (before(d, i, b.d1, b.i1)) {
        b.d2 = b.d1;
        b.i2 = b.i1;
        b.d1 = d;
        b.i1 = i;
    } else if (before(d, i, b.d2, b.i2)) {
        b.d2 = d;
        b.i2 = i;
    }
}

// The best two of two best-two lists.
__device__ __forceinline__ Best2 fold(const Best2& a, const Best2& b) {
    Best2 r;
    if (before(a.d1, a.i1, b.d1, b.i1)) {
        r.d1 = a.d1;
        r.i1 = a.i1;
        const bool sa = before(a.d2, a.i2, b.d1, b.i1);
        r.d2 = sa ? a.d2 : b.d1;
        r.i2 = sa ? a.i2 : b.i1;
    } else {
        r.d1 = b.d1;
        r.i1 = b.i1;
        const bool sb = before(b.d2, b.i2, a.d1, a.i1);
        r.d2 = sb ? b.d2 : a.d1;
        r.i2 = sb ? b.i2 : a.i1;
    }
    return r;
}

// The rows' squared norms, each an FMA chain in index order, and, for rows in
// host memory, their device copy. 32 rows per CTA: a warp reads whole rows
// (512 contiguous bytes, the host link's best case) into shared memory, then
// the 32 lanes of one warp sum a row each. 2 x 7.5 MB of pageable rows come in
// at 200 GB/s (76 us; as copies, about 120 us before the norms began).
constexpr int kNormRows = 32, kNormThreads = 256;
struct NormJob {
    const float* src;
    float* dst;   // device copy, or null where src is on the device
    float* norm;  // n_pad values; rows from n on: +inf, never a candidate
    uint32_t n, n_pad;
};
// most: receives the largest squared norm of b's rows (its bits; zero before).
__global__ void __launch_bounds__(kNormThreads) k_sq_norms(NormJob a, NormJob b, uint32_t blocks_a,
                                                           uint32_t* __restrict__ most) {
    __shared__ float row[kNormRows][kD + 1];
    const NormJob& j = blockIdx.x < blocks_a ? a : b;
    const uint32_t r0 = (blockIdx.x - (blockIdx.x < blocks_a ? 0u : blocks_a)) * kNormRows;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4 v[kNormRows / 8];
#pragma unroll
    for (int i = 0; i < kNormRows / 8; ++i) {
        const uint32_t r = r0 + warp + 8 * i;
        v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r < j.n) v[i] = reinterpret_cast<const float4*>(j.src + (size_t)r * kD)[lane];
    }
#pragma unroll
    for (int i = 0; i < kNormRows / 8; ++i) {
        const uint32_t r = r0 + warp + 8 * i;
        if (j.dst && r < j.n) reinterpret_cast<float4*>(j.dst + (size_t)r * kD)[lane] = v[i];
        float* d = row[warp + 8 * i] + 4 * lane;
        d[0] = v[i].x;
        d[1] = v[i].y;
        d[2] = v[i].z;
        d[3] = v[i].w;
    }
    __syncthreads();
    if (warp || r0 + lane >= j.n_pad) return;
    float s = 0.0f;
#pragma unroll 16
    for (int k = 0; k < kD; ++k) s = fmaf(row[lane][k], row[lane][k], s);
    j.norm[r0 + lane] = r0 + lane < j.n ? s : INFINITY;
    // squared norms are not negative (a NaN's bits are above infinity's), so their bits order them
    if (blockIdx.x >= blocks_a && r0 + lane < j.n) atomicMax(most, __float_as_uint(fabsf(s)));
}

constexpr int kCand = 4;
// A TF32 product is within 2^-9 |q| |t| of the exact one (each operand within
// 2^-10 of its f32 value), so a value |t|^2 - 2 q.t is within kTf32Err |q| |t|
// of the exact one, its f32 roundings included.
constexpr float kTf32Err = 0.0045f;

// ---------------------------------------------------------------------------
// 5th-generation tensor cores (tcgen05) with TMA-staged operands.
//
// The (query tile, train tile) pairs, query tile by query tile, are split
// evenly over one CTA per multiprocessor; a CTA's share covers one or a few
// query tiles (segments). The query tile (128 rows x 128 floats, 64 KB) and
// the train tiles (128 rows, double-buffered) are loaded by TMA
// (cp.async.bulk.tensor, 128-byte swizzle: four 32-float boxes per tile) into
// the K-major layout the MMA reads. One thread issues
// tcgen05.mma.kind::tf32 (M = 128 queries, N = 128 train, K = 8 per
// instruction, 16 per tile) into one of two 128-column f32 accumulators in
// tensor memory, so the epilogue of one tile overlaps the products of the
// next. The epilogue warps own the accumulator's lanes: a thread reads one
// query row's products of a quarter of the tile with tcgen05.ld and keeps the
// row's 4 best columns of these quarters of the segment by |t|^2 - 2 q.t.
//
// The epilogue bounds the kernel. A compare and a branch per column made a
// serial chain of 64 branches per tile in which some lane of a warp almost
// always had a new candidate (325 us for 14671 x 14747, 6000 cycles per tile
// against 1200 for its products). Now a lane looks at four columns at once:
// only their smallest is compared with the lane's bound, and four columns that
// hold a candidate go to the lane's queue in shared memory by predicated
// stores, without a branch. Queues are emptied once per tile (or when one may
// overflow), all lanes together, so a warp pays for its longest queue and not
// for every column that some lane wants. A queue's columns are inserted in
// column order, so the 4 best are the same as one by one. The bound is the
// 4th best, or what TF32's error leaves a chance against the 2nd best if that
// is lower. Sixteen epilogue warps (four per scheduler) hide the chains of
// each other.
//
// Roles: warps 0-15 epilogue (warp w: tensor-memory lanes 32 (w % 4) .., a
// quarter w / 4 of each tile's columns), warp 16 TMA producer, warp 17 MMA
// issuer and tensor-memory owner. Every mbarrier
// wait is bounded; a wait that runs out sets the error word and the CTA
// leaves through the same exit (tensor memory is always freed).
constexpr int kUM = 128, kUN = 128;                   // MMA M (queries) and N (train rows per tile)
constexpr int kUEpi = 512, kUThreads = kUEpi + 64;  // warps 0-15 epilogue, 16 TMA, 17 MMA
constexpr int kUCols = kUN / (kUEpi / 128);          // columns of a tile per epilogue warp
constexpr int kUParts = kUN / kUCols;                // candidate lists per row and segment
constexpr uint32_t kUAtom = kUM * 128;                // one 32-float K slice of a 128-row tile: 16 KB
constexpr uint32_t kUTile = 4 * kUAtom;               // 64 KB
constexpr int kUQueue = 4;  // queued column quads per epilogue thread
constexpr uint32_t kUSmem = 3 * kUTile + kUQueue * kUEpi * 16 + 1024 + 512;  // query tile, two train stages, queues,
                                                                           // alignment, barriers
constexpr uint32_t kUTmemCols = 2 * kUN;
constexpr uint32_t kUSpin = 1u << 26;                 // bounded waits (~seconds)

// bounded mbarrier waits of this kernel
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity) { return sift::mbar_wait(b, parity, kUSpin); }
// Shared-memory matrix descriptor of a K-major operand with 128-byte
// swizzling: 8-row groups of 128-byte rows, 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// Instruction descriptor: D f32, A and B tf32, both K-major, N = 128, M = 128.
constexpr uint32_t kUIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(kUN >> 3) << 17) | ((uint32_t)(kUM >> 4) << 24);

__device__ __forceinline__ void umma_tf32(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}" ::"r"(
            dtmem),
        "l"(adesc), "l"(bdesc), "r"(kUIdesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// starts the read of 16 columns; the values are there after tmem_ld_wait
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
          "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait(float (&r)[16]) {
    // the registers pass through, so no use of them can move above the wait
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]),
                   "+f"(r[8]), "+f"(r[9]), "+f"(r[10]), "+f"(r[11]), "+f"(r[12]), "+f"(r[13]), "+f"(r[14]), "+f"(r[15])
                 :
                 : "memory");
}

// How the pairs of tiles are split: `per` consecutive pairs per CTA; a query
// tile's pairs lie in CTAs first .. first + slots - 1.
struct Split {
    uint32_t qt, tt, per;  // query tiles, train tiles, pairs per CTA
    __host__ __device__ uint64_t pairs() const { return (uint64_t)qt * tt; }
    __host__ __device__ uint32_t first(uint32_t q) const { return (uint32_t)((uint64_t)q * tt / per); }
    __host__ __device__ uint32_t slots(uint32_t q) const {
        return (uint32_t)(((uint64_t)q * tt + tt - 1) / per) - first(q) + 1;
    }
    __host__ __device__ uint32_t max_slots() const { return tt ? (uint32_t)(((uint64_t)tt + per - 2) / per) + 1 : 0; }
    __host__ __device__ uint32_t ctas() const { return (uint32_t)((pairs() + per - 1) / per); }
};
// A queue entry of four columns whose smallest value is below the bound:
// predicated, no branch. Entry addresses go by kUEpi * 16 bytes, `which` gets
// the quad's bit.
__device__ __forceinline__ void push_below(float4 d, float bound, uint32_t& addr, uint32_t& which, uint32_t bit) {
    const float m = fminf(fminf(d.x, d.y), fminf(d.z, d.w));
    asm volatile(
        "{\n .reg .pred p;\n setp.lt.f32 p, %2, %3;\n @p st.shared.v4.f32 [%0], {%4, %5, %6, %7};\n"
        " @p add.u32 %0, %0, %8;\n @p or.b32 %1, %1, %9;\n}"
        : "+r"(addr), "+r"(which)
        : "f"(m), "f"(bound), "f"(d.x), "f"(d.y), "f"(d.z), "f"(d.w), "n"(kUEpi * 16), "r"(bit)
        : "memory");
}

// A candidate: |t|^2 - 2 q.t as the tensor cores see it, and t's index (-1:
// none). A row's candidates are contiguous: by slot, part of the tile's
// columns, place.
struct Cand {
    float d;
    int i;
};

__global__ void __launch_bounds__(kUThreads, 1)
    k_match_umma(const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmt,
                 const float* __restrict__ qn, const float* __restrict__ tn, const uint32_t* __restrict__ most, Split sp,
                 Cand* __restrict__ cand, uint32_t* __restrict__ err) {
    extern __shared__ uint8_t usm_raw[];
    uint8_t* usm = reinterpret_cast<uint8_t*>(((uintptr_t)usm_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* qs = usm;                     // [4 K slices][128 rows][128 B], swizzled
    uint8_t* ts = usm + kUTile;            // [2 stages] of the same
    float4* queue = reinterpret_cast<float4*>(usm + 3 * kUTile);  // [kUQueue][kUEpi] column quads
    uint64_t* bars = reinterpret_cast<uint64_t*>(queue + kUQueue * kUEpi);
    uint64_t* q_full = bars;               // query tile landed
    uint64_t* t_full = bars + 1;           // [2] train stage landed
    uint64_t* t_empty = bars + 3;          // [2] train stage consumed by the MMAs
    uint64_t* acc_full = bars + 5;         // [2] accumulator complete
    uint64_t* acc_empty = bars + 7;        // [2] accumulator read by the epilogue
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 9);
    uint32_t* bad = tmem_slot + 1;         // a wait of this CTA ran out
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint64_t lo = (uint64_t)blockIdx.x * sp.per, hi = min(lo + sp.per, sp.pairs());
    const int ntile = hi > lo ? (int)(hi - lo) : 0;
    const uint32_t qt0 = (uint32_t)(lo / sp.tt), tl0 = (uint32_t)(lo - (uint64_t)qt0 * sp.tt);  // the first pair
    if (tid == 0) {
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(t_full + i, 1);
            mbar_init(t_empty + i, 1);
            mbar_init(acc_full + i, 1);
            mbar_init(acc_empty + i, kUEpi);
        }
        *bad = 0u;
        mbar_init_fence();
    }
    if (warp == kUEpi / 32 + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kUTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == kUEpi / 32) {
        if (lane == 0) {
            // each segment's query tile, its train tiles through two stages
            int issued = 0, seg = -1;
            uint32_t qt = qt0, tl = tl0;
            for (int j = 0; j < ntile; ++j) {
                const int st = j & 1;
                bool ok = j < 2 || mbar_wait(t_empty + st, ((j >> 1) - 1) & 1);
                const bool next_q = j == 0 || tl == 0;
                // the last segment's products must have read the query tile
                if (ok && next_q && j > 0) ok = mbar_wait(t_empty + ((j - 1) & 1), ((j - 1) >> 1) & 1);
                if (!ok) {
                    atomicOr(bad, 1u);
                    break;
                }
                if (next_q) {
                    ++seg;
                    mbar_expect_tx(q_full, kUTile);
                    for (int a = 0; a < 4; ++a) tma_load_2d(qs + a * kUAtom, &tmq, 32 * a, (int)qt * kUM, q_full);
                }
                mbar_expect_tx(t_full + st, kUTile);
                for (int a = 0; a < 4; ++a)
                    tma_load_2d(ts + st * kUTile + a * kUAtom, &tmt, 32 * a, (int)tl * kUN, t_full + st);
                issued = j + 1;
                if (++tl == sp.tt) {
                    tl = 0;
                    ++qt;
                }
            }
            // no copy of this CTA may still be landing when it exits (on the
            // normal path these phases completed long ago)
            bool landed = seg < 0 || mbar_wait(q_full, seg & 1);
            for (int j = issued - 2 < 0 ? 0 : issued - 2; j < issued; ++j)
                landed = mbar_wait(t_full + (j & 1), (j >> 1) & 1) && landed;
            if (!landed) atomicOr(bad, 1u);
        }
    } else if (warp == kUEpi / 32 + 1) {
        if (lane == 0) {
            bool ok = true;
            int seg = -1;
            uint32_t tl = tl0;
            for (int j = 0; ok && j < ntile; ++j) {
                const int st = j & 1, b = j & 1;
                if (j == 0 || tl == 0) ok = mbar_wait(q_full, ++seg & 1);
                if (++tl == sp.tt) tl = 0;
                ok = ok && mbar_wait(t_full + st, (j >> 1) & 1);
                if (ok && j >= 2) ok = mbar_wait(acc_empty + b, ((j >> 1) - 1) & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t qa = smem_u32(qs), ta = smem_u32(ts + st * kUTile);
#pragma unroll
                for (int k = 0; k < kD / 8; ++k) {
                    // K slice k / 4, 32-byte step k % 4 inside the swizzled 128-byte rows
                    const uint32_t off = (uint32_t)(k >> 2) * kUAtom + (uint32_t)(k & 3) * 32u;
                    umma_tf32(tmem + (uint32_t)(b * kUN), umma_desc(qa + off), umma_desc(ta + off), k > 0 ? 1u : 0u);
                }
                umma_commit(t_empty + st);
                umma_commit(acc_full + b);
            }
            if (!ok) atomicOr(bad, 1u);
        }
    } else {
        // epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. (query
        // rows) and columns kUCols (w / 4) .. of each tile; its candidates
        // are ranked by |t|^2 - 2 q.t (the row's |q|^2 is common to all)
        const int quarter = warp & 3, part = warp >> 2;
        const uint32_t r = (uint32_t)(quarter * 32 + lane), lists = (uint32_t)kUParts * sp.max_slots();
        const uint32_t queue0 = smem_u32(queue + tid);
        // twice the error that a value of this row can have
        const float tmax = sqrtf(__uint_as_float(*most));
        float window = 0.0f, bound = INFINITY;
        float c0 = INFINITY, c1 = INFINITY, c2 = INFINITY, c3 = INFINITY;
        int k0 = -1, k1 = -1, k2 = -1, k3 = -1;
        // columns rise, so a tie never goes before an earlier one
        auto insert = [&](float d, int col) {
            {
                const bool b3 = d < c3, b0 = d < c0, b1 = d < c1, b2 = d < c2;
                c3 = b2 ? c2 : (b3 ? d : c3);
                k3 = b2 ? k2 : (b3 ? col : k3);
                c2 = b1 ? c1 : (b2 ? d : c2);
                k2 = b1 ? k1 : (b2 ? col : k2);
                c1 = b0 ? c0 : (b1 ? d : c1);
                k1 = b0 ? k0 : (b1 ? col : k1);
                c0 = b0 ? d : c0;
                k0 = b0 ? col : k0;
            }
        };
        bool ok = true;
        uint32_t qt = qt0, tl = tl0;
        for (int j = 0; j < ntile; ++j) {
            const int b = j & 1;
            const int col0 = (int)tl * kUN + part * kUCols;
            if (j == 0 || tl == 0) {
                window = 2.0f * kTf32Err * sqrtf(qn[qt * kUM + r]) * tmax;
                bound = INFINITY;
            }
            // the columns' train norms (padded with +inf past the end)
            float4 tv[kUCols / 4];
#pragma unroll
            for (int q = 0; q < kUCols / 4; ++q) tv[q] = reinterpret_cast<const float4*>(tn + col0)[q];
            if (ok) ok = mbar_wait(acc_full + b, (j >> 1) & 1);
            if (__all_sync(0xffffffffu, ok)) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * kUN + part * kUCols);
                float v[kUCols / 16][16];
#pragma unroll
                for (int c = 0; c < kUCols / 16; ++c) tmem_ld16(taddr + 16u * c, v[c]);
#pragma unroll
                for (int c = 0; c < kUCols / 16; ++c) tmem_ld_wait(v[c]);
                // every column is in registers: the accumulator is free
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(acc_empty + b);
                uint32_t addr = queue0, which = 0;
#pragma unroll
                for (int q = 0; q < kUCols / 4; ++q) {
                    const float2 two = make_float2(-2.0f, -2.0f);
                    const float4 t = tv[q];
                    const float* x = &v[q / 4][4 * (q % 4)];
                    const float2 d01 = __ffma2_rn(two, make_float2(x[0], x[1]), make_float2(t.x, t.y));
                    const float2 d23 = __ffma2_rn(two, make_float2(x[2], x[3]), make_float2(t.z, t.w));
                    push_below(make_float4(d01.x, d01.y, d23.x, d23.y), bound, addr, which, 1u << q);
                    if (q % 2 == 0) continue;
                    // room for the next two quads; nothing waits past the tile
                    const bool end = q == kUCols / 4 - 1;
                    if (__any_sync(0xffffffffu, addr > queue0 + (end ? 0 : (kUQueue - 2) * kUEpi * 16))) {
                        const int most_queued = __reduce_max_sync(0xffffffffu, __popc(which));
                        const float4* e = queue + tid;
#pragma unroll 1
                        for (int i = 0; i < most_queued; ++i, e += kUEpi) {
                            if (which) {
                                const int col = col0 + 4 * (__ffs(which) - 1);
                                which &= which - 1u;
                                const float4 d = *e;
                                // the lanes' columns below the bound, one from
                                // each lane at a time (mostly one in all)
                                uint32_t in = (d.x < bound ? 1u : 0u) | (d.y < bound ? 2u : 0u) |
                                              (d.z < bound ? 4u : 0u) | (d.w < bound ? 8u : 0u);
                                while (in) {
                                    const int at = __ffs(in) - 1;
                                    in &= in - 1u;
                                    insert(at & 2 ? (at & 1 ? d.w : d.z) : (at & 1 ? d.y : d.x), col + at);
                                }
                            }
                        }
                        __syncwarp();
                        addr = queue0;
                        bound = fminf(c3, c1 + window);  // (a NaN window bounds nothing)
                    }
                }
            } else {
                ok = false;
                atomicOr(bad, 1u);
                mbar_arrive(acc_empty + b);
            }
            const bool last = j + 1 == ntile || tl + 1 == sp.tt;
            if (last) {  // the segment's candidates
                const uint32_t list = (uint32_t)kUParts * (blockIdx.x - sp.first(qt)) + (uint32_t)part;
                Cand* c = cand + ((size_t)(qt * kUM + r) * lists + list) * kCand;
                reinterpret_cast<int4*>(c)[0] = make_int4(__float_as_int(c0), k0, __float_as_int(c1), k1);
                reinterpret_cast<int4*>(c)[1] = make_int4(__float_as_int(c2), k2, __float_as_int(c3), k3);
                c0 = c1 = c2 = c3 = INFINITY;
                k0 = k1 = k2 = k3 = -1;
            }
            if (++tl == sp.tt) {
                tl = 0;
                ++qt;
            }
        }
    }
    // every tensor-core operation of this CTA is complete before the barrier:
    // the epilogue waited for the last accumulator (or the MMA thread stopped)
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*bad && tid == 0) atomicOr(err, 1u);
    if (warp == kUEpi / 32 + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kUTmemCols) : "memory");
    }
}

// The best two of a query's candidates by exact f32 dot products (an FMA
// chain in index order), as distances; a warp per query, its lanes over the
// candidates. A candidate is dropped without its dot product when its value
// cannot be among the best two (kTf32Err).
constexpr int kRankWarps = 8, kRankRows = 8, kRankStride = kD + 4;  // 528-byte rows: lanes on rows in distinct banks
__global__ void __launch_bounds__(32 * kRankWarps) k_match_rank(const float* __restrict__ q,
                                                                const float* __restrict__ qn, uint32_t nq,
                                                                const float* __restrict__ t,
                                                                const float* __restrict__ tn, Split sp,
                                                                const Cand* __restrict__ cand,
                                                                SiftCudaMatch* __restrict__ out,
                                                                const uint32_t* __restrict__ err,
                                                                uint32_t* __restrict__ err_out) {
    __shared__ SiftCudaMatch found[kRankWarps];
    __shared__ int kept_of[kRankWarps][32 + kRankRows];
    __shared__ __align__(16) float stage[kRankWarps][(kRankRows + 1) * kRankStride];  // candidate rows, the query
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t row = blockIdx.x * kRankWarps + warp;
    const uint32_t bad = *err;
    if (err_out && blockIdx.x == 0 && threadIdx.x == 0) *err_out = bad;
    if (row < nq) {
        constexpr uint32_t kList = kUParts * kCand;  // candidates per slot
        const uint32_t n = sp.tt && !bad ? kList * sp.slots(row / kUM) : 0u;
        const Cand* c = cand + (size_t)row * kList * sp.max_slots();
        float* rows = stage[warp];
        float* qs = rows + kRankRows * kRankStride;
        reinterpret_cast<float4*>(qs)[lane] = reinterpret_cast<const float4*>(q + (size_t)row * kD)[lane];
        const float qnr = qn[row], ql = kTf32Err * sqrtf(qnr);
        // the second smallest upper bound of the row's candidates (NaN
        // bounds, of infinite values, drop nothing)
        float u1 = INFINITY, u2 = INFINITY;
        for (uint32_t e = lane; e < n; e += 32) {
            const Cand x = c[e];
            if (x.i < 0) continue;
            const float u = x.d + ql * sqrtf(tn[x.i]);
            if (u < u1) {
                u2 = u1;
                u1 = u;
            } else if (u < u2) {
                u2 = u;
            }
        }
        __syncwarp();
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const float o1 = __shfl_xor_sync(0xffffffffu, u1, m), o2 = __shfl_xor_sync(0xffffffffu, u2, m);
            u2 = fminf(fmaxf(u1, o1), fminf(u2, o2));
            u1 = fminf(u1, o1);
        }
        // the kept candidates are collected and, up to kRankRows at a time,
        // the warp brings their rows in, whole rows, and a lane each sums its
        // product
        Best2 b{INFINITY, INFINITY, -1, -1};
        int* kept = kept_of[warp];
        int count = 0;
        auto sum_products = [&](int m) {
            __syncwarp();
            const int i = lane < m ? kept[lane] : 0;
            const float tnr = lane < m ? tn[i] : 0.0f;
            float4 v[kRankRows];
#pragma unroll
            for (int r = 0; r < kRankRows; ++r)
                if (r < m)
                    v[r] = reinterpret_cast<const float4*>(t + (size_t)__shfl_sync(0xffffffffu, i, r) * kD)[lane];
#pragma unroll
            for (int r = 0; r < kRankRows; ++r)
                if (r < m) reinterpret_cast<float4*>(rows + r * kRankStride)[lane] = v[r];
            __syncwarp();
            if (lane < m) {
                const float4* tv = reinterpret_cast<const float4*>(rows + lane * kRankStride);
                const float4* qv = reinterpret_cast<const float4*>(qs);
                float dot = 0.0f;
#pragma unroll 8
                for (int k4 = 0; k4 < kD / 4; ++k4) {
                    const float4 a4 = qv[k4], c4 = tv[k4];
                    dot = fmaf(a4.x, c4.x, dot);
                    dot = fmaf(a4.y, c4.y, dot);
                    dot = fmaf(a4.z, c4.z, dot);
                    dot = fmaf(a4.w, c4.w, dot);
                }
                push(b, fmaf(-2.0f, dot, qnr + tnr), i);
            }
            __syncwarp();
        };
        for (uint32_t e0 = 0; e0 < n; e0 += 32) {
            Cand x{0.0f, -1};
            if (e0 + lane < n) x = c[e0 + lane];
            const bool keep = x.i >= 0 && !(x.d - ql * sqrtf(tn[max(x.i, 0)]) > u2);
            const uint32_t m = __ballot_sync(0xffffffffu, keep);
            if (keep) kept[count + __popc(m & ((1u << lane) - 1u))] = x.i;
            count += __popc(m);
            while (count >= kRankRows || (count > 0 && e0 + 32 >= n)) {
                const int now = min(count, kRankRows);
                sum_products(now);
                // the others move to the front
                const int i = lane < count - now ? kept[now + lane] : 0;
                __syncwarp();
                count -= now;
                if (lane < count) kept[lane] = i;
            }
        }
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            Best2 o;
            o.d1 = __shfl_xor_sync(0xffffffffu, b.d1, m);
            o.d2 = __shfl_xor_sync(0xffffffffu, b.d2, m);
            o.i1 = __shfl_xor_sync(0xffffffffu, b.i1, m);
            o.i2 = __shfl_xor_sync(0xffffffffu, b.i2, m);
            b = fold(b, o);
        }
        if (lane == 0) {
            SiftCudaMatch m;
            m.train_idx = b.i1;
            m.distance = b.i1 >= 0 ? sqrtf(fmaxf(b.d1, 0.0f)) : INFINITY;
            m.second_idx = b.i2;
            m.second_distance = b.i2 >= 0 ? sqrtf(fmaxf(b.d2, 0.0f)) : INFINITY;
            found[warp] = m;
        }
    }
    __syncthreads();
    // the CTA's results in one write (out may be host memory)
    const uint32_t r = blockIdx.x * kRankWarps + threadIdx.x;
    if (threadIdx.x < kRankWarps && r < nq) out[r] = found[threadIdx.x];
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }
// train norms, padded to whole 128-descriptor tiles
size_t tn_floats(uint32_t nt) { return ((size_t)nt + 127) / 128 * 128; }

Split split_of(uint32_t nq, uint32_t nt) {
    Split sp;
    sp.qt = (nq + kUM - 1) / kUM;
    sp.tt = (nt + kUN - 1) / kUN;
    sp.per = (uint32_t)std::max<uint64_t>((sp.pairs() + 151) / 152, 1);
    return sp;
}

// Scratch: query norms, train norms, the error word, candidates.
struct Scratch {
    size_t qn, tn, err, cand, total;
    Scratch(uint32_t nq, uint32_t nt) {
        const Split sp = split_of(nq, nt);
        const size_t cands = (size_t)sp.max_slots() * kUParts * kCand * sp.qt * kUM;
        qn = 0;
        tn = qn + align256((size_t)sp.qt * kUM * 4);
        err = tn + align256(tn_floats(nt) * 4);
        cand = err + 256;
        total = cand + align256(cands * sizeof(Cand));
    }
};

// Rows x 128 floats, boxes of 32 floats (128 bytes, the swizzle span) x 128
// rows; rows past the end read as zeros.
bool descriptor_map(CUtensorMap* m, const float* base, uint32_t rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)kD, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)kD * sizeof(float)};
    const cuuint32_t box[2] = {32u, 128u};
    const cuuint32_t estr[2] = {1u, 1u};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

size_t match_scratch_bytes(uint32_t nq, uint32_t nt) { return Scratch(nq, nt).total; }

// h_q, h_t: host rows that the device can read, copied to d_q and d_t on the
// way (null: d_q and d_t hold the rows). err_out: where the error word goes
// beside the results, or null.
int launch_match(const float* d_q, uint32_t nq, const float* d_t, uint32_t nt, SiftCudaMatch* d_out, void* scratch,
                 cudaStream_t st, const float* h_q, const float* h_t, uint32_t* err_out) {
    if (nq == 0) return 0;
    const Split sp = split_of(nq, nt);
    const Scratch sc(nq, nt);
    char* p = static_cast<char*>(scratch);
    float* qn = reinterpret_cast<float*>(p + sc.qn);
    float* tn = reinterpret_cast<float*>(p + sc.tn);
    uint32_t* err = reinterpret_cast<uint32_t*>(p + sc.err);  // set by a tensor-core CTA whose wait ran out
    Cand* cand = reinterpret_cast<Cand*>(p + sc.cand);
    uint32_t* most = err + 1;  // bits of the largest squared train norm
    if (cudaMemsetAsync(err, 0, 2 * sizeof(uint32_t), st) != cudaSuccess) return -1;
    const NormJob a{h_q ? h_q : d_q, h_q ? const_cast<float*>(d_q) : nullptr, qn, nq, sp.qt * (uint32_t)kUM};
    const NormJob b{h_t ? h_t : d_t, h_t ? const_cast<float*>(d_t) : nullptr, tn, nt, (uint32_t)tn_floats(nt)};
    const uint32_t ba = (a.n_pad + kNormRows - 1) / kNormRows, bb = (b.n_pad + kNormRows - 1) / kNormRows;
    k_sq_norms<<<ba + bb, kNormThreads, 0, st>>>(a, b, ba, most);
    if (sp.tt) {
        CUtensorMap mq, mt;
        if (!descriptor_map(&mq, d_q, nq) || !descriptor_map(&mt, d_t, nt)) return -1;
        if (cudaFuncSetAttribute(k_match_umma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUSmem) != cudaSuccess)
            return -1;
        k_match_umma<<<sp.ctas(), kUThreads, kUSmem, st>>>(mq, mt, qn, tn, most, sp, cand, err);
    }
    k_match_rank<<<(nq + kRankWarps - 1) / kRankWarps, 32 * kRankWarps, 0, st>>>(d_q, qn, nq, d_t, tn, sp, cand, d_out,
                                                                              err, err_out);
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace sift
