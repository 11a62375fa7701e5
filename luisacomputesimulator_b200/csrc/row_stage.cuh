// row_stage.cuh -- products of 32-row slices of a 3x3-block CSR matrix, one warp per slice.
//
// Four lanes share a row (lane g of four takes blocks rp + g, rp + g + 4, ...), which read straight from global
// memory costs nine 4-byte loads at a 36-byte stride.  With 2,048 threads per SM those loads hide each other's latency
// (k_spmv); a cluster that owns a scene has 256 to 512 threads per SM and waits for them.  So the blocks of 8
// consecutive rows -- one contiguous run of the CSR -- are brought into shared memory by bulk copies (two stages per
// warp, the next run in flight while one is multiplied); there the 9-word stride of the blocks is free of bank
// conflicts.  Measured figures stand at the kernels that use it.
#pragma once
#include <cstdint>

#include "lcs_common.cuh"

namespace lcs {
namespace stage {

// Blocks per copy: 8 rows of a cloth have 96 (6 edges and 6 wings each), irregular ones about 100; a group
// of 8 longer rows takes several copies.
constexpr uint32_t kWin = 104;
constexpr uint32_t kValBytes = kWin * 36 + 16;   // runs start anywhere in the CSR: up to 12 bytes before them
constexpr uint32_t kColBytes = kWin * 4 + 16;
constexpr uint32_t kStageBytes = kValBytes + kColBytes;
constexpr uint32_t kWarpBytes = 2 * kStageBytes;
static_assert(kValBytes % 16 == 0 && kColBytes % 16 == 0, "bulk copies are 16-byte aligned");
constexpr uint32_t kPollNs = 1000;         // a poll of a copy's barrier suspends for at most this long
constexpr uint32_t kWaitLimit = 1u << 20;  // polls before a warp gives up on a copy: about a second

struct Csr {
    const uint32_t* rp;
    const uint32_t* col;
    const float* val;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void bar_expect(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// the barrier's phase waits for `bytes` more than the copies bring
__device__ __forceinline__ void bar_expect_more(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool bar_try(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(kPollNs) : "memory");
    return ok != 0;
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// y += M v for a column-major 3x3 block
__device__ __forceinline__ void add_block(const float* m, const float4 v, float3& y)
{
    y.x += __fmaf_rn(m[6], v.z, __fmaf_rn(m[3], v.y, m[0] * v.x));
    y.y += __fmaf_rn(m[7], v.z, __fmaf_rn(m[4], v.y, m[1] * v.x));
    y.z += __fmaf_rn(m[8], v.z, __fmaf_rn(m[5], v.y, m[2] * v.x));
}

// One warp's copies of matrix A's blocks in flight.  All members are uniform over the warp.
struct Warp {
    unsigned char* buf;   // kWarpBytes, 16-byte aligned
    uint64_t* bar;        // two barriers (null: nothing is staged)
    Csr A, B;
    uint32_t nnz;         // blocks of A (the copies never read past them)
    bool bulk;            // A's arrays are 16-byte aligned and no copy has failed; else the blocks are read directly
    uint32_t use = 0;     // copies consumed: stage use & 1, parity (use >> 1) & 1
    uint32_t ahead = 0;   // copies in flight (0 to 2)
    uint32_t limit = kWaitLimit;
    bool failed = false;  // a copy did not arrive within the limit

    __device__ __forceinline__ void init(unsigned char* b, uint64_t* barriers, const Csr& a, const Csr& extra,
                                         uint32_t n_rows)
    {
        buf = b;
        bar = barriers;
        A = a;
        B = extra;
        nnz = a.rp ? __ldg(&a.rp[n_rows]) : 0u;
        bulk = ((reinterpret_cast<uintptr_t>(a.val) | reinterpret_cast<uintptr_t>(a.col)) & 15u) == 0;
        if (bar && lane_id() == 0) {
            bar_init(&bar[0]);
            bar_init(&bar[1]);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
    }

    // bytes copied for words [w0 & ~3, ...) of an array of `total` words, n of them wanted from w0
    static __device__ __forceinline__ uint32_t copy_bytes(uint64_t w0, uint32_t n, uint64_t total)
    {
        const uint64_t from = w0 & ~3ull, to = (w0 + n + 3) & ~3ull;
        return 4u * (uint32_t)((to <= total ? to : (total & ~3ull)) - from);
    }

    __device__ __forceinline__ void issue(uint32_t k0, uint32_t n)
    {
        if (lane_id() == 0) {
            const uint32_t s = (use + ahead) & 1u;
            unsigned char* d = buf + s * kStageBytes;
            const uint64_t w0 = 9ull * k0;
            const uint32_t vb = copy_bytes(w0, 9 * n, 9ull * nnz), cb = copy_bytes(k0, n, nnz);
            bar_expect(&bar[s], vb + cb);
            if (vb) bulk_load(d, A.val + (w0 & ~3ull), vb, &bar[s]);
            if (cb) bulk_load(d + kValBytes, A.col + (k0 & ~3u), cb, &bar[s]);
        }
        ++ahead;
    }

    // whether the oldest copy in flight has arrived, within the limit
    __device__ __forceinline__ bool arrived()
    {
        const uint32_t s = use & 1u, parity = (use >> 1) & 1u;
        uint32_t it = 0;
        bool ok;
        while (!(ok = bar_try(&bar[s], parity)) && ++it < limit) {
        }
        return __all_sync(0xFFFFFFFFu, ok);
    }

    // Waits for the oldest copy.  A warp that gives up never looks at a stage again (its words may be anything): it
    // issues no further copies and reads the blocks directly from there on.
    __device__ __forceinline__ void wait()
    {
        if (arrived()) return;
        failed = true;
        bulk = false;
    }

    // before the end of a warp that gave up: one more bounded wait for each copy it left in flight
    __device__ __forceinline__ void drain()
    {
        for (; ahead > 0; ++use, --ahead) arrived();
    }
};

// A slice of 32 rows [base, base + 32) below `row_end`: lane l holds the block ranges of row base + l (empty beyond).
struct Slice {
    uint32_t lo, hi;    // blocks of A
    uint32_t blo, bhi;  // blocks of B

    __device__ __forceinline__ void load(const Warp& w, uint32_t base, uint32_t row_end)
    {
        lo = hi = blo = bhi = 0;
        if (base >= row_end) return;
        const uint32_t r = min(base + lane_id(), row_end), r1 = min(r + 1, row_end);
        if (w.A.rp) {
            lo = __ldg(&w.A.rp[r]);
            hi = __ldg(&w.A.rp[r1]);
        }
        if (w.B.rp) {
            blo = __ldg(&w.B.rp[r]);
            bhi = __ldg(&w.B.rp[r1]);
        }
    }
    __device__ __forceinline__ uint32_t first() const { return __shfl_sync(0xFFFFFFFFu, lo, 0); }
    __device__ __forceinline__ uint32_t last() const { return __shfl_sync(0xFFFFFFFFu, hi, 31); }
    // the end of the group of 8 rows that block k of A lies in (k < last())
    __device__ __forceinline__ uint32_t group_end(uint32_t k) const
    {
        const uint32_t past = __ballot_sync(0xFFFFFFFFu, hi > k);  // rows that end after k; the first of them holds it
        return __shfl_sync(0xFFFFFFFFu, hi, (__ffs(past) - 1) | 7);
    }
    // puts the window that starts at block k in flight, or none if A has no blocks there
    __device__ __forceinline__ void prefetch(Warp& w, uint32_t k) const
    {
        if (!w.bulk || k >= last()) return;
        w.issue(k, min(kWin, group_end(k) - k));
    }
};

// acc += blocks k, k + G, ... < end of a matrix times x, read directly
template <int G, class Load>
__device__ __forceinline__ void direct_blocks(const Csr& M, uint32_t k, uint32_t end, const Load& ld, float3& acc)
{
#pragma unroll 1
    for (; k < end; k += G) {
        const float4 v = ld(__ldg(&M.col[k]));
        float m[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) m[e] = __ldg(&M.val[9 * (size_t)k + e]);
        add_block(m, v, acc);
    }
}

template <int G>
__device__ __forceinline__ void group_sum(float3& v)
{
#pragma unroll
    for (int o = G >> 1; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xFFFFFFFFu, v.x, o);
        v.y += __shfl_xor_sync(0xFFFFFFFFu, v.y, o);
        v.z += __shfl_xor_sync(0xFFFFFFFFu, v.z, o);
    }
}

// Off-diagonal product (A + B) x of the slice's rows: on return lane l holds row l's sum.
// `next` is the warp's next slice: its first window is put in flight while this slice ends (and this slice's first
// window may be in flight already).  B (contacts) is read directly: copies of its short, uneven runs made a batched
// solve 6% slower with few contacts and 45% with many.  ld(col) reads one vector of x.
// Staged = false reads A directly too (no shared memory, no barriers): for launches whose CTAs fill the GPU with threads,
// and for a warp's single slice, where the copies only add their latency.
template <bool Staged, class Load>
__device__ __forceinline__ float3 slice_product(Warp& w, const Slice& cur, const Slice& next, const Load& ld)
{
    const uint32_t lane = lane_id(), g = lane >> 2, lig = lane & 3u;
    const uint32_t a_first = cur.first(), a_last = cur.last();
    const bool has_b = __any_sync(0xFFFFFFFFu, cur.blo < cur.bhi);
    if (Staged && w.ahead == 0) cur.prefetch(w, a_first);
    float3 keep = make_float3(0.f, 0.f, 0.f);
    uint32_t k0 = a_first;
    if (Staged && k0 == a_last) next.prefetch(w, next.first());
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
        float3 acc = make_float3(0.f, 0.f, 0.f);
        const uint32_t ge = __shfl_sync(0xFFFFFFFFu, cur.hi, 8 * j + 7);
        const uint32_t rs = __shfl_sync(0xFFFFFFFFu, cur.lo, 8 * j + g);
        const uint32_t re = __shfl_sync(0xFFFFFFFFu, cur.hi, 8 * j + g);
        uint32_t k = rs + lig;
        while (Staged && w.bulk && k0 < ge) {
            const uint32_t nb = min(kWin, ge - k0), k1 = k0 + nb;
            if (w.ahead == 0) w.issue(k0, nb);
            if (k1 < a_last) cur.prefetch(w, k1);
            else next.prefetch(w, next.first());
            w.wait();
            if (w.failed) break;
            unsigned char* d = w.buf + (w.use & 1u) * kStageBytes;
            float* sv = reinterpret_cast<float*>(d) + ((9u * k0) & 3u);
            uint32_t* sc = reinterpret_cast<uint32_t*>(d + kValBytes) + (k0 & 3u);
            if (k1 + 4 > w.nnz) {  // the last words of the arrays, where a 16-byte copy would pass their end
                const int have = (int)(Warp::copy_bytes(9ull * k0, 9 * nb, 9ull * w.nnz) / 4) - (int)((9u * k0) & 3u);
                for (int c = max(have, 0) + (int)lane; c < (int)(9 * nb); c += 32)
                    sv[c] = __ldg(&w.A.val[9ull * k0 + c]);
                const int havec = (int)(Warp::copy_bytes(k0, nb, w.nnz) / 4) - (int)(k0 & 3u);
                for (int c = max(havec, 0) + (int)lane; c < (int)nb; c += 32) sc[c] = __ldg(&w.A.col[k0 + c]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
            }
            const uint32_t kend = min(re, k1);
            for (; k < kend; k += 16) {
                float4 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (k + 4 * u < kend) v[u] = ld(sc[k + 4 * u - k0]);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (k + 4 * u < kend) add_block(sv + 9 * (k + 4 * u - k0), v[u], acc);
            }
            // a row cut by the window's end goes on at its next block of this lane
            if (k1 < re) k = rs + lig + (rs + lig < k1 ? (k1 - rs - lig + 3) / 4 * 4 : 0u);
            __syncwarp();  // the stage is free for the copy after next
            ++w.use;
            --w.ahead;
            k0 = k1;
        }
        if (!Staged || !w.bulk) {  // k: the lane's next block, also where the copies ended in the middle of the row
            direct_blocks<4>(w.A, k, re, ld, acc);
            k0 = ge;
        }
        if (has_b) {
            const uint32_t bs = __shfl_sync(0xFFFFFFFFu, cur.blo, 8 * j + g);
            const uint32_t be = __shfl_sync(0xFFFFFFFFu, cur.bhi, 8 * j + g);
            direct_blocks<4>(w.B, bs + lig, be, ld, acc);
            __syncwarp();
        }
        group_sum<4>(acc);
        if (lig == (uint32_t)j) keep = acc;
    }
    // lane 4 g + j holds row 8 j + g; lane l takes row l
    const int from = 4 * (lane & 7u) + (lane >> 3);
    return make_float3(__shfl_sync(0xFFFFFFFFu, keep.x, from), __shfl_sync(0xFFFFFFFFu, keep.y, from),
                       __shfl_sync(0xFFFFFFFFu, keep.z, from));
}

}  // namespace stage
}  // namespace lcs
