// k_lists.cu -- neighbour lists (CSR) of the exact self join.
//
// The reference returns only the total (gpu_join.cu:210-322); its result-set
// kernels (kernel_join.cu:139-162) are dead code.  Here the join emits its
// neighbour pairs while it counts them: the tensor-core screen appends one
// in-record per row and chunk of columns with certain neighbours, the band
// recheck and the FP64 arbiter append single pairs.  Every neighbour pair is
// emitted exactly once (the screens visit each unordered pair once; kBandBoth
// marks pairs that credit both points), so the per-point counts give the CSR
// offsets, and a scatter through per-point cursors fills the lists; a check then
// requires every cursor to end exactly at the next point's offset, and a sort of
// every list puts it in ascending order (deterministic output).
#include <type_traits>

#include <cub/cub.cuh>

#include "ejoin_internal.cuh"

namespace ejoin {
namespace {

__global__ void widen_kernel(const int32_t* __restrict__ c, uint64_t n, unsigned long long* out) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = (uint32_t)c[i];
}

__device__ __forceinline__ void put(unsigned long long* cur, uint32_t* nb, uint64_t total,
                                    uint32_t at, uint32_t value, unsigned* err) {
    const unsigned long long slot = atomicAdd(&cur[at], 1ull);
    if (slot < total) nb[slot] = value;
    else atomicOr(err, 1u);
}

// in-records: the pairs (i, j0 + c) for the set bits c (packed indices)
__global__ void scatter_in_kernel(const BandRec* __restrict__ rec, uint64_t nrec,
                                  const uint32_t* __restrict__ perm, uint64_t n,
                                  unsigned long long* cur, uint32_t* nb, uint64_t total,
                                  unsigned* err) {
    const uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (e >= nrec) return;
    const BandRec r = rec[e];
    const uint32_t j0 = r.j0 & ~kBandBoth;
    const bool both = (r.j0 & kBandBoth) != 0;
    if (r.i >= n) {
        atomicOr(err, 2u);
        return;
    }
    const uint32_t oi = perm ? perm[r.i] : r.i;
    uint32_t m = r.mask;
    while (m) {
        const uint32_t c = __ffs(m) - 1;
        m &= m - 1;
        const uint32_t j = j0 + c;
        if (j >= n) {
            atomicOr(err, 2u);
            continue;
        }
        const uint32_t oj = perm ? perm[j] : j;
        put(cur, nb, total, oi, oj, err);
        if (both) put(cur, nb, total, oj, oi, err);
    }
}

// single pairs (i, j | both) (packed indices)
__global__ void scatter_pairs_kernel(const BandPair* __restrict__ pq, uint64_t np,
                                     const uint32_t* __restrict__ perm, uint64_t n,
                                     unsigned long long* cur, uint32_t* nb, uint64_t total,
                                     unsigned* err) {
    const uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (e >= np) return;
    const BandPair p = pq[e];
    const uint32_t i = p.i, j = p.j & ~kBandBoth;
    if (i >= n || j >= n) {
        atomicOr(err, 2u);
        return;
    }
    const uint32_t oi = perm ? perm[i] : i, oj = perm ? perm[j] : j;
    put(cur, nb, total, oi, oj, err);
    if (p.j & kBandBoth) put(cur, nb, total, oj, oi, err);
}

__global__ void check_cursor_kernel(const unsigned long long* __restrict__ cur,
                                    const unsigned long long* __restrict__ off, uint64_t n,
                                    unsigned* err) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < n && cur[i] != off[i + 1]) atomicOr(err, 4u);
}

// Sorts the lists of at most kShort entries, a warp per list: the list in shared
// memory, every entry's place the number of smaller ones (they are distinct),
// one comparison per pair of entries against broadcast reads.  Longer lists are
// noted for the kernels that follow: in mid up to kMid entries, in longs beyond.
// (A segmented sort over all lists took 443 us for 4.8 M entries in lists of 32.)
// Comparisons bound it: 140,000 lists of up to 128, 29 on average, take 73 us with
// four entries per lane for all, 54 with as many as the list needs.
struct ListSpans {
    unsigned long long *begin, *end;
    unsigned* count;
};
constexpr uint32_t kShort = 128, kSortWarps = 8, kMid = 1024;
__global__ void __launch_bounds__(kSortWarps * 32)
    sort_lists_kernel(const unsigned long long* __restrict__ off, uint64_t n,
                      const uint32_t* __restrict__ raw, uint32_t* __restrict__ nb,
                      ListSpans mid, ListSpans longs) {
    __shared__ __align__(16) uint32_t keys[kSortWarps][kShort];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x / 32;
    const uint64_t i = blockIdx.x * (uint64_t)kSortWarps + w;
    if (i >= n) return;
    const unsigned long long o0 = off[i], o1 = off[i + 1];
    if (o1 - o0 > kShort) {
        if (lane == 0) {
            const ListSpans& to = o1 - o0 > kMid ? longs : mid;
            const unsigned at = atomicAdd(to.count, 1u);
            to.begin[at] = o0;
            to.end[at] = o1;
        }
        return;
    }
    const uint32_t len = (uint32_t)(o1 - o0);
    auto sort = [&](auto rc) {  // with R entries per lane
        constexpr uint32_t R = decltype(rc)::value;
        uint32_t key[R], rank[R];
#pragma unroll
        for (uint32_t r = 0; r < R; ++r) {
            const uint32_t e = lane + 32 * r;
            // (no entry is as large: indices stay below 2^31)
            key[r] = e < len ? raw[o0 + e] : 0xffffffffu;
            rank[r] = 0;
            keys[w][e] = key[r];
        }
        __syncwarp();
        for (uint32_t e = 0; e < len; e += 4) {
            const uint4 k = *reinterpret_cast<const uint4*>(&keys[w][e]);
#pragma unroll
            for (uint32_t r = 0; r < R; ++r)
                rank[r] += (k.x < key[r]) + (k.y < key[r]) + (k.z < key[r]) + (k.w < key[r]);
        }
#pragma unroll
        for (uint32_t r = 0; r < R; ++r)
            if (lane + 32 * r < len) nb[o0 + rank[r]] = key[r];
    };
    if (len <= 32) sort(std::integral_constant<uint32_t, 1>{});
    else if (len <= 64) sort(std::integral_constant<uint32_t, 2>{});
    else sort(std::integral_constant<uint32_t, kShort / 32>{});
}

// The same for lists of kShort + 1 to kMid entries, a block per list, two entries
// per thread and pass: comparisons bound it.  (2.1 M entries in 10,072 lists of up
// to 828: 94 us; the segmented sort took 660.  The comparisons grow with the square
// of the length, so the longest lists stay with that sort.)
constexpr uint32_t kMidThreads = 128;
__global__ void __launch_bounds__(kMidThreads)
    sort_mid_kernel(const uint32_t* __restrict__ raw, uint32_t* __restrict__ nb, ListSpans mid) {
    __shared__ __align__(16) uint32_t keys[kMid];
    const uint32_t t = threadIdx.x, nlists = *mid.count;
    for (uint32_t i = blockIdx.x; i < nlists; i += gridDim.x) {
        const unsigned long long o0 = mid.begin[i];
        const uint32_t len = min((uint32_t)(mid.end[i] - o0), kMid), len4 = (len + 3) & ~3u;
        for (uint32_t e = t; e < len4; e += kMidThreads) keys[e] = e < len ? raw[o0 + e] : 0xffffffffu;
        __syncthreads();
        for (uint32_t e0 = t; e0 < len; e0 += 2 * kMidThreads) {
            const uint32_t e1 = e0 + kMidThreads;
            const uint32_t k0 = keys[e0], k1 = e1 < len ? keys[e1] : 0u;
            uint32_t r0 = 0, r1 = 0;
            for (uint32_t e = 0; e < len4; e += 4) {
                const uint4 k = *reinterpret_cast<const uint4*>(&keys[e]);
                r0 += (k.x < k0) + (k.y < k0) + (k.z < k0) + (k.w < k0);
                r1 += (k.x < k1) + (k.y < k1) + (k.z < k1) + (k.w < k1);
            }
            nb[o0 + r0] = k0;
            if (e1 < len) nb[o0 + r1] = k1;
        }
        __syncthreads();  // keys are replaced
    }
}

}  // namespace

int csr_offsets(const int32_t* counts, uint64_t n, uint64_t total, unsigned long long* offsets,
                cudaStream_t s) {
    if (n > 0x7fffffffull) return set_error(EJOIN_EUNSUPPORTED, "neighbour lists: too many points");
    if (n) {
        DBuf<unsigned long long> w;
        EJ_TRY(w.alloc(n, s, "list lengths"));
        widen_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(counts, n, w.p);
        EJ_CUDA(cudaGetLastError());
        size_t tb = 0;
        EJ_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, w.p, offsets, (int)n, s));
        DBuf<uint8_t> tmp;
        EJ_TRY(tmp.alloc(tb, s, "scan scratch"));
        EJ_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, w.p, offsets, (int)n, s));
        note_launch(2);
    }
    const unsigned long long t = total;
    EJ_CUDA(cudaMemcpyAsync(offsets + n, &t, sizeof t, cudaMemcpyHostToDevice, s));
    EJ_CUDA(cudaStreamSynchronize(s));
    return EJOIN_OK;
}

int csr_fill(const unsigned long long* offsets, uint64_t n, uint64_t total, const BandRec* inq,
             uint64_t nin, const BandPair* pq, uint64_t np, const uint32_t* perm, uint32_t* nb,
             cudaStream_t s) {
    if (total > 0x7fffffffull)
        return set_error(EJOIN_EUNSUPPORTED, "neighbour lists: %llu pairs exceed 2^31 - 1",
                         (unsigned long long)total);
    if (total == 0) return EJOIN_OK;
    DBuf<unsigned long long> cur;
    DBuf<uint32_t> raw;
    DBuf<unsigned> err;
    EJ_TRY(cur.alloc(n, s, "list cursors"));
    EJ_TRY(raw.alloc(total, s, "unsorted lists"));
    EJ_TRY(err.alloc(1, s, "list check"));
    EJ_TRY(err.zero(s));
    EJ_CUDA(cudaMemcpyAsync(cur.p, offsets, n * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, s));
    if (nin)
        scatter_in_kernel<<<(unsigned)((nin + 255) / 256), 256, 0, s>>>(inq, nin, perm, n, cur.p,
                                                                        raw.p, total, err.p);
    if (np)
        scatter_pairs_kernel<<<(unsigned)((np + 255) / 256), 256, 0, s>>>(pq, np, perm, n, cur.p,
                                                                          raw.p, total, err.p);
    check_cursor_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(cur.p, offsets, n, err.p);
    EJ_CUDA(cudaGetLastError());
    note_launch(3);
    // (total entries bound the lists of each kind)
    const uint64_t most_mid = total / (kShort + 1) + 1, most_long = total / (kMid + 1) + 1;
    DBuf<unsigned long long> spans;
    DBuf<unsigned> nl;
    EJ_TRY(spans.alloc(2 * (most_mid + most_long), s, "long lists"));
    EJ_TRY(nl.alloc(2, s, "long lists"));
    EJ_TRY(nl.zero(s));
    const ListSpans mid{spans.p, spans.p + most_mid, nl.p};
    const ListSpans longs{mid.end + most_mid, mid.end + most_mid + most_long, nl.p + 1};
    sort_lists_kernel<<<(unsigned)((n + kSortWarps - 1) / kSortWarps), kSortWarps * 32, 0, s>>>(
        offsets, n, raw.p, nb, mid, longs);
    sort_mid_kernel<<<(unsigned)std::min<uint64_t>(most_mid, 152 * 16), kMidThreads, 0, s>>>(raw.p, nb, mid);
    EJ_CUDA(cudaGetLastError());
    note_launch(2);
    unsigned h[2] = {0, 0};
    EJ_CUDA(cudaMemcpyAsync(&h[0], err.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    EJ_CUDA(cudaMemcpyAsync(&h[1], longs.count, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    EJ_CUDA(cudaStreamSynchronize(s));
    if (h[0]) return set_error(EJOIN_EINTERNAL, "neighbour lists: emitted pairs disagree with the counts (%u)", h[0]);
    if (h[1]) {
        size_t tb = 0;
        EJ_CUDA(cub::DeviceSegmentedSort::SortKeys(nullptr, tb, raw.p, nb, (int)total, (int)h[1],
                                                   longs.begin, longs.end, s));
        DBuf<uint8_t> tmp;
        EJ_TRY(tmp.alloc(tb, s, "sort scratch"));
        EJ_CUDA(cub::DeviceSegmentedSort::SortKeys(tmp.p, tb, raw.p, nb, (int)total, (int)h[1],
                                                   longs.begin, longs.end, s));
        note_launch(2);
    }
    return EJOIN_OK;
}

}  // namespace ejoin
