// k_misc.cu -- tile-pair work lists, totals and count scatter.
//
// Work list: blocks of two 128-row tiles (I0, I1) x two 128-column tiles (Ja, Jb)
// covering the upper-triangle tile pairs (I <= J), in blocked order
// (tri_decode_blocked), so that the CTAs running concurrently share operand rows in
// L2, and the band records that they write can be rechecked from rows in L2.
// Each entry carries a mask of its active tile pairs (in the upper triangle,
// below the last data tile, and not proven empty by the learned projection; see
// k_learn.cu for the bound).  The two column tiles of a block need not be
// adjacent: the column tiles with an active pair in the block's rows are paired
// within a super-block, so that a block's second half is idle only for the last,
// odd one.
#include <cub/cub.cuh>

#include "ejoin_internal.cuh"

namespace ejoin {
namespace {

constexpr uint32_t SB = kSuperTiles;  // super-block edge (tiles)

// Squared gap between two projected boxes, rounded down (so `> thr` proves
// that every pair of points drawn from the two boxes is farther apart than
// the projected threshold).  Empty boxes (lo = +inf, hi = -inf) are far from
// everything.
__device__ __forceinline__ bool boxes_far(const float* __restrict__ lo, const float* __restrict__ hi,
                                          uint64_t I, uint64_t J, uint32_t k, float thr) {
    float g2 = 0.0f;
    for (uint32_t a = 0; a < k; ++a) {
        const float l1 = lo[I * k + a], h1 = hi[I * k + a];
        const float l2 = lo[J * k + a], h2 = hi[J * k + a];
        const float gap = fmaxf(0.0f, fmaxf(__fsub_rd(l2, h1), __fsub_rd(l1, h2)));
        g2 = __fmaf_rd(gap, gap, g2);
    }
    return g2 > thr;
}

// Entry e of the triangle row <= column < n in blocked order: super-rows of H rows;
// a super-row's diagonal triangle (row-major) comes first, then, W columns at a
// time, all its rows (row-major inside).  Closed form: the entries ahead of a
// super-row are those of the plain row-major triangle ahead of its first row.
// With H rows' operands resident in L2, the columns' are read from memory once
// per super-row.
__device__ __forceinline__ void tri_decode_blocked(uint64_t e, uint64_t n, uint64_t H, uint64_t W,
                                                   uint64_t& row, uint64_t& col) {
    tri_decode(e, n, row, col);
    const uint64_t r0 = row / H * H;
    const uint64_t rem = e - (r0 * n - (r0 ? r0 * (r0 - 1) / 2 : 0));
    const uint64_t h = min(H, n - r0), tri = h * (h + 1) / 2;
    if (rem < tri) {
        tri_decode(rem, h, row, col);
        row += r0;
        col += r0;
    } else {
        const uint64_t r1 = rem - tri, b = r1 / (h * W), r2 = r1 - b * h * W;
        const uint64_t c0 = r0 + H + b * W, w = min(W, n - c0);
        row = r0 + r2 / w;
        col = c0 + r2 % w;
    }
}
// Rows per super-row: 16,384 points, in units of 2 tiles (blocks) and of SB tiles.
constexpr uint64_t kRowPairs = 64, kRowSupers = 2 * kRowPairs / SB, kColPairs = 8;

struct BoxArgs {
    const float *lo, *hi, *slo, *shi;
    uint32_t k;
    float thr;
};

// Surviving super-block pairs (SI <= SJ), appended in warp-aggregated batches.
__global__ void superpairs_kernel(uint64_t nS, BoxArgs b, uint32_t* out, unsigned long long* count) {
    const uint64_t sp = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t nsp = nS * (nS + 1) / 2;
    bool keep = false;
    if (sp < nsp) {
        uint64_t SI, SJ;
        tri_decode_blocked(sp, nS, kRowSupers, 1, SI, SJ);
        keep = !boxes_far(b.slo, b.shi, SI, SJ, b.k, b.thr);
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (!m) return;
    const unsigned lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(count, (unsigned long long)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (keep) out[base + __popc(m & ((1u << lane) - 1u))] = (uint32_t)sp;
}

// One block of SB * SB / 2 threads per surviving super-block pair.  Thread
// (r, pp) tests the tile pairs (I, 2 pp) and (I, 2 pp + 1) of row tile I = SI SB
// + r (column tiles counted from the super-block's first); the up to 16 active
// column tiles of row I are gathered from its 8 threads with two ballots.  Rows
// go together in pairs: the row with the most active tiles left, and the row
// whose tiles it extends the least.
// The column tiles active in either row are paired in ascending order, a block
// per pair (Jb = Ja when the last has one column tile).  On 1M points in 256
// clusters on 8 dimensions this makes 5% fewer blocks than pairing neighbouring
// rows.  count[0] += blocks, count[1] += active tile pairs.
constexpr uint32_t EXPAND_THREADS = SB * SB / 2;
__global__ void __launch_bounds__(EXPAND_THREADS) expand_kernel(const uint32_t* __restrict__ sps,
                                                                uint64_t nTa, uint64_t nS, BoxArgs b,
                                                                uint2* out,
                                                                unsigned long long* count) {
    __shared__ uint64_t sSI, sSJ;
    __shared__ uint32_t rowmask[SB];
    __shared__ uint32_t prow[SB / 2], pmask[SB / 2];  // pairs: r0 | r1 << 8, masks m0 | m1 << 16
    __shared__ uint32_t pbase[SB / 2 + 1];            // their first blocks
    __shared__ unsigned long long sbase;
    if (threadIdx.x == 0) {
        uint64_t SI, SJ;
        tri_decode_blocked(sps[blockIdx.x], nS, kRowSupers, 1, SI, SJ);
        sSI = SI;
        sSJ = SJ;
    }
    __syncthreads();
    const uint32_t pp = threadIdx.x % (SB / 2), r = threadIdx.x / (SB / 2);
    const uint64_t I = sSI * SB + r;
    const uint64_t J0 = sSJ * SB;  // first column tile of the super-block
    uint32_t mask = 0;
    for (uint32_t h = 0; h < 2; ++h) {
        const uint64_t J = J0 + 2 * pp + h;
        bool act = I < nTa && J < nTa && I <= J;
        if (act) act = !boxes_far(b.lo, b.hi, I, J, b.k, b.thr);
        mask |= act ? (1u << h) : 0u;
    }
    // the row's active tiles: 8 lanes of the warp hold 2 bits each
    const unsigned lane = threadIdx.x & 31;
    const unsigned g0 = __ballot_sync(0xffffffffu, mask & 1u), g1 = __ballot_sync(0xffffffffu, mask & 2u);
    const unsigned sh = lane & ~7u;  // first lane of this row's 8
    uint32_t act16 = 0;
#pragma unroll
    for (uint32_t t = 0; t < 8; ++t)
        act16 |= (((g0 >> (sh + t)) & 1u) << (2 * t)) | (((g1 >> (sh + t)) & 1u) << (2 * t + 1));
    if (pp == 0) rowmask[r] = act16;
    __syncthreads();
    if (threadIdx.x < 32) {
        // lane r: row r
        const uint32_t mine = lane < SB ? rowmask[lane] : 0u;
        uint32_t left = mine, base = 0, tiles = __reduce_add_sync(0xffffffffu, __popc(mine));
        for (uint32_t p = 0; p < SB / 2; ++p) {
            // most tiles first, the lowest row of equals
            const uint32_t kx = __reduce_max_sync(0xffffffffu, left ? __popc(left) * 32u + 31u - lane : 0u);
            uint32_t r0 = 0, r1 = 0, m0 = 0, m1 = 0;
            if (kx) {
                r0 = 31u - (kx & 31u);
                m0 = __shfl_sync(0xffffffffu, left, r0);
                if (lane == r0) left = 0;
                const uint32_t ky = __reduce_min_sync(
                    0xffffffffu, left ? (__popc(m0 | left) - __popc(left)) * 32u + lane : 0xffffffffu);
                r1 = r0;
                if (ky != 0xffffffffu) {
                    r1 = ky & 31u;
                    m1 = __shfl_sync(0xffffffffu, left, r1);
                    if (lane == r1) left = 0;
                    if (r1 < r0) {
                        uint32_t t = r0;
                        r0 = r1;
                        r1 = t;
                        t = m0;
                        m0 = m1;
                        m1 = t;
                    }
                }
            }
            if (lane == 0) {
                prow[p] = r0 | (r1 << 8);
                pmask[p] = m0 | (m1 << 16);
                pbase[p] = base;
            }
            base += (__popc(m0 | m1) + 1) / 2;
        }
        if (lane == 0) {
            pbase[SB / 2] = base;
            sbase = base ? atomicAdd(&count[0], (unsigned long long)base) : 0ull;
            if (tiles) atomicAdd(&count[1], (unsigned long long)tiles);
        }
    }
    __syncthreads();
    // thread (p, k): block k of row pair p
    const uint32_t p = threadIdx.x / (SB / 2), k = threadIdx.x % (SB / 2);
    if (p >= SB / 2 || k >= pbase[p + 1] - pbase[p]) return;
    const uint32_t r0 = prow[p] & 255u, di = (prow[p] >> 8) - r0;
    const uint32_t m0 = pmask[p] & 0xffffu, m1 = pmask[p] >> 16;
    uint32_t m = m0 | m1;
    for (uint32_t j = 0; j < 2 * k; ++j) m &= m - 1;  // drop the first 2 k tiles
    const uint32_t ta = __ffs(m) - 1;
    m &= m - 1;
    const bool two = m != 0;
    const uint32_t tb = two ? __ffs(m) - 1 : ta;
    const uint32_t on = ((m0 >> ta) & 1u) | (((m1 >> ta) & 1u) << 2) |
                        (two ? (((m0 >> tb) & 1u) << 1) | (((m1 >> tb) & 1u) << 3) : 0u);
    out[sbase + pbase[p] + k] = make_uint2((uint32_t)(sSI * SB + r0) | (di << 24) | (on << 28),
                                           (uint32_t)(J0 + ta) | ((tb - ta) << 24));
}

// The 256 x 256 block of row pair P (tiles 2 P, 2 P + 1 of nTa) and column pair Q
// (of nTb), all tile pairs active (tri: those with row tile <= column tile).
__device__ __forceinline__ uint2 pair_block(uint64_t P, uint64_t Q, uint64_t nTa, uint64_t nTb,
                                            bool tri) {
    const uint64_t I = 2 * P, J = 2 * Q;
    const bool i1 = I + 1 < nTa, j1 = J + 1 < nTb;
    // (I0, Ja), (I0, Jb), (I1, Ja), (I1, Jb): only (I1, Ja) of a diagonal block is
    // below the triangle
    const uint32_t on = 1u | (j1 ? 2u : 0u) | (i1 && !(tri && P == Q) ? 4u : 0u) | (i1 && j1 ? 8u : 0u);
    return make_uint2((uint32_t)I | (i1 ? 1u << 24 : 0u) | (on << 28),
                      (uint32_t)J | (j1 ? 1u << 24 : 0u));
}

// Work list of a self-join without pruning: the triangle P <= Q of the np pairs of
// row tiles in blocked order.
__global__ void tri_work_kernel(uint64_t nTa, uint64_t total, uint2* out) {
    const uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (e >= total) return;
    uint64_t P, Q;
    tri_decode_blocked(e, (nTa + 1) / 2, kRowPairs, kColPairs, P, Q);
    out[e] = pair_block(P, Q, nTa, nTa, true);
}

// Work list of a join of two point sets (rows: the pairs of A's nTa tiles,
// columns: the pairs of B's nTb tiles), all blocks, in super-blocks of kRowPairs
// row pairs x kColPairs column pairs (row-major inside, super-blocks row-major).
// Closed form: every super-row but the last holds kRowPairs npb entries, every
// super-block but the last of its super-row qh kColPairs entries (qh row pairs in
// the super-row).
__global__ void cross_work_kernel(uint64_t nTa, uint64_t nTb, uint64_t total, uint2* out) {
    const uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (e >= total) return;
    const uint64_t npa = (nTa + 1) / 2, npb = (nTb + 1) / 2;
    const uint64_t SI = e / (kRowPairs * npb), rem = e - SI * kRowPairs * npb;
    const uint64_t qh = min(kRowPairs, npa - SI * kRowPairs);
    const uint64_t SP = rem / (qh * kColPairs), rem2 = rem - SP * qh * kColPairs;
    const uint64_t pw = min(kColPairs, npb - SP * kColPairs);
    out[e] = pair_block(SI * kRowPairs + rem2 / pw, SP * kColPairs + rem2 % pw, nTa, nTb, false);
}

// Band records -> pairs: a thread per record; block-level exclusive scan of
// the popcounts, one global reservation per block.
constexpr uint32_t EXPAND_BAND_THREADS = 256;
__global__ void __launch_bounds__(EXPAND_BAND_THREADS) band_expand_kernel(
    const BandRec* __restrict__ rec, uint64_t nrec, BandPair* out, uint64_t cap,
    unsigned long long* cursor) {
    using Scan = cub::BlockScan<uint32_t, EXPAND_BAND_THREADS>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ unsigned long long sbase;
    const uint64_t e = blockIdx.x * (uint64_t)EXPAND_BAND_THREADS + threadIdx.x;
    BandRec r{0, 0, 0, 0};
    if (e < nrec) r = rec[e];
    const uint32_t cnt = __popc(r.mask);
    uint32_t off = 0, total = 0;
    Scan(tmp).ExclusiveSum(cnt, off, total);
    if (threadIdx.x == 0) sbase = total ? atomicAdd(cursor, (unsigned long long)total) : 0ull;
    __syncthreads();
    uint64_t o = sbase + off;
    uint32_t m = r.mask;
    const uint32_t flag = r.j0 & kBandBoth, j0 = r.j0 & ~kBandBoth;
    while (m) {
        const uint32_t c = __ffs(m) - 1;
        m &= m - 1;
        if (o < cap) out[o] = BandPair{r.i, (j0 + c) | flag};
        ++o;
    }
}

__global__ void sum_counts_kernel(const int32_t* counts, uint64_t n, unsigned long long* total) {
    unsigned long long s = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        s += (unsigned long long)(uint32_t)counts[i];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(total, s);
}

__global__ void scatter_counts_kernel(const int32_t* src, const uint32_t* perm, uint64_t n,
                                      int32_t* dst) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < n) dst[perm[i]] = src[i];
}

}  // namespace

// With boxes: super-block pairs first (one thread each), then the blocks of the
// survivors (one thread block each).  Without: all blocks at once, their number
// known (no read-back: with the survivors' kernels and their sort this list took
// 65 us of a call, now one launch).  nT: row tiles (even); nTa: tiles holding data
// rows.
int build_worklist(uint64_t nT, uint64_t nTa, const LearnedBoxes* boxes, float thr, WorkList& out,
                   cudaStream_t s) {
    out.n = out.tiles = 0;
    if (nT == 0) return EJOIN_OK;
    if (nT % 2 || nTa > nT || nT > 0xffffffull) return set_error(EJOIN_EINTERNAL, "work list: bad tile count");
    const uint64_t nS = (nT + SB - 1) / SB;
    const uint64_t nsp = nS * (nS + 1) / 2;
    if (nsp > 0xffffffffull) return set_error(EJOIN_EUNSUPPORTED, "work list too large");
    if (!boxes) {
        const uint64_t np = (nTa + 1) / 2;
        out.n = np * (np + 1) / 2;
        out.tiles = nTa * (nTa + 1) / 2;
        if (out.n == 0) return EJOIN_OK;
        if ((out.n + 255) / 256 > 0x7fffffffull) return set_error(EJOIN_EUNSUPPORTED, "work list too large");
        EJ_TRY(out.e.alloc(out.n, s, "work list"));
        tri_work_kernel<<<(unsigned)((out.n + 255) / 256), 256, 0, s>>>(nTa, out.n, out.e.p);
        EJ_CUDA(cudaGetLastError());
        note_launch();
        return EJOIN_OK;
    }
    const BoxArgs b{boxes->lo.p, boxes->hi.p, boxes->slo.p, boxes->shi.p, boxes->k, thr};
    DBuf<uint32_t> sps;
    DBuf<unsigned long long> cnt;
    EJ_TRY(sps.alloc(nsp, s, "super-block pairs"));
    EJ_TRY(cnt.alloc(3, s, "work-list counters"));
    EJ_TRY(cnt.zero(s));
    superpairs_kernel<<<(unsigned)((nsp + 255) / 256), 256, 0, s>>>(nS, b, sps.p, cnt.p);
    EJ_CUDA(cudaGetLastError());
    note_launch();
    unsigned long long nkeep = 0;
    EJ_CUDA(cudaMemcpyAsync(&nkeep, cnt.p, sizeof nkeep, cudaMemcpyDeviceToHost, s));
    EJ_CUDA(cudaStreamSynchronize(s));
    // (a super-block pair makes at most 8 x 8 blocks)
    EJ_TRY(out.e.alloc(nkeep ? nkeep * (SB * SB / 4) : 1, s, "work list"));
    if (nkeep) {
        if (nkeep > 0x7fffffffull) return set_error(EJOIN_EUNSUPPORTED, "work list too large");
        // back into blocked order: consecutive work then shares row blocks
        DBuf<uint32_t> sorted;
        EJ_TRY(sorted.alloc(nkeep, s, "sorted super-block pairs"));
        size_t tb = 0;
        EJ_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tb, sps.p, sorted.p, (int)nkeep, 0, 32, s));
        DBuf<uint8_t> tmp;
        EJ_TRY(tmp.alloc(tb, s, "sort scratch"));
        EJ_CUDA(cub::DeviceRadixSort::SortKeys(tmp.p, tb, sps.p, sorted.p, (int)nkeep, 0, 32, s));
        note_launch(4);
        expand_kernel<<<(unsigned)nkeep, EXPAND_THREADS, 0, s>>>(sorted.p, nTa, nS, b, out.e.p,
                                                                 cnt.p + 1);
        EJ_CUDA(cudaGetLastError());
        note_launch();
    }
    unsigned long long tot[2] = {0, 0};
    EJ_CUDA(cudaMemcpyAsync(tot, cnt.p + 1, sizeof tot, cudaMemcpyDeviceToHost, s));
    EJ_CUDA(cudaStreamSynchronize(s));
    out.n = tot[0];
    out.tiles = tot[1];
    return EJOIN_OK;
}

int launch_band_expand(const BandRec* rec, uint64_t nrec, BandPair* out, uint64_t cap,
                       cudaStream_t s) {
    if (nrec == 0) return EJOIN_OK;
    DBuf<unsigned long long> cur;
    EJ_TRY(cur.alloc(1, s, "band cursor"));
    EJ_TRY(cur.zero(s));
    band_expand_kernel<<<(unsigned)((nrec + EXPAND_BAND_THREADS - 1) / EXPAND_BAND_THREADS),
                         EXPAND_BAND_THREADS, 0, s>>>(rec, nrec, out, cap, cur.p);
    EJ_CUDA(cudaGetLastError());
    note_launch();
    return EJOIN_OK;
}

int build_worklist_cross(uint64_t nTa, uint64_t nTb, WorkList& out, cudaStream_t s) {
    out.n = (nTa + 1) / 2 * ((nTb + 1) / 2);
    out.tiles = nTa * nTb;
    if (out.n == 0) return EJOIN_OK;
    EJ_TRY(out.e.alloc(out.n, s, "work list"));
    cross_work_kernel<<<(unsigned)((out.n + 255) / 256), 256, 0, s>>>(nTa, nTb, out.n, out.e.p);
    EJ_CUDA(cudaGetLastError());
    note_launch();
    return EJOIN_OK;
}

// One entry of every `stride` consecutive ones of a work list, at a place that a hash
// of the stride's number picks (the same for the same list).  Always the first entry
// would see the same few rows and one column pair in kColPairs of every super-row:
// the blocked order repeats every kRowPairs x kColPairs entries, a multiple of most
// strides.  (150,016 points in batches of 2,048, the first 256 of each far from
// everything: the first entries saw none of 9.3 M records.)
__global__ void sample_work_kernel(const uint2* __restrict__ work, uint64_t nwork,
                                   uint64_t nsample, uint32_t stride, uint2* __restrict__ out) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= nsample) return;
    // (a multiply-shift hash: any odd constant with mixed bits)
    uint32_t h = (uint32_t)i * 0x9E3779B1u;
    h = (h ^ (h >> 15)) * 0x2C1B3C6Du;
    h ^= h >> 13;
    out[i] = work[min(i * stride + __umulhi(h, stride), nwork - 1)];
}

int sample_worklist(const uint2* work, uint64_t nwork, uint32_t stride, DBuf<uint2>& out,
                    uint64_t* nsample_out, cudaStream_t s) {
    const uint64_t ns = stride ? (nwork + stride - 1) / stride : 0;
    *nsample_out = ns;
    if (ns == 0) return EJOIN_OK;
    EJ_TRY(out.alloc(ns, s, "sampled work list"));
    sample_work_kernel<<<(unsigned)((ns + 255) / 256), 256, 0, s>>>(work, nwork, ns, stride, out.p);
    EJ_CUDA(cudaGetLastError());
    note_launch();
    return EJOIN_OK;
}

int sum_counts(const int32_t* counts, uint64_t n, unsigned long long* dev_total, cudaStream_t s) {
    if (n == 0) return EJOIN_OK;
    uint64_t blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    sum_counts_kernel<<<(unsigned)blocks, 256, 0, s>>>(counts, n, dev_total);
    EJ_CUDA(cudaGetLastError());
    note_launch();
    return EJOIN_OK;
}

int scatter_counts(const int32_t* src, const uint32_t* perm, uint64_t n, int32_t* dst,
                   cudaStream_t s) {
    if (n == 0) return EJOIN_OK;
    scatter_counts_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, perm, n, dst);
    EJ_CUDA(cudaGetLastError());
    note_launch();
    return EJOIN_OK;
}

}  // namespace ejoin
