// k_umma.cu -- the tcgen05 Gram screen (EJOIN_BF16 / BF16_SPLIT / FP16 / FP8_E4M3).
//
// Re-designs the reference's main tensor path,
// distanceCalculationBruteForceTensorHalf (kernel_join.cu:328-524): there a
// warp computes -2*Q*C^T + |c|^2 for 16 queries x 16 candidates per wmma
// m16n16k16, round-trips every k-chunk through shared memory, re-adds the
// query norms in scalar code and bumps one global counter per hit with
// sqrt(|d2|) <= eps.  Here:
//
//  * A persistent pair of CTAs (a cluster of two, one CTA per SM) walks a list
//    of blocks of 256 rows (row tiles I0, I1, one per CTA) x 256 columns (column
//    tiles Ja, Jb), taking runs of consecutive list entries.  Neither pair of
//    tiles need be adjacent.  Each of the four 128x128 tile pairs carries an
//    "active" bit: it lies in the upper triangle (J >= I) and was not pruned;
//    an inactive one is computed but ignored.
//  * The pair shares each MMA (tcgen05 cta_group::2, M = N = 256, K = 16 per
//    instruction): a CTA stages its own 128 rows of A and half of B, and its
//    tensor memory receives its own rows.  With one CTA per MMA (M = 128) a CTA
//    staged all 256 rows of B: 48 KB per K-slab instead of 32 KB through the
//    SM's 64 bytes per clock from L2, and 12 instead of 8 KB of shared memory
//    read per MMA -- 1M x 128 FP16 was bound by that stream (109 ms for the
//    launch, 95 ms with pairs at the clock that the power limit leaves; 2M pairs
//    of tiles of 500k x 256 BF16 hi+lo 111 and 102 ms).
//  * Warp 0 of each CTA streams its K-slabs into a 4-stage ring with TMA
//    (128-byte swizzle; three stages are too few: 4M x 64 pruned took 17.2
//    instead of 13.2 ms).  One lane of warp 1 of rank 0 issues the MMAs into one
//    of two 128x256 FP32 accumulators per CTA, so the next block's MMAs run
//    while 16 epilogue warps read the previous one.
//  * Operand rows are [hi | lo] (k_prep.cu) with separate aug tiles of 16
//    elements per row (stored in the order that the 32-byte swizzle wants).
//    With the hi+lo split the MMAs form hi*hi + hi*lo + lo*hi.  The aug MMA adds
//    -alpha_i - alpha_j, so the accumulator holds C_ij = q_i.q_j - alpha_i -
//    alpha_j and the rigorous screen is a sign test:
//        C >= 0          pair certainly within eps        (counted)
//        C < -W_iK       pair certainly outside eps
//        otherwise       band: queued for the FP64 recheck
//    W_iK = beta_i + max beta over the 32-column chunk K >= beta_i + beta_j
//    (one value per row and column chunk, so the test costs one add per
//    element, like a tile-wide width, with a narrower band).
//  * Each epilogue warp reads its two 32x32 chunks one after the other with
//    tcgen05.ld.red (the load also returns each lane's maximum: the rows whose
//    maximum + W is negative are certainly out).  The few rows left are put down
//    in shared memory and counted later, while the warp waits for an
//    accumulator; a chunk with many of them has its sign bits packed (one funnel
//    shift per element) and its columns counted by a 32x32 bit transpose.  Row
//    and column counts are reductions to global memory (off-diagonal tiles
//    credit both points), band records go to queue space of the warp's own.  No
//    distance reaches global memory.
//  * What bounds it (cycles per block, MMA time / bare pipeline / with the
//    tensor-memory loads / all): 1M x 128 FP16 1152 / 1199 / 1526 / 1566; 250k x
//    1024 E4M3 4224 / 4480 / 4502 / 4540; 4M x 64 pruned BF16 hi+lo 1664 / 1725 /
//    1757 / 2322 (blocks with many hits hold up one warp of 32); 150k x 64 FP16
//    640 / 827 / 1310 / 1740.  Long launches also meet the power limit (1.65 to
//    1.75 of 2.07 GHz).
//
// Every wait is bounded (umma_ptx.cuh); on expiry all roles stop, in-flight
// copies and MMAs are drained (bounded) and tensor memory is freed.
#include <algorithm>

#include "tmap.cuh"
#include "umma_ptx.cuh"

namespace ejoin {
namespace {

// Shared memory of a CTA.  A stage holds one K-slab: this CTA's 128 of the
// pair's 256 rows of A and 128 of its 256 rows of B (128 bytes each), and space
// for the aug tiles of A and B, which come with a block's last slab.  Every
// part starts on a 1024-byte boundary.
constexpr int SLAB = 128 * 128;  // 128 rows x 128 bytes
constexpr int AUG = 128 * 32;    // 128 rows x 32 bytes (16 elements)
constexpr int STAGE_BYTES = 2 * SLAB + 2 * AUG;
constexpr int NST = 4;
constexpr size_t RING_BYTES = (size_t)NST * STAGE_BYTES;
constexpr int NUM_EPI_WARPS = 16;          // 4 per SM sub-partition (latency hiding)
constexpr int NTHREADS = (2 + NUM_EPI_WARPS) * 32;
constexpr uint32_t ACC_COLS = 256;         // one 128x256 FP32 accumulator
constexpr uint32_t TMEM_COLS = 2 * ACC_COLS;
constexpr uint32_t FULL = 0xffffffffu;
// Rows of hits an epilogue warp can put down (put_rows): HROWS of HROW_PITCH
// floats; a chunk with more than HCHUNK of them is classified by bit masks.
constexpr uint32_t HROWS = 24, HCHUNK = 12, HROW_PITCH = 36;
constexpr uint32_t HIT_FLOATS = HROWS * HROW_PITCH;  // per warp

// Work-list entry: x = I0 | (I1 - I0) << 24 | active mask << 28, y = Ja | (Jb -
// Ja) << 24.  CTA r of the pair has row tile I_r; half 0 of its block is column
// tile Ja, half 1 is Jb; mask bit 2 r + h: half h of CTA r's block is counted.
__device__ __forceinline__ uint32_t e_row(uint2 e, uint32_t r) {
    return (e.x & 0xffffffu) + (r ? (e.x >> 24) & 15u : 0u);
}
__device__ __forceinline__ uint32_t e_on(uint2 e, uint32_t r, uint32_t h) {
    return (e.x >> (28u + 2u * r + h)) & 1u;
}
__device__ __forceinline__ uint32_t e_col(uint2 e, uint32_t h) {
    const uint32_t ja = e.y & 0xffffffu;
    return h ? ja + (e.y >> 24) : ja;
}

struct GramArgs {
    const uint2* work;
    uint64_t nwork;
    const float* cmax;  // per 32-row chunk of B: max beta
    const float* beta;  // per row: beta (out margin, Gram units)
    const float* tsig;  // FP8: per-tile minimum row scale (null for 16-bit operands)
    const float* sig;   // FP8: per-row scale
    int32_t* counts;
    BandRec* band;
    uint64_t band_cap;
    DevStatus* st;
    uint32_t nhi;    // data slabs (128-byte rows) per part
    uint32_t fmt;    // 16-bit operands: 0 = FP16, 1 = BF16 (instruction-descriptor format)
    uint32_t lrun;   // log2 of the run length: entries a CTA takes consecutively
    uint32_t cross;  // rows of A against a different set B: count rows only
    Emit em;         // neighbour-list emission (em.cnt null: counts only)
};

__device__ __forceinline__ uint2 entry_or_end(const GramArgs& a, uint64_t u) {
    return u < a.nwork ? __ldg(&a.work[u]) : make_uint2(0xffffffffu, 0xffffffffu);
}

// The work-list entries of this CTA pair: runs of 2^lrun consecutive entries,
// runs dealt round-robin (so the pairs running at the same time stay within a
// window of the list that shares operand rows in L2).
__device__ __forceinline__ uint64_t first_item(uint32_t lrun) {
    return (uint64_t)(blockIdx.x / 2) << lrun;
}
__device__ __forceinline__ uint64_t next_item(uint64_t u, uint32_t lrun) {
    ++u;
    if ((u & ((1ull << lrun) - 1ull)) == 0) u += (uint64_t)(gridDim.x / 2 - 1) << lrun;
    return u;
}

struct Ctl {
    uint64_t full[NST], empty[NST];
    uint64_t tfull[2], tempty[2];
    uint64_t fin;
    uint32_t tmem_base;
};

constexpr size_t SMEM_BYTES =
    1024 + RING_BYTES + (size_t)NUM_EPI_WARPS * HIT_FLOATS * sizeof(float) + sizeof(Ctl);
static_assert(SMEM_BYTES <= 232448, "shared memory budget");

// 32x32 bit-matrix transpose across the warp: lane r holds row r (bit c =
// column c); afterwards lane c holds column c (bit r = row r).
__device__ __forceinline__ uint32_t transpose32(uint32_t x, uint32_t lane) {
    const uint32_t masks[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
    uint32_t j = 16;
#pragma unroll
    for (int l = 0; l < 5; ++l, j >>= 1) {
        const uint32_t m = masks[l];
        const uint32_t y = __shfl_xor_sync(FULL, x, j);
        x = (lane & j) ? (((y >> j) & m) | (x & ~m)) : ((x & m) | ((y & m) << j));
    }
    return x;
}

// Element offset of K-slab `step` of a block: [hi0, lo0, hi1, lo1, ...] with
// the split, [hi0, hi1, ...] without.
template <int OPK>
__device__ __forceinline__ uint32_t slab_x(uint32_t step, uint32_t nhi, uint32_t split) {
    constexpr uint32_t E = OPK ? 128u : 64u;  // elements per 128-byte slab row
    if (split) return (step & 1) ? E * nhi + E * (step >> 1) : E * (step >> 1);
    return E * step;
}

// Column counts of one 32 x 32 in-mask (lane = row), added to the counts of
// the chunk's 32 columns in global memory (reductions without a result, which
// the warp does not wait for): sparse masks (at most 3 bits per lane) add per
// bit, denser ones transpose the bit block across the warp and add one count
// per column.
__device__ __forceinline__ void col_counts(uint32_t inm, int32_t* cnt, uint32_t lane) {
    const uint32_t mp = __reduce_max_sync(FULL, __popc(inm));
    if (mp == 0) return;
    if (mp <= 3) {
        uint32_t m = inm;
        while (m) {
            const uint32_t c = __ffs(m) - 1;
            m &= m - 1;
            atomicAdd(&cnt[c], 1);
        }
    } else {
        const int cc = __popc(transpose32(inm, lane));
        if (cc) atomicAdd(&cnt[lane], cc);
    }
}

// In / band bit masks of one 32 x 32 chunk (lane = row, v[c] = column c).
__device__ __forceinline__ void classify(const uint32_t (&v)[32], float W, uint32_t& inm,
                                         uint32_t& bandm) {
    // sign bits, four independent 8-column chains
    uint32_t ng[4] = {0, 0, 0, 0}, nw[4] = {0, 0, 0, 0};
#pragma unroll
    for (int c = 7; c >= 0; --c)
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const uint32_t x = v[8 * g + c];
            ng[g] = __funnelshift_l(x, ng[g], 1);
            nw[g] = __funnelshift_l(__float_as_uint(__uint_as_float(x) + W), nw[g], 1);
        }
    const uint32_t neg = ng[0] | (ng[1] << 8) | (ng[2] << 16) | (ng[3] << 24);
    const uint32_t negw = nw[0] | (nw[1] << 8) | (nw[2] << 16) | (nw[3] << 24);
    inm = ~neg;
    bandm = neg & ~negw;
}

// Space of one epilogue warp in a record queue: kResChunk records at a time, so
// that one returning global atomic serves many blocks.  base / left: the unused
// part of the current chunk.
constexpr uint32_t kResChunk = 128;
struct QueueSpace {
    unsigned long long base = 0;
    uint32_t left = 0;
};

// A record (row, col, mask) from every lane with mask != 0 (at most 32: ranks
// from a ballot); the first `left` of them fill the current chunk, the rest
// start a new one.  Returns the number of records.
static_assert(kResChunk >= 32, "the records of one call fit one new chunk");
__device__ __forceinline__ uint32_t put_records(BandRec* q, uint64_t cap,
                                                unsigned long long* reserved, QueueSpace& sp,
                                                uint32_t mask, uint32_t row, uint32_t col,
                                                uint32_t lane) {
    const uint32_t b = __ballot_sync(FULL, mask != 0), n = __popc(b);
    if (n == 0) return 0;
    unsigned long long nbase = 0;
    const bool grow = n > sp.left;
    if (grow) {
        if (lane == 0) nbase = atomicAdd(reserved, (unsigned long long)kResChunk);
        nbase = __shfl_sync(FULL, nbase, 0);
    }
    if (mask) {
        const uint32_t e = __popc(b & ((1u << lane) - 1u));
        const unsigned long long g = e < sp.left ? sp.base + e : nbase + (e - sp.left);
        if (g < cap) q[g] = BandRec{row, col, mask, 0u};
    }
    if (grow) {
        sp.base = nbase + (n - sp.left);
        sp.left = kResChunk - (n - sp.left);
    } else {
        sp.base += n;
        sp.left -= n;
    }
    return n;
}

// Empty records (mask 0, no pairs) in the unused tail of the space.
__device__ __forceinline__ void pad_records(BandRec* q, uint64_t cap, const QueueSpace& sp,
                                            uint32_t lane) {
    for (uint32_t e = lane; e < sp.left; e += 32)
        if (sp.base + e < cap) q[sp.base + e] = BandRec{0u, 0u, 0u, 0u};
}

// OPK 0: 16-bit operands, data MMAs kind::f16; OPK 1: E4M3 operands, data
// MMAs kind::f8f6f4 (K = 32 per instruction, same 32-byte k-steps), the aug
// MMA stays kind::f16 in BF16 and accumulates into the same tensor memory.
template <int OPK, bool SPLIT>
__global__ void __launch_bounds__(NTHREADS, 1)
    gram_kernel(const __grid_constant__ CUtensorMap tqa, const __grid_constant__ CUtensorMap tqb,
                const __grid_constant__ CUtensorMap taa, const __grid_constant__ CUtensorMap tab,
                const GramArgs a) {
    extern __shared__ uint8_t smraw[];
    uint8_t* stages = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
    // after the ring: the epilogue warps' hit rows, then the control block
    float* hits = reinterpret_cast<float*>(stages + RING_BYTES);
    Ctl& S = *reinterpret_cast<Ctl*>(hits + NUM_EPI_WARPS * HIT_FLOATS);
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    const uint32_t rank = ptx::cluster_ctarank();

    if (warp == 1) {
        ptx::tmem_alloc<2>(&S.tmem_base, TMEM_COLS);
        ptx::tmem_relinquish<2>();
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; ++s) {
            ptx::mbar_init(&S.full[s], 1);
            ptx::mbar_init(&S.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(&S.tfull[b], 1);
            ptx::mbar_init(&S.tempty[b], 2 * NUM_EPI_WARPS);
        }
        ptx::mbar_init(&S.fin, 1);
        ptx::fence_barrier_init();
        ptx::tma_prefetch_desc(&tqa);
        ptx::tma_prefetch_desc(&tqb);
        ptx::tma_prefetch_desc(&taa);
        ptx::tma_prefetch_desc(&tab);
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync();  // the pair's barriers are ready
    ptx::tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    const uint32_t nsteps = a.nhi * (SPLIT ? 2u : 1u);

    if (warp == 0) {
        // ------------------------------------------------ TMA producer
        // Each CTA loads its own halves of A and B; both CTAs' copies complete
        // on rank 0's barriers, where the MMAs are issued.
        if (lane == 0) {
            const uint32_t full0 = ptx::mapa(&S.full[0], 0);
            uint32_t st = 0, ph = 0;
            uint32_t issued_ph = 0;  // bit s: phase of stage s's last copy
            uint32_t issued = 0;     // bit s: stage s had a copy
            bool ok = true;
            // test hook (DevStatus::withhold = w > 0): the w-th stage is never
            // issued, so the waits on it expire; the producer stops before its
            // place in the ring comes round again, so the drain below never
            // waits for it
            uint32_t withhold = *(volatile unsigned*)&a.st->withhold;
            // entries are read one block ahead (their latency hides behind a block)
            uint64_t u = first_item(a.lrun);
            uint2 wnext = entry_or_end(a, u);
            while (ok && u < a.nwork) {
                const uint2 w = wnext;
                u = next_item(u, a.lrun);
                wnext = entry_or_end(a, u);
                // row tile of this CTA; its half of B is column tile Ja (rank 0) or Jb
                const uint32_t ta = e_row(w, rank), tb = e_col(w, rank);
                for (uint32_t step = 0; step < nsteps; ++step) {
                    if (!ptx::mbar_wait(&S.empty[st], ph ^ 1u, a.st, 10)) {
                        ok = false;
                        break;
                    }
                    uint8_t* sa = stages + (size_t)st * STAGE_BYTES;
                    const int32_t x = (int32_t)slab_x<OPK>(step, a.nhi, SPLIT);
                    const bool aug = step + 1 == nsteps;
                    if (withhold == 0 || --withhold != 0) {
                        const uint32_t bar = full0 + 8u * st;
                        if (rank == 0)
                            ptx::mbar_arrive_expect_tx(&S.full[st],
                                                       aug ? 2 * STAGE_BYTES : 4 * SLAB);
                        ptx::tma_load_2d_pair(sa, &tqa, x, (int32_t)(ta * 128u), bar);
                        ptx::tma_load_2d_pair(sa + SLAB, &tqb, x, (int32_t)(tb * 128u), bar);
                        if (aug) {
                            // 32 rows of 128 bytes each (store_aug)
                            ptx::tma_load_2d_pair(sa + 2 * SLAB, &taa, 0, (int32_t)(ta * 64u), bar);
                            ptx::tma_load_2d_pair(sa + 2 * SLAB + AUG, &tab, 0,
                                                  (int32_t)(tb * 64u + 32u), bar);
                        }
                        issued_ph = (issued_ph & ~(1u << st)) | (ph << st);
                        issued |= 1u << st;
                    }
                    if (++st == NST) {
                        st = 0;
                        ph ^= 1u;
                    }
                }
            }
            // drain: every issued copy has landed before the CTA can exit (the
            // pair leaves together, so rank 0, whose barriers take both CTAs'
            // copies, waits for both).  When the two CTAs gave up at different
            // places, rank 1 may have copies that rank 0 does not wait for:
            // it allows them 1 ms.
            for (uint32_t s = 0; s < NST && (rank == 0 || ok); ++s) {
                if (!((issued >> s) & 1u)) continue;
                const uint32_t sph = (issued_ph >> s) & 1u;
                // (rank 1: the arrivals of rank 0's commits have come, none is
                // still on its way; none will come once a role has given up)
                if (rank == 0) ptx::mbar_wait_drain(&S.full[s], sph);
                else ok = ptx::mbar_wait(&S.empty[s], sph, a.st, 12);
            }
            if (rank != 0 && !ok) ptx::pause_ns(1000000);
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        // The whole warp runs the loop and one elected lane issues; what it
        // issues per slab is straight-line code (run-time loops and branches in
        // the elected lane's code made an MMA cost 98 cycles and a commit 95,
        // where the MMA itself takes the tensor pipe 128: blocks of 5 or 9 MMAs
        // were bound by their issue).  For the same reason a block has few
        // waits: the aug tiles come with the last slab, and the accumulator is
        // waited for together with the first.
        if (rank == 0) {
            const uint32_t idesc = OPK ? ptx::idesc_f32acc(0, 0, 256, ACC_COLS)
                                       : ptx::idesc_f32acc(a.fmt, a.fmt, 256, ACC_COLS);
            const uint32_t idesc_aug = OPK ? ptx::idesc_f32acc(1, 1, 256, ACC_COLS) : idesc;
            auto mma = [&](uint32_t d, uint64_t ad, uint64_t bd, uint32_t acc_) {
                if (OPK) ptx::mma_f8<2>(d, ad, bd, idesc, acc_);
                else ptx::mma_f16<2>(d, ad, bd, idesc, acc_);
            };
            const uint64_t desc0 = ptx::sdesc_sw128(ptx::smem_u32(stages));
            const uint64_t gdesc0 = ptx::sdesc_sw32(ptx::smem_u32(stages + 2 * SLAB));
            uint32_t st = 0, ph = 0, it = 0;
            auto advance = [&]() {
                if (++st == NST) {
                    st = 0;
                    ph ^= 1u;
                }
            };
            // Order by magnitude (the accumulation bound of screen_params in
            // api.cu relies on it): the first slab's hi*lo and lo*hi products,
            // then the hi*hi ones, then the later slabs, and the aug step
            // (-alpha_i - alpha_j) last.
            auto slab = [&](uint32_t d_tmem, uint32_t s_hi, uint32_t s_lo, uint32_t acc) {
                const uint64_t ah = desc0 + (uint64_t)(s_hi * (STAGE_BYTES >> 4));
                const uint64_t bh = ah + (SLAB >> 4);
                if (SPLIT) {
                    const uint64_t al = desc0 + (uint64_t)(s_lo * (STAGE_BYTES >> 4));
                    const uint64_t bl = al + (SLAB >> 4);
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; ++kk) {
                        mma(d_tmem, ah + 2 * kk, bl + 2 * kk, kk ? 1u : acc);
                        mma(d_tmem, al + 2 * kk, bh + 2 * kk, 1);
                    }
                }
#pragma unroll
                for (uint32_t kk = 0; kk < 4; ++kk)
                    mma(d_tmem, ah + 2 * kk, bh + 2 * kk, SPLIT || kk ? 1u : acc);
            };
            for (uint64_t u = first_item(a.lrun); u < a.nwork; u = next_item(u, a.lrun), ++it) {
                const uint32_t b = it & 1u, use = it >> 1;
                const uint32_t d_tmem = tmem + b * ACC_COLS;
                // (every wait ends in a vote: lanes of which one gave up while another
                // saw the phase complete must not part ahead of elect_one)
                uint32_t s_hi, s_lo;
                auto take = [&](bool free) {
                    bool got = free && ptx::mbar_wait(&S.full[st], ph, a.st, 20);
                    s_hi = s_lo = st;
                    advance();
                    if (SPLIT) {
                        got = got && ptx::mbar_wait(&S.full[st], ph, a.st, 20);
                        s_lo = st;
                        advance();
                    }
                    return __all_sync(FULL, got) != 0;
                };
                bool ok = take(ptx::mbar_wait(&S.tempty[b], (use & 1u) ^ 1u, a.st, 21));
                for (uint32_t c = 1; ok && c < a.nhi; ++c) {
                    ptx::tc_fence_after();
                    if (ptx::elect_one()) {
                        slab(d_tmem, s_hi, s_lo, c > 1);
                        ptx::mma_commit<2>(&S.empty[s_hi]);
                        if (SPLIT) ptx::mma_commit<2>(&S.empty[s_lo]);
                    }
                    __syncwarp();
                    ok = take(true);
                }
                if (!ok) break;
                ptx::tc_fence_after();
                if (ptx::elect_one()) {
                    slab(d_tmem, s_hi, s_lo, a.nhi > 1);
                    // aug: A side (alpha_i, -1) x B side (-1, alpha_j), one K = 16 step
                    const uint64_t ag = gdesc0 + (uint64_t)(s_lo * (STAGE_BYTES >> 4));
                    ptx::mma_f16<2>(d_tmem, ag, ag + (AUG >> 4), idesc_aug, 1);
                    ptx::mma_commit<2>(&S.tfull[b]);
                    ptx::mma_commit<2>(&S.empty[s_hi]);
                    if (SPLIT) ptx::mma_commit<2>(&S.empty[s_lo]);
                }
                __syncwarp();
            }
            if (ptx::elect_one()) ptx::mma_commit<2>(&S.fin);
            __syncwarp();
        }
        // drain (both CTAs): all MMAs and the arrivals of their commits are
        // complete before tensor memory is freed
        ptx::mbar_wait_drain(&S.fin, 0);
    } else {
        // ------------------------------------------------ epilogue warps
        // warp e reads lane quarter (warp % 4) and the 64 columns 64 * (e / 4),
        // which lie in half h = e / 8 (column tile Ja or Jb); the CTA's own rows
        // (row tile I of its rank) are in its own tensor memory
        const uint32_t ew = warp - 2;          // 0..15
        const uint32_t q = warp & 3u;          // tensor-memory lane quarter
        const uint32_t cg = ew >> 2;           // 64-column group
        const uint32_t h = cg >> 1;            // half
        const uint32_t lt = (1u << lane) - 1u;
        float* hit = hits + ew * HIT_FLOATS;
        const uint32_t tempty0 = ptx::mapa(&S.tempty[0], 0);  // rank 0's barriers
        uint32_t it = 0;
        // band width of row i against a 32-column chunk K of column tile J:
        // W >= beta_i + max beta over K >= beta_i + beta_j for every j in K
        // (Gram units; FP8 operands: divided by sigma_i sigma_J,min, the
        // accumulator's unit for pair (i, j) being 1 / (sigma_i sigma_j)); the
        // sum is rounded up by the 2^-20 relative margin, division by the
        // power-of-two scales is exact.  0 for an inactive half.
        // Latency: entries are read two blocks ahead and the raw margins one
        // block ahead, both consumed a block later, so no global-load latency
        // lands on a block's own path.
        struct Margins {
            float b, t0, t1, sr, st;
        };
        auto is_active = [&](uint2 e) { return e.x != 0xffffffffu && e_on(e, rank, h); };
        auto load_margins = [&](uint2 e) -> Margins {
            Margins m{0.0f, 0.0f, 0.0f, 1.0f, 1.0f};
            if (is_active(e)) {
                const uint32_t Je = e_col(e, h);
                const uint32_t r = e_row(e, rank) * 128u + q * 32u + lane;
                // the warp's two 32-column chunks (an even chunk index)
                const float2 t = __ldg(reinterpret_cast<const float2*>(a.cmax) + Je * 2u + (cg & 1u));
                m.b = __ldg(&a.beta[r]);
                m.t0 = t.x;
                m.t1 = t.y;
                if (OPK) {
                    m.sr = __ldg(&a.sig[r]);
                    m.st = __ldg(&a.tsig[Je]);
                }
            }
            return m;
        };
        auto width = [&](const Margins& m, float t) -> float {
            const float sm = m.b + t;
            float Wv = fmaf(fabsf(sm), 9.5367431640625e-07f, sm);
            if (OPK) Wv = Wv / (m.sr * m.st);
            return Wv;
        };
        uint64_t u = first_item(a.lrun);
        uint64_t un = next_item(u, a.lrun);
        uint2 w = entry_or_end(a, u);
        uint2 wn = entry_or_end(a, un);
        Margins mc = load_margins(w);
        float W0 = width(mc, mc.t0), W1 = width(mc, mc.t1);
        // Per block: wait for the accumulator, load the two 32-column chunks
        // (one at a time, 32 live values) and put down the rows that can hold an
        // in or band pair (the lane's maximum + W >= 0), release the
        // accumulator.  On most data such rows are few, and they are counted
        // later, four at a time with eight lanes per row, while the warp waits
        // for an accumulator: neither a busy block's counting nor the packing of
        // the sign bits of 1024 pairs for a handful of hits holds the MMAs up.
        // A chunk with more than HCHUNK such rows is classified by bit masks.
        //
        // Counts and band records leave the warp without any cross-warp step:
        // counts are reductions to global memory (dense chunks: a lane keeps its
        // row's count in a register while consecutive blocks share the row
        // tile), and band records go to queue space the warp reserved.
        uint32_t v[32];
        float mx = 0.0f;
        const uint32_t tq = tmem + ((q * 32u) << 16) + cg * 64u;
        QueueSpace bsp, esp;
        unsigned long long npairs = 0;  // band pairs of this lane's records
        uint32_t nrecs = 0, nin = 0;    // the warp's band and in-records
        int rowcnt = 0;                 // in-pairs of this lane's row in row tile I (dense chunks)
        uint32_t I = e_row(w, rank);
        // ring of rows put down: slots tail, tail + 1, ... hold npend rows of 32
        // accumulators, W, the row and the first column (| kBandBoth)
        uint32_t tail = 0, npend = 0;
        auto put_rows = [&](uint32_t hm, float W, uint32_t row, uint32_t col) {
            if ((hm >> lane) & 1u) {
                uint32_t slot = tail + npend + __popc(hm & lt);
                if (slot >= HROWS) slot -= HROWS;
                float* p = hit + slot * HROW_PITCH;
#pragma unroll
                for (int c = 0; c < 32; c += 4)
                    *reinterpret_cast<uint4*>(p + c) = make_uint4(v[c], v[c + 1], v[c + 2], v[c + 3]);
                *reinterpret_cast<uint4*>(p + 32) = make_uint4(__float_as_uint(W), row, col, 0u);
            }
            npend += __popc(hm);
        };
        auto put_band = [&](uint32_t mask, uint32_t row, uint32_t col) {
            nrecs += put_records(a.band, a.band_cap, &a.st->band_count, bsp, mask, row, col, lane);
            npairs += __popc(mask);
        };
        auto put_in = [&](uint32_t mask, uint32_t row, uint32_t col) {
            nin += put_records(a.em.inq, a.em.inq_cap, &a.em.cnt[0], esp, mask, row, col, lane);
        };
        // up to four rows of the ring: eight lanes per row, four columns per lane
        auto count_rows = [&]() {
            __syncwarp();
            const uint32_t g = lane >> 3, n = min(npend, 4u);
            uint32_t slot = tail + g;
            if (slot >= HROWS) slot -= HROWS;
            const float* p = hit + slot * HROW_PITCH;
            const float4 x = *reinterpret_cast<const float4*>(p + 4 * (lane & 7u));
            const uint4 m = *reinterpret_cast<const uint4*>(p + 32);
            const float W = __uint_as_float(m.x);
            const float xs[4] = {x.x, x.y, x.z, x.w};
            // sign tests, as in classify
            uint32_t inm = 0, bdm = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const bool in = __float_as_int(xs[k]) >= 0;
                inm |= in ? 1u << k : 0u;
                bdm |= !in && __float_as_int(xs[k] + W) >= 0 ? 1u << k : 0u;
            }
            if (g >= n) inm = bdm = 0;
            const uint32_t col = m.z + 4u * (lane & 7u);
            if (inm) {
                atomicAdd(&a.counts[m.y], __popc(inm));
                if (m.z & kBandBoth) {
                    int32_t* cc = a.counts + (col & ~kBandBoth);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if ((inm >> k) & 1u) atomicAdd(cc + k, 1);
                }
            }
            if (a.em.cnt) put_in(inm, m.y, col);
            put_band(bdm, m.y, col);
            __syncwarp();
            tail += n;
            if (tail >= HROWS) tail -= HROWS;
            npend -= n;
        };
        for (; u < a.nwork; ++it) {
            const uint32_t b = it & 1u, use = it >> 1;
            u = un;
            un = next_item(un, a.lrun);
            const uint2 wnn = entry_or_end(a, un);
            const Margins mn = load_margins(wn);
            if (e_row(w, rank) != I) {  // warp-uniform
                if (rowcnt) atomicAdd(&a.counts[I * 128u + q * 32u + lane], rowcnt);
                rowcnt = 0;
                I = e_row(w, rank);
            }
            const uint32_t J = e_col(w, h);
            const bool active = is_active(w);
            const uint32_t taddr = tq + b * ACC_COLS;
            // the bit masks of dense chunks
            uint32_t in0 = 0, bd0 = 0, in1 = 0, bd1 = 0;
            bool dense = false;
            const bool diag = a.cross || (I == J);  // credit rows only
            const uint32_t row = I * 128u + q * 32u + lane;
            const uint32_t col0 = (J * 128u + (cg & 1u) * 64u) | (diag ? 0u : kBandBoth);
            // rows put down earlier are counted until the accumulator is ready
            // and the ring has room for this block's (votes, so that the lanes
            // stay together)
            bool ok = true;
            for (;;) {
                const bool ready = __all_sync(FULL, ptx::mbar_test_wait(&S.tfull[b], use & 1u));
                if (ready) break;
                if (npend == 0) {
                    ok = __all_sync(FULL, ptx::mbar_wait(&S.tfull[b], use & 1u, a.st, 30));
                    break;
                }
                count_rows();
            }
            if (!ok) break;
            ptx::tc_fence_after();
            if (active) {
                // (rounding of the FP32 add is monotone, so max + W >= 0 whenever
                // any element is >= -W: the other rows are certainly out)
                ptx::tmem_ld_max_32x32b_x32(taddr, v, mx);
                ptx::tmem_ld_wait_regs(v, mx);
                const uint32_t hm = __ballot_sync(FULL, mx + W0 >= 0.0f);
                if (__popc(hm) > min(HCHUNK, HROWS - npend)) {
                    classify(v, W0, in0, bd0);
                    dense = true;
                } else if (hm) {
                    put_rows(hm, W0, row, col0);
                }
                ptx::tmem_ld_max_32x32b_x32(taddr + 32u, v, mx);
                ptx::tmem_ld_wait_regs(v, mx);
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive_cluster(tempty0 + b * 8u);
            if (active) {
                const uint32_t hm = __ballot_sync(FULL, mx + W1 >= 0.0f);
                if (__popc(hm) > min(HCHUNK, HROWS - npend)) {
                    classify(v, W1, in1, bd1);
                    dense = true;
                } else if (hm) {
                    put_rows(hm, W1, row, col0 + 32u);
                }
            }
            if (dense) {  // warp-uniform
                put_band(bd0, row, col0);
                put_band(bd1, row, col0 + 32u);
                if (!diag) {
                    int32_t* cc = a.counts + (col0 & ~kBandBoth);
                    col_counts(in0, cc, lane);
                    col_counts(in1, cc + 32, lane);
                }
                rowcnt += __popc(in0) + __popc(in1);
                if (a.em.cnt) {
                    put_in(in0, row, col0);
                    put_in(in1, row, col0 + 32u);
                }
            }
            W0 = width(mn, mn.t0);
            W1 = width(mn, mn.t1);
            w = wn;
            wn = wnn;
        }
        while (npend) count_rows();
        if (rowcnt) atomicAdd(&a.counts[I * 128u + q * 32u + lane], rowcnt);
        pad_records(a.band, a.band_cap, bsp, lane);
        if (a.em.cnt) pad_records(a.em.inq, a.em.inq_cap, esp, lane);
#pragma unroll
        for (int o = 16; o; o >>= 1) npairs += __shfl_xor_sync(FULL, npairs, o);
        if (lane == 0 && nrecs) {
            atomicAdd(&a.st->band_pairs, npairs);
            atomicAdd(&a.st->band_records, (unsigned long long)nrecs);
        }
        if (lane == 0 && nin) atomicAdd(&a.st->in_records, (unsigned long long)nin);
    }

    ptx::tc_fence_before();
    __syncthreads();
    // neither CTA of a pair leaves (or frees tensor memory) while the other
    // may still reach its shared memory
    ptx::cluster_sync();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc<2>(tmem, TMEM_COLS);
    }
}

}  // namespace

uint64_t gram_queue_slack(uint64_t nwork, int num_sms) {
    return 2 * std::min<uint64_t>(nwork, (uint64_t)num_sms / 2) * NUM_EPI_WARPS * kResChunk;
}

int launch_gram16(const GramSide& A, const GramSide& B, const ScreenParams& P, const uint2* work,
                  uint64_t nwork, const float* cmax, const float* beta, const float* tsig,
                  const float* sig, bool cross, int32_t* counts, BandRec* band, uint64_t band_cap,
                  DevStatus* st, const Emit* em, int num_sms, cudaStream_t s) {
    if (nwork == 0) return EJOIN_OK;
    if (num_sms < 2) return set_error(EJOIN_EINTERNAL, "gram: no CTA pair fits");
    const bool fp8 = P.fmt == Fmt::E4M3;
    if (A.n_pad % 128 || B.n_pad % 256 || P.dp % (fp8 ? 128 : 64))
        return set_error(EJOIN_EINTERNAL, "gram: bad padding");
    if (A.n_pad > 0x7fffff00ull || B.n_pad > 0x7fffff00ull)
        return set_error(EJOIN_EUNSUPPORTED, "gram16: too many rows");
    CUtensorMap ma, mb, maa, mab;
    const CUtensorMapDataType adt =
        P.fmt == Fmt::FP16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    if (fp8) {
        EJ_TRY(make_tmap_2d(&ma, A.Q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, P.width, A.n_pad, 128, 128));
        EJ_TRY(make_tmap_2d(&mb, B.Q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, P.width, B.n_pad, 128, 128));
    } else {
        EJ_TRY(make_tmap_2d(&ma, A.Q, adt, 2, P.width, A.n_pad, 64, 128));
        EJ_TRY(make_tmap_2d(&mb, B.Q, adt, 2, P.width, B.n_pad, 64, 128));
    }
    EJ_TRY(make_tmap_2d(&maa, A.aug, adt, 2, 64, A.n_pad / 2, 64, 32, false));
    EJ_TRY(make_tmap_2d(&mab, B.aug, adt, 2, 64, B.n_pad / 2, 64, 32, false));
    GramArgs a;
    a.work = work;
    a.nwork = nwork;
    a.cmax = cmax;
    a.beta = beta;
    a.tsig = fp8 ? tsig : nullptr;
    a.sig = fp8 ? sig : nullptr;
    a.em = em ? *em : Emit{nullptr, 0, nullptr, 0, nullptr};
    a.cross = cross ? 1u : 0u;
    if ((uintptr_t)cmax & 7) return set_error(EJOIN_EINTERNAL, "gram: chunk margins misaligned");
    if (!cmax || !beta || (fp8 && (!tsig || !sig))) return set_error(EJOIN_EINTERNAL, "gram: margins missing");
    a.counts = counts;
    a.band = band;
    a.band_cap = band_cap;
    a.st = st;
    a.nhi = P.dp / (fp8 ? 128 : 64);
    a.fmt = P.fmt == Fmt::BF16 ? 1u : 0u;
    // runs of consecutive entries per CTA pair (up to 16) while each still gets
    // several runs
    const uint64_t workers = (uint64_t)num_sms / 2;
    uint32_t lrun = 4;
    while (lrun > 0 && nwork < workers * (4ull << lrun)) --lrun;
    a.lrun = lrun;
    const uint64_t runs = (nwork + (1ull << lrun) - 1) >> lrun;
    auto kern = fp8 ? gram_kernel<1, false>
                    : (P.split ? gram_kernel<0, true> : gram_kernel<0, false>);
    EJ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * std::min(runs, workers)));
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    EJ_CUDA(cudaLaunchKernelEx(&cfg, kern, ma, mb, maa, mab, a));
    EJ_CUDA(cudaGetLastError());
    note_launch();
    return EJOIN_OK;
}

}  // namespace ejoin
