// k_direct.cu -- FP64 CUDA-core kernels with the reference's exact arithmetic.
//
//  * direct_selfjoin_kernel: the exact arbiter (EJOIN_FP64_DIRECT, reference
//    searchMode 1, kernel_join.cu:168-200).  The reference runs one thread
//    per query over all N candidates and bumps one global 64-bit counter per
//    hit; here a CTA takes one 64x64 tile pair of the upper triangle (I <= J),
//    stages both row blocks in shared memory k-chunk by k-chunk, every thread
//    keeps a 4x4 block of independent FP64 chains, and the hits become
//    per-point counts (row counts for I, column counts for J when I < J).
//    d2(a, b) and d2(b, a) are bitwise equal ((a-b)^2 == (b-a)^2), so the
//    upper triangle is exact.  A pair whose partial sum exceeds T is dropped:
//    every later step adds a square to it (rounding is monotone), so its d2
//    exceeds T too (tile_pairs).
//  * direct_query_kernel: the same tile over (query rows) x (all points).
//  * band_recheck_kernel: one thread per band pair, the same chain.
//
// Every chain follows the reference's compiled arithmetic (exact_d2:
// fma(t0, t0, fl(t1*t1)), then fma(t, t, acc) in index order).  Zero padding
// of the k loop is exact: fma(0, 0, acc) == acc for acc >= +0.
#include <cuda_fp16.h>

#include <algorithm>

#include "ejoin_internal.cuh"

namespace ejoin {
namespace {

constexpr int TB = 64;        // tile edge (points)
constexpr int KC = 16;        // k-chunk staged per step
constexpr int KS = 4;         // coordinates between two looks at the partial sums
constexpr int PADK = TB + 1;  // smem row pitch (doubles) of the k-major stage
// pairs kept in a list once no more of a tile's 4096 are left
constexpr uint32_t LMAX = 1024;

// Stage rows [r0, r0+64) x coords [k0, k0+KC) of X (row stride ld) into
// S[k][r] (k-major).  rows >= n and coords >= d are zero.
__device__ __forceinline__ void stage_tile(double (*S)[PADK], const double* __restrict__ X,
                                           uint64_t n, uint32_t d, uint64_t r0, uint32_t k0,
                                           const uint64_t* __restrict__ rowmap, uint64_t nmap) {
#pragma unroll
    for (int e = threadIdx.x; e < TB * KC; e += 256) {
        int r = e / KC, k = e % KC;
        uint64_t row = r0 + r;
        uint32_t kk = k0 + k;
        double v = 0.0;
        if (rowmap) {
            if (row < nmap && kk < d) v = X[rowmap[row] * (uint64_t)d + kk];
        } else if (row < n && kk < d) {
            v = X[row * (uint64_t)d + kk];
        }
        S[k][r] = v;
    }
}

// Coordinates [k0, k0 + KS) of one 64x64 tile of exact squared distances.
// Thread (ty, tx) owns rows ty + 16*rr and columns tx + 16*cc.  `first` starts
// every chain with fma(t0, t0, fl(t1*t1)), the reference's compiled form of its
// first two terms (exact_d2); zero-padded coordinates give t = 0 there too.
__device__ __forceinline__ void tile_chains(double acc[4][4], double (*SA)[PADK],
                                            double (*SB)[PADK], int ty, int tx, int k0, bool first) {
    int j0 = 0;
    if (first) {
        double a0[4], a1[4], b0[4], b1[4];
#pragma unroll
        for (int rr = 0; rr < 4; ++rr) {
            a0[rr] = SA[0][ty + 16 * rr];
            a1[rr] = SA[1][ty + 16 * rr];
        }
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            b0[cc] = SB[0][tx + 16 * cc];
            b1[cc] = SB[1][tx + 16 * cc];
        }
#pragma unroll
        for (int rr = 0; rr < 4; ++rr)
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const double t0 = __dsub_rn(a0[rr], b0[cc]);
                const double t1 = __dsub_rn(a1[rr], b1[cc]);
                acc[rr][cc] = __fma_rn(t0, t0, __dmul_rn(t1, t1));
            }
        j0 = 2;
    }
#pragma unroll 2
    for (int k = k0 + j0; k < k0 + KS; ++k) {
        double a[4], b[4];
#pragma unroll
        for (int rr = 0; rr < 4; ++rr) a[rr] = SA[k][ty + 16 * rr];
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) b[cc] = SB[k][tx + 16 * cc];
#pragma unroll
        for (int rr = 0; rr < 4; ++rr)
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                double t = __dsub_rn(a[rr], b[cc]);
                acc[rr][cc] = __fma_rn(t, t, acc[rr][cc]);
            }
    }
}

struct TileSmem {
    double A[KC][PADK], B[KC][PADK];
    double lacc[2][LMAX];   // pairs left: partial sum, row | column << 8
    uint16_t lrc[2][LMAX];
    uint32_t cnt[3];        // pairs left, in turn
};

// All pairs of a 64 x 64 tile whose d2 is <= T: hit(row, column) by some thread
// for each.  nr / nc: rows and columns that hold points; stage(k0) fills S.A and
// S.B with coordinates [k0, k0 + KC).
//
// FP64 arithmetic is what this costs (2 instructions per pair and coordinate; an
// SM starts two FP64 operations a clock: 4096 clocks per coordinate of a tile), so
// every KS coordinates the pairs whose partial sum exceeds T are dropped -- by
// the high words, an integer comparison: larger high word, larger sum, and a
// NaN's exceeds T's too; equal ones stay -- and once at most LMAX pairs are left
// they go on as a list, a pair per thread, without the dropped ones.  500 rows
// against 200k x 64 points in 64 clusters: 23.5 ms without dropping, 2.4 ms with.
template <typename Stage, typename Hit>
__device__ __forceinline__ void tile_pairs(TileSmem& S, uint32_t d, double T, uint32_t nr,
                                           uint32_t nc, Stage&& stage, Hit&& hit) {
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const uint32_t lane = threadIdx.x & 31;
    const int hT = __double2hiint(T);  // T >= 0
    double acc[4][4];
    uint32_t left = 0;  // bit 4 rr + cc: the pair is still in
#pragma unroll
    for (int rr = 0; rr < 4; ++rr)
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            acc[rr][cc] = 0.0;
            if (ty + 16 * rr < (int)nr && tx + 16 * cc < (int)nc) left |= 1u << (4 * rr + cc);
        }
    bool list = false;
    uint32_t cur = 0, n = 0, turn = 0;
    if (threadIdx.x < 3) S.cnt[threadIdx.x] = 0;
    // slots for c pairs of this lane among the turn's (returns the first)
    auto reserve = [&](uint32_t c) {
        uint32_t incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        uint32_t base = 0;
        if (lane == 31 && incl) base = atomicAdd(&S.cnt[turn], incl);
        return __shfl_sync(0xffffffffu, base, 31) + incl - c;
    };
    // the turn's total (all threads), and the next turn
    auto total = [&]() {
        __syncthreads();
        const uint32_t c = S.cnt[turn];
        if (threadIdx.x == 0) S.cnt[(turn + 2) % 3] = 0;
        turn = (turn + 1) % 3;
        return c;
    };
    for (uint32_t k0 = 0; k0 < d; k0 += KC) {
        __syncthreads();
        stage(k0);
        __syncthreads();
        uint32_t ks = 0;
        for (; !list && ks < KC && k0 + ks < d; ks += KS) {
            tile_chains(acc, S.A, S.B, ty, tx, ks, k0 + ks == 0);
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (__double2hiint(acc[e / 4][e % 4]) > hT) left &= ~(1u << e);
            const uint32_t at = reserve(__popc(left));
            n = total();
            if (n == 0) return;
            if (n <= LMAX) {
                uint32_t o = at;
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if ((left >> e) & 1u) {
                        S.lacc[0][o] = acc[e / 4][e % 4];
                        S.lrc[0][o] = (uint16_t)((ty + 16 * (e / 4)) | ((tx + 16 * (e % 4)) << 8));
                        ++o;
                    }
                list = true;
                __syncthreads();
            }
        }
        if (list && ks < KC && k0 + ks < d) {
            // the rest of the chunk for the pairs left (padding adds zero)
            for (uint32_t e0 = 0; e0 < n; e0 += 256) {
                const uint32_t e = e0 + threadIdx.x;
                double v = 0.0;
                uint32_t rc = 0;
                bool in = e < n;
                if (in) {
                    v = S.lacc[cur][e];
                    rc = S.lrc[cur][e];
                    const uint32_t r = rc & 255u, c = rc >> 8;
                    for (uint32_t k = ks; k < KC; ++k) {
                        const double t = __dsub_rn(S.A[k][r], S.B[k][c]);
                        v = __fma_rn(t, t, v);
                    }
                    in = __double2hiint(v) <= hT;
                }
                const uint32_t o = reserve(in ? 1u : 0u);
                if (in) {
                    S.lacc[cur ^ 1][o] = v;
                    S.lrc[cur ^ 1][o] = (uint16_t)rc;
                }
            }
            n = total();
            if (n == 0) return;
            cur ^= 1u;
        }
    }
    if (list) {
        for (uint32_t e = threadIdx.x; e < n; e += 256)
            if (S.lacc[cur][e] <= T) hit(S.lrc[cur][e] & 255u, S.lrc[cur][e] >> 8);
    } else {
#pragma unroll
        for (int e = 0; e < 16; ++e)
            if (((left >> e) & 1u) && acc[e / 4][e % 4] <= T)
                hit((uint32_t)(ty + 16 * (e / 4)), (uint32_t)(tx + 16 * (e % 4)));
    }
}

__global__ void __launch_bounds__(256, 3) direct_selfjoin_kernel(const double* __restrict__ X,
                                                              uint64_t n, uint32_t d, double T,
                                                              uint64_t nT, uint64_t tiles,
                                                              int32_t* counts, Emit em) {
    __shared__ TileSmem S;
    __shared__ int rowc[TB], colc[TB];
    const uint64_t t = blockIdx.x + (uint64_t)blockIdx.y * gridDim.x;
    if (t >= tiles) return;
    uint64_t I, J;
    tri_decode(t, nT, I, J);
    if (threadIdx.x < TB) {
        rowc[threadIdx.x] = 0;
        colc[threadIdx.x] = 0;
    }
    const bool diag = (I == J);
    tile_pairs(
        S, d, T, (uint32_t)min((uint64_t)TB, n - I * TB), (uint32_t)min((uint64_t)TB, n - J * TB),
        [&](uint32_t k0) {
            stage_tile(S.A, X, n, d, I * TB, k0, nullptr, 0);
            stage_tile(S.B, X, n, d, J * TB, k0, nullptr, 0);
        },
        [&](uint32_t r, uint32_t c) {
            atomicAdd(&rowc[r], 1);
            if (!diag) atomicAdd(&colc[c], 1);
            emit_pair(em, BandPair{(uint32_t)(I * TB + r),
                                   (uint32_t)(J * TB + c) | (diag ? 0u : kBandBoth)});
        });
    __syncthreads();
    if (threadIdx.x < TB) {
        uint64_t i = I * TB + threadIdx.x, j = J * TB + threadIdx.x;
        if (rowc[threadIdx.x] && i < n) atomicAdd(&counts[i], rowc[threadIdx.x]);
        if (colc[threadIdx.x] && j < n) atomicAdd(&counts[j], colc[threadIdx.x]);
    }
}

// Query rows: rows[q] of X, or (Xq non-null) row q of a separate array Xq.
__global__ void __launch_bounds__(256, 3) direct_query_kernel(const double* __restrict__ X, uint64_t n,
                                                           uint32_t d, double T,
                                                           const uint64_t* __restrict__ rows,
                                                           const double* __restrict__ Xq,
                                                           uint64_t nq, int32_t* counts) {
    __shared__ TileSmem S;
    __shared__ int rowc[TB];
    const uint64_t Q = blockIdx.y, J = blockIdx.x;
    if (threadIdx.x < TB) rowc[threadIdx.x] = 0;
    tile_pairs(
        S, d, T, (uint32_t)min((uint64_t)TB, nq - Q * TB), (uint32_t)min((uint64_t)TB, n - J * TB),
        [&](uint32_t k0) {
            if (Xq) stage_tile(S.A, Xq, nq, d, Q * TB, k0, nullptr, 0);
            else stage_tile(S.A, X, n, d, Q * TB, k0, rows, nq);
            stage_tile(S.B, X, n, d, J * TB, k0, nullptr, 0);
        },
        [&](uint32_t r, uint32_t) { atomicAdd(&rowc[r], 1); });
    __syncthreads();
    if (threadIdx.x < TB) {
        uint64_t q = Q * TB + threadIdx.x;
        if (rowc[threadIdx.x] && q < nq) atomicAdd(&counts[q], rowc[threadIdx.x]);
    }
}

__global__ void __launch_bounds__(256) band_recheck_kernel(const double* __restrict__ X, uint32_t d,
                                                           const uint32_t* __restrict__ perm,
                                                           double T,
                                                           const BandPair* __restrict__ band,
                                                           uint64_t nband, uint64_t n,
                                                           int32_t* counts, DevStatus* st) {
    uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    unsigned hit = 0;
    BandPair bp = {0u, 0u};
    if (e < nband) bp = band[e];
    const uint32_t i = bp.i, j = bp.j & ~kBandBoth;
    // padding rows (index >= n) hold no point: such pairs are never neighbours
    if (e < nband && i < n && j < n) {
        uint64_t oi = perm ? perm[i] : i, oj = perm ? perm[j] : j;
        double d2 = exact_d2(X + oi * (uint64_t)d, X + oj * (uint64_t)d, d);
        if (d2 <= T) {
            hit = 1;
            atomicAdd(&counts[i], 1);
            if (bp.j & kBandBoth) atomicAdd(&counts[j], 1);
        }
    }
    unsigned c = __reduce_add_sync(0xffffffffu, hit);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&st->band_hits, (unsigned long long)c);
}

// Two-stage recheck of the band of the tensor-core screen.  For every band
// pair, S = sum_c fl32(zf_ic - zf_jc)^2 over the FP32 coordinates of the
// packed rows (any summation order: the bound covers it), then a rigorous
// decision that scales with the pair's own distance:
//   |w| = |zf_i - zf_j| differs from the exact scaled distance by at most
//   rad_i + rad_j, and S from |w|^2 by the relative c32 (+ abs32), so
//   S / (1 - c32) <= (sqrt(Tlo) - rad)^2   => neighbour
//   S / (1 + c32) >  (sqrt(Thi) + rad)^2   => not a neighbour
// i.e. S + abs32 <= (sqrt(Tlo) - rad)^2 (1 - c32) and
//      S - abs32 >  (sqrt(Thi) + rad)^2 (1 + c32).
// Both tests run in FP32 with every operation rounded in the safe direction
// (the constants are rounded outward on the host), so they stay rigorous
// without FP64, whose throughput on GB300 is a small fraction of FP32's.  An
// infinite radius (bad or padding row) decides nothing.
// Only the pairs left undecided (a tiny fraction) run the exact FP64 chain of
// the reference arithmetic on the original rows.  Returns whether (i, j) is a
// neighbour pair; counts the exact runs.
__device__ __forceinline__ bool recheck_decide(const double* __restrict__ X, uint32_t d,
                                               const uint32_t* __restrict__ perm, double T,
                                               const Recheck32& R, uint32_t i, uint32_t j,
                                               float S, unsigned& exact_runs) {
    const float rr = __fadd_ru(R.rad[i], R.radb[j]);
    const float lo = __fsub_rd(R.f_sTlo, rr);
    if (lo >= 0.0f && __fadd_ru(S, R.f_abs) <= __fmul_rd(__fmul_rd(lo, lo), R.f_kin)) return true;
    const float hi = __fadd_ru(R.f_sThi, rr);
    if (__fsub_rd(S, R.f_abs) > __fmul_ru(__fmul_ru(hi, hi), R.f_kout)) return false;
    ++exact_runs;
    const uint64_t oi = perm ? perm[i] : i, oj = R.permb ? R.permb[j] : j;
    return exact_d2(X + oi * (uint64_t)d, R.Xb + oj * (uint64_t)d, d) <= T;
}

__device__ __forceinline__ void recheck_totals(DevStatus* st, unsigned hits, unsigned exact_runs) {
    const unsigned c = __reduce_add_sync(0xffffffffu, hits);
    const unsigned x = __reduce_add_sync(0xffffffffu, exact_runs);
    if ((threadIdx.x & 31) == 0) {
        if (c) atomicAdd(&st->band_hits, (unsigned long long)c);
        if (x) atomicAdd(&st->exact_rechecks, (unsigned long long)x);
    }
}

// Read-only row loads that do not allocate in L1: the band rows are
// gathered with little reuse, and allocating them thrashed L1 (measured on
// c4: the recheck ran 1.4x faster without allocation).  32 bytes (p 32-byte
// aligned) or 16 bytes (p 16-byte aligned).
__device__ __forceinline__ void ldg8(const float* p, float (&r)[8]) {
    asm("ld.global.nc.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]),
          "=f"(r[7])
        : "l"(p));
}
// cached forms, for the row a warp reuses across consecutive pairs
__device__ __forceinline__ void ldg8c(const float* p, float (&r)[8]) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]),
          "=f"(r[7])
        : "l"(p));
}

// Short rows (below 64 coordinates; rows are padded to whole 32 bytes): a thread
// per pair streams both rows with 32-byte loads (four partial sums): 32 pairs in
// flight per warp.  The kernel is bound by L1 wavefronts (each lane reads its own
// row), so wide loads move the most bytes per wavefront.
__global__ void __launch_bounds__(256) band_recheck_thread_kernel(const double* __restrict__ X,
                                                                  uint32_t d,
                                                                  const uint32_t* __restrict__ perm,
                                                                  double T, Recheck32 R,
                                                                  const BandPair* __restrict__ band,
                                                                  uint64_t nband, uint64_t n,
                                                                  int32_t* counts, DevStatus* st,
                                                                  Emit em) {
    unsigned hits = 0, exact_runs = 0;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < nband;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const BandPair bp = band[e];
        const uint32_t i = bp.i, j = bp.j & ~kBandBoth;
        if (i >= n || j >= R.nb) continue;
        float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
        const float* a = R.Xf + (uint64_t)i * R.ds;
        const float* b = R.Xfb + (uint64_t)j * R.ds;
#pragma unroll 2
        for (uint32_t c = 0; c < R.ds; c += 8) {
            float u[8], v[8];
            ldg8(a + c, u);
            ldg8(b + c, v);
#pragma unroll
            for (int k = 0; k < 8; k += 4) {
                const float t0 = u[k] - v[k], t1 = u[k + 1] - v[k + 1];
                const float t2 = u[k + 2] - v[k + 2], t3 = u[k + 3] - v[k + 3];
                s0 = fmaf(t0, t0, s0);
                s1 = fmaf(t1, t1, s1);
                s2 = fmaf(t2, t2, s2);
                s3 = fmaf(t3, t3, s3);
            }
        }
        if (recheck_decide(X, d, perm, T, R, i, j, (s0 + s1) + (s2 + s3), exact_runs)) {
            atomicAdd(&counts[i], 1);
            if (bp.j & kBandBoth) atomicAdd(&counts[j], 1);
            emit_pair(em, bp);
            ++hits;
        }
    }
    recheck_totals(st, hits, exact_runs);
}

// First decision of a band pair from the FP16 copies (S = their squared
// distance, computed in FP32 like the FP32 one: the conversions are exact):
// 1 = in, 0 = out, -1 = undecided.  The copies' radii (rad + |zh - zf|)
// replace the FP32 radii; otherwise the same directed-rounding tests as
// recheck_decide.
__device__ __forceinline__ int decide16(const Recheck32& R, uint32_t i, uint32_t j, float S) {
    const float rr = __fadd_ru(R.radh[i], R.radhb[j]);
    const float lo = __fsub_rd(R.f_sTlo, rr);
    if (lo >= 0.0f && __fadd_ru(S, R.f_abs) <= __fmul_rd(__fmul_rd(lo, lo), R.f_kin)) return 1;
    const float hi = __fadd_ru(R.f_sThi, rr);
    if (__fsub_rd(S, R.f_abs) > __fmul_ru(__fmul_ru(hi, hi), R.f_kout)) return 0;
    return -1;
}

// 8 FP16 values (16 bytes, p 16-byte aligned): the cached form for the row a
// warp reuses, the no-allocate form for the gathered one.
__device__ __forceinline__ uint4 ldg8hc(const uint16_t* p) {
    uint4 r;
    asm("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ uint4 ldg8h(const uint16_t* p) {
    uint4 r;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(p));
    return r;
}
__device__ __forceinline__ float sqdiff_h2(uint32_t a, uint32_t b, float S) {
    const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&a));
    const float2 fb = __half22float2(*reinterpret_cast<const __half2*>(&b));
    const float t0 = fa.x - fb.x, t1 = fa.y - fb.y;
    return fmaf(t1, t1, fmaf(t0, t0, S));
}

// Longer rows: a warp takes ppw <= 32 band pairs, 32 / G at a time: G lanes
// stream the two rows of a pair (eight values per lane and load; rows are padded
// to whole 32 bytes) and add up S, and lane p then decides pair p.  With FP16
// copies (R.Xh) a first pass over them decides almost every pair of a wide band
// at half the bytes; only the pairs it leaves open stream the FP32 rows.
//
// NV > 0 (G = 32, FP16 copies, ds <= 256 NV): the rows of the FP16 pass stream
// through a queue of kStreamSlots rows per warp in shared memory (a lane copies and
// reads the same 16-byte pieces, so nothing but its own copies is waited for), and
// row i, which consecutive pairs often share (the screen's records hold up to 32
// columns of a row), is fetched once and kept in registers as FP32.  34.4 M pairs of
// 1024 coordinates: 10.9 ms with both rows loaded for every pair, which waited for
// one pair's loads at a time; now 8.3, bound by issue (conversions, FMAs).  Row i in
// registers without the queue took 10.7, and pairs sorted by blocks of 4096 rows,
// so that all rows come from L2, gain 0.2 ms for a sort of 1.1.
// (Blocks: four waves of the three that fit an SM; 64 and 3 per SM both took 8.6 ms.)
constexpr uint32_t kStreamSlots = 4, kStreamBlocks = 152 * 12;
constexpr uint32_t stream_smem(int NV) { return 8 * kStreamSlots * NV * 512; }
template <uint32_t G, int NV = 0>
__global__ void __launch_bounds__(256, NV ? 3 : 5) band_recheck_warp_kernel(const double* __restrict__ X,
                                                                uint32_t d,
                                                                const uint32_t* __restrict__ perm,
                                                                double T, Recheck32 R,
                                                                const BandPair* __restrict__ band,
                                                                uint64_t nband, uint32_t ppw,
                                                                uint64_t n, int32_t* counts,
                                                                DevStatus* st, Emit em) {
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr uint32_t NG = 32 / G;
    const uint32_t lane = threadIdx.x & 31, g = lane / G, l = lane % G;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32;
    const uint64_t nwarps = (uint64_t)gridDim.x * blockDim.x / 32;
    unsigned hits = 0, exact_runs = 0;
    // the warp's queue: shared-memory addresses of the lane's piece of its first and
    // last slot; pieces beyond the rows' end stay zero
    extern __shared__ uint4 stream_sm[];
    const uint32_t q_first = (uint32_t)__cvta_generic_to_shared(stream_sm) +
                             (threadIdx.x / 32) * (kStreamSlots * NV * 512) + 16 * lane;
    const uint32_t q_last = q_first + (kStreamSlots - 1) * NV * 512;
    if constexpr (NV > 0)
        for (uint32_t v = 0; v < kStreamSlots * NV; ++v)
            if (8 * (lane + 32 * (v % NV)) >= R.ds)
                stream_sm[((threadIdx.x / 32) * kStreamSlots * NV + v) * 32 + lane] = make_uint4(0u, 0u, 0u, 0u);
    for (uint64_t base = warp * ppw; base < nband; base += nwarps * ppw) {
        const uint64_t e = lane < ppw ? base + lane : nband;
        BandPair bp = {0xffffffffu, 0xffffffffu};
        if (e < nband) bp = band[e];
        const uint32_t mi = bp.i, mj = bp.j & ~kBandBoth;
        const bool valid = e < nband && mi < n && mj < R.nb;
        // S of those of the pairs q0 .. q0 + NG - 1 that `which` names, from sum(row i,
        // row j) over the lanes of a group; lane q0 + g keeps pair q0 + g's
        auto sums = [&](uint32_t q0, uint32_t which, float& mine, auto&& sum) {
            const uint32_t i = __shfl_sync(FULL, mi, q0 + g), j = __shfl_sync(FULL, mj, q0 + g);
            float S = 0.0f;
            if ((which >> (q0 + g)) & 1u) S = sum((uint64_t)i * R.ds, (uint64_t)j * R.ds);
            for (int o = G / 2; o; o >>= 1) S += __shfl_xor_sync(FULL, S, o);
            const float got = __shfl_sync(FULL, S, (lane % NG) * G);
            if (lane - lane % NG == q0) mine = got;
        };
        bool open = valid, hit = false;
        const uint32_t named = __ballot_sync(FULL, valid);
        float mh = 0.0f;
        if constexpr (NV > 0) {
            static_assert(G == 32);
            // pairs whose row i is not that of the pair before
            const uint32_t below = named & ((1u << lane) - 1u);
            const uint32_t before = __shfl_sync(FULL, mi, below ? 31 - __clz(below) : 0);
            const uint32_t fresh = __ballot_sync(FULL, valid && (!below || before != mi));
            uint32_t togo = named, put = q_first, get = q_first;
            bool row_i = true;  // the next row to fetch: i of the next pair, or its j
            auto fetch = [&]() {  // warp-uniform; a group even when nothing is left
                if (togo) {
                    const uint32_t q = __ffs(togo) - 1;
                    const bool first = row_i && ((fresh >> q) & 1u);
                    const uint32_t row = __shfl_sync(FULL, first ? mi : mj, q);
                    const uint16_t* src = (first ? R.Xh : R.Xhb) + ((uint64_t)row * R.ds + 8 * lane);
                    row_i = !first;
                    if (!first) togo &= togo - 1;
#pragma unroll
                    for (int v = 0; v < NV; ++v)
                        if (8 * (lane + 32 * v) < R.ds)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(put + v * 512),
                                         "l"(src + 256 * v)
                                         : "memory");
                }
                put = put == q_last ? q_first : put + NV * 512;
                asm volatile("cp.async.commit_group;\n" ::: "memory");
            };
            float2 fa[4 * NV];
            auto next_row = [&](auto&& use) {
                asm volatile("cp.async.wait_group %0;\n" ::"n"(kStreamSlots - 2) : "memory");
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    uint4 u;
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                                 : "r"(get + v * 512)
                                 : "memory");
                    const uint32_t h[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        use(4 * v + k, __half22float2(*reinterpret_cast<const __half2*>(&h[k])));
                }
                get = get == q_last ? q_first : get + NV * 512;
                fetch();  // into the slot read one row earlier
            };
            for (uint32_t k = 0; k < kStreamSlots - 1; ++k) fetch();
            for (uint32_t left = named; left; left &= left - 1) {
                const uint32_t q = __ffs(left) - 1;
                if ((fresh >> q) & 1u) next_row([&](int k, float2 f) { fa[k] = f; });
                float2 s2 = make_float2(0.0f, 0.0f);
                next_row([&](int k, float2 f) {
                    const float2 t = __ffma2_rn(f, make_float2(-1.0f, -1.0f), fa[k]);  // fa - f
                    s2 = __ffma2_rn(t, t, s2);
                });
                float S = s2.x + s2.y;
                for (int o = 16; o; o >>= 1) S += __shfl_xor_sync(FULL, S, o);
                if (lane == q) mh = S;
            }
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");  // (empty groups)
        } else if (G < 32 && R.Xh) {
            for (uint32_t q0 = 0; q0 < ppw; q0 += NG)
                sums(q0, named, mh, [&](uint64_t oi, uint64_t oj) {
                    const uint16_t *a = R.Xh + oi, *b = R.Xhb + oj;
                    float S = 0.0f;
#pragma unroll 4
                    for (uint32_t c = 8 * l; c < R.ds; c += 8 * G) {
                        const uint4 u = ldg8hc(a + c), w = ldg8h(b + c);
                        S = sqdiff_h2(u.x, w.x, S);
                        S = sqdiff_h2(u.y, w.y, S);
                        S = sqdiff_h2(u.z, w.z, S);
                        S = sqdiff_h2(u.w, w.w, S);
                    }
                    return S;
                });
        }
        if (R.Xh && valid) {
            const int dec = decide16(R, mi, mj, mh);
            if (dec >= 0) {
                open = false;
                hit = dec == 1;
            }
        }
        float mine = 0.0f;
        const uint32_t left = __ballot_sync(FULL, open);
        for (uint32_t q0 = 0; q0 < ppw; q0 += NG)
            if ((left >> q0) & ((1u << NG) - 1u))  // warp-uniform
                sums(q0, left, mine, [&](uint64_t oi, uint64_t oj) {
                    const float *a = R.Xf + oi, *b = R.Xfb + oj;
                    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll 2
                    for (uint32_t c = 8 * l; c < R.ds; c += 8 * G) {
                        float u[8], w[8];
                        ldg8c(a + c, u);
                        ldg8(b + c, w);
#pragma unroll
                        for (int k = 0; k < 8; k += 2) {
                            const float t0 = u[k] - w[k], t1 = u[k + 1] - w[k + 1];
                            s0 = fmaf(t0, t0, s0);
                            s1 = fmaf(t1, t1, s1);
                        }
                    }
                    return s0 + s1;
                });
        if (open) hit = recheck_decide(X, d, perm, T, R, mi, mj, mine, exact_runs);
        if (hit) {
            atomicAdd(&counts[mi], 1);
            if (bp.j & kBandBoth) atomicAdd(&counts[mj], 1);
            emit_pair(em, bp);
            ++hits;
        }
    }
    recheck_totals(st, hits, exact_runs);
}

}  // namespace

static float f32_down(double v) {
    float f = (float)v;
    if ((double)f > v) f = nextafterf(f, -INFINITY);
    return f;
}
static float f32_up(double v) {
    float f = (float)v;
    if ((double)f < v) f = nextafterf(f, INFINITY);
    return f;
}

void finish_recheck32(Recheck32& R) {
    R.f_sTlo = f32_down(R.sTlo);
    R.f_sThi = f32_up(R.sThi);
    // 4 units of FP64 rounding cover the evaluation of 1 -/+ c32 in FP64
    R.f_kin = f32_down((1.0 - R.c32) * (1.0 - 4 * kU));
    R.f_kout = f32_up((1.0 + R.c32) * (1.0 + 4 * kU));
    R.f_abs = f32_up(R.abs32 * (1.0 + 4 * kU));
}

int launch_band_recheck2(const double* X, uint64_t n, uint32_t d, const uint32_t* perm, double T,
                         const Recheck32& R, const BandPair* band, uint64_t nband, int32_t* counts,
                         DevStatus* st, const Emit* em, cudaStream_t s) {
    if (nband == 0) return EJOIN_OK;
    const Emit e = em ? *em : Emit{nullptr, 0, nullptr, 0, nullptr};
    if (R.ds % 8 || R.ds < d || (((uintptr_t)R.Xf | (uintptr_t)R.Xfb) & 31) ||
        (((uintptr_t)R.Xh | (uintptr_t)R.Xhb) & 15))
        return set_error(EJOIN_EINTERNAL, "recheck: coordinates misaligned");
    constexpr uint64_t kBlocks = 152ull * 64;
    // measured on GB300: a thread per pair wins below 64 coordinates (d = 26: 22.9
    // ms against 34.5 with eight lanes), eight lanes from there (d = 64: 0.64
    // against 0.69 ms; d = 128: 0.93 ms against 1.2 with a warp), and a warp beyond
    // 256 (d = 1024 after the FP8 screen: 11.0 ms against 12.1, and 8.3 streamed, as
    // above)
    if (R.ds < 64) {
        const unsigned blocks = (unsigned)std::min<uint64_t>((nband + 255) / 256, kBlocks / 2);
        band_recheck_thread_kernel<<<blocks, 256, 0, s>>>(X, d, perm, T, R, band, nband, n, counts, st, e);
    } else {
        // a warp walks its pairs one after the other, a gather's latency each, so a
        // small band is spread over 152 x 64 warps
        const uint32_t ppw = (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(1, nband / kBlocks));
        const uint64_t warps = (nband + ppw - 1) / ppw;
        // (FP16 copies come with rows of at most 1024 coordinates)
        const int nv = R.ds <= 256 || !R.Xh ? 0 : R.ds <= 512 ? 2 : 4;
        const unsigned blocks =
            (unsigned)std::min<uint64_t>((warps + 7) / 8, nv ? kStreamBlocks : kBlocks);
        if (R.Xh && R.ds > 1024) return set_error(EJOIN_EINTERNAL, "recheck: FP16 rows too long");
        auto fn = R.ds <= 256 ? band_recheck_warp_kernel<8>
                  : nv == 0   ? band_recheck_warp_kernel<32>
                  : nv == 2   ? band_recheck_warp_kernel<32, 2>
                              : band_recheck_warp_kernel<32, 4>;
        if (nv) {
            EJ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stream_smem(nv)));
            EJ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         cudaSharedmemCarveoutMaxShared));
        }
        fn<<<blocks, 256, stream_smem(nv), s>>>(X, d, perm, T, R, band, nband, ppw, n, counts, st, e);
    }
    EJ_CUDA(cudaGetLastError());
    note_launch();
    return EJOIN_OK;
}

int launch_direct_selfjoin(const double* X, uint64_t n, uint32_t d, double T, int32_t* counts,
                           const Emit* em, cudaStream_t s) {
    if (n == 0) return EJOIN_OK;
    uint64_t nT = (n + TB - 1) / TB;
    uint64_t tiles = nT * (nT + 1) / 2;
    uint64_t gx = tiles < 1048576ull ? tiles : 1048576ull;
    uint64_t gy = (tiles + gx - 1) / gx;
    if (gy > 65535)
        return set_error(EJOIN_EUNSUPPORTED, "direct join: %llu tile pairs exceed the grid",
                         (unsigned long long)tiles);
    const Emit e = em ? *em : Emit{nullptr, 0, nullptr, 0, nullptr};
    direct_selfjoin_kernel<<<dim3((unsigned)gx, (unsigned)gy), 256, 0, s>>>(X, n, d, T, nT, tiles,
                                                                            counts, e);
    EJ_CUDA(cudaGetLastError());
    note_launch();
    return EJOIN_OK;
}

int launch_direct_query(const double* X, uint64_t n, uint32_t d, double T, const uint64_t* rows,
                        uint64_t nq, int32_t* counts, cudaStream_t s, const double* Xq) {
    if (n == 0 || nq == 0) return EJOIN_OK;
    const uint64_t gx = (n + TB - 1) / TB;
    if (gx > 0x7fffffffull) return set_error(EJOIN_EUNSUPPORTED, "query grid too large");
    // the grid's y extent is limited: queries in chunks of 65535 tiles
    const uint64_t chunk = 65535ull * TB;
    for (uint64_t q0 = 0; q0 < nq; q0 += chunk) {
        const uint64_t m = std::min<uint64_t>(chunk, nq - q0);
        direct_query_kernel<<<dim3((unsigned)gx, (unsigned)((m + TB - 1) / TB)), 256, 0, s>>>(
            X, n, d, T, rows ? rows + q0 : nullptr, Xq ? Xq + q0 * (uint64_t)d : nullptr, m,
            counts + q0);
        EJ_CUDA(cudaGetLastError());
        note_launch();
    }
    return EJOIN_OK;
}

int launch_band_recheck(const double* X, uint64_t n, uint32_t d, const uint32_t* perm, double T,
                        const BandPair* band, uint64_t nband, int32_t* counts, DevStatus* st,
                        cudaStream_t s) {
    if (nband == 0) return EJOIN_OK;
    uint64_t blocks = (nband + 255) / 256;
    if (blocks > 0x7fffffffull) return set_error(EJOIN_EUNSUPPORTED, "band too large");
    band_recheck_kernel<<<(unsigned)blocks, 256, 0, s>>>(X, d, perm, T, band, nband, n, counts,
                                                         st);
    EJ_CUDA(cudaGetLastError());
    note_launch();
    return EJOIN_OK;
}

}  // namespace ejoin
