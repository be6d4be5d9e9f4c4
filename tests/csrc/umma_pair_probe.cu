// umma_pair_probe.cu -- GPU self-test of the MMAs that two CTAs share (test only).
//
// A cluster of two CTAs computes one 256 x 256 FP32 tile D = A * B^T the way the join's
// Gram kernel does: every CTA loads its 128 rows of A and of B (K-major, 128-byte
// swizzle) by TMA, both CTAs' copies complete on rank 0's barrier, one lane of rank 0
// issues cta_group::2 MMAs with M = N = 256, and each CTA reads its own 128 rows from its
// tensor memory.  With the hi+lo split the products are issued in the join's order; the
// aug operands, if there are any, come last, from tiles that store_aug wrote.  All waits
// are bounded (umma_ptx.cuh).
#include <cuda_runtime.h>
#include <stdint.h>

#include "tmap.cuh"
#include "umma_ptx.cuh"

using namespace ejoin;

namespace {

constexpr uint32_t FULL = 0xffffffffu;
constexpr int SLAB = 128 * 128;  // 128 rows x 128 bytes
constexpr int AUG = 128 * 32;    // 128 rows x 32 bytes
constexpr int STAGE = 2 * SLAB;  // a slab of A, a slab of B
constexpr int MAX_SLABS = 6;

// vals: [256][32], the A side and the B side of a row.
__global__ void aug_kernel(const uint16_t* vals, uint16_t* Aug) {
    const uint32_t p = blockIdx.x * 128 + threadIdx.x;
    uint16_t v[32];
    for (int i = 0; i < 32; ++i) v[i] = vals[p * 32 + i];
    ptx::store_aug(Aug, p, v);
}

// slabs: K-slabs of the operands, hi slabs then (split) as many lo slabs.
__global__ void __launch_bounds__(128, 1)
    pair_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                const __grid_constant__ CUtensorMap taug, int slabs, int split, int aug, int fmt,
                float* D, DevStatus* st) {
    extern __shared__ uint8_t smraw[];
    uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
    uint8_t* sg = sm + slabs * STAGE;
    __shared__ uint64_t full, done;
    __shared__ uint32_t tmem_base;
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    const uint32_t rank = ptx::cluster_ctarank();
    if (warp == 0) {
        ptx::tmem_alloc<2>(&tmem_base, 256);
        ptx::tmem_relinquish<2>();
    }
    if (threadIdx.x == 0) {
        ptx::mbar_init(&full, 1);
        ptx::mbar_init(&done, 1);
        ptx::fence_barrier_init();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync();
    ptx::tc_fence_after();
    const uint32_t tmem = tmem_base;
    if (threadIdx.x == 0) {
        const uint32_t bar = ptx::mapa(&full, 0);
        const int ew = fmt == 2 ? 128 : 64;  // elements per 128-byte row
        if (rank == 0)
            ptx::mbar_arrive_expect_tx(&full, 2u * (slabs * STAGE + (aug ? 2 * AUG : 0)));
        for (int s = 0; s < slabs; ++s) {
            ptx::tma_load_2d_pair(sm + s * STAGE, &ta, s * ew, (int32_t)(rank * 128), bar);
            ptx::tma_load_2d_pair(sm + s * STAGE + SLAB, &tb, s * ew, (int32_t)(rank * 128), bar);
        }
        if (aug) {
            ptx::tma_load_2d_pair(sg, &taug, 0, (int32_t)(rank * 64), bar);
            ptx::tma_load_2d_pair(sg + AUG, &taug, 0, (int32_t)(rank * 64 + 32), bar);
        }
    }
    __syncthreads();
    if (rank == 0 && warp == 1) {
        const bool ok = __all_sync(FULL, ptx::mbar_wait(&full, 0, st, 1));
        ptx::tc_fence_after();
        if (ok && ptx::elect_one()) {
            const uint32_t idesc = fmt == 2 ? ptx::idesc_f32acc(0, 0, 256, 256)
                                            : ptx::idesc_f32acc(fmt, fmt, 256, 256);
            const uint32_t idesc_aug = fmt == 2 ? ptx::idesc_f32acc(1, 1, 256, 256) : idesc;
            const uint64_t d0 = ptx::sdesc_sw128(ptx::smem_u32(sm));
            auto mma = [&](int sa, int sb, int kk, uint32_t acc) {
                const uint64_t a = d0 + (uint64_t)(sa * (STAGE >> 4) + 2 * kk);
                const uint64_t b = d0 + (uint64_t)(sb * (STAGE >> 4) + (SLAB >> 4) + 2 * kk);
                if (fmt == 2) ptx::mma_f8<2>(tmem, a, b, idesc, acc);
                else ptx::mma_f16<2>(tmem, a, b, idesc, acc);
            };
            const int nhi = split ? slabs / 2 : slabs;
            for (int c = 0; c < nhi; ++c) {
                if (split)
                    for (int kk = 0; kk < 4; ++kk) {
                        mma(c, nhi + c, kk, (c | kk) != 0);
                        mma(nhi + c, c, kk, 1);
                    }
                for (int kk = 0; kk < 4; ++kk) mma(c, c, kk, split || (c | kk) != 0);
            }
            if (aug) {
                const uint64_t g = ptx::sdesc_sw32(ptx::smem_u32(sg));
                ptx::mma_f16<2>(tmem, g, g + (AUG >> 4), idesc_aug, 1);
            }
            ptx::mma_commit<2>(&done);
        }
        __syncwarp();
    }
    if (__all_sync(FULL, ptx::mbar_wait(&done, 0, st, 2))) {
        ptx::tc_fence_after();
        for (uint32_t c = 0; c < 8; ++c) {
            uint32_t r[32];
            ptx::tmem_ld_32x32b_x32(tmem + ((warp * 32) << 16) + 32 * c, r);
            ptx::tmem_ld_wait();
            float* row = D + (size_t)(rank * 128 + warp * 32 + lane) * 256 + 32 * c;
            for (int j = 0; j < 32; ++j) row[j] = __uint_as_float(r[j]);
        }
    } else if (rank == 0 && threadIdx.x == 0) {
        ptx::mbar_wait_drain(&full, 0);  // the copies of both CTAs
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync();
    if (warp == 0) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc<2>(tmem, 256);
    }
}

}  // namespace

// A, B: 256 rows of `slabs` x 128 bytes; fmt 0 FP16, 1 BF16, 2 E4M3; aug (or null):
// [256][32] 16-bit values, the A and the B side of every row (BF16 with E4M3).
// D: [256][256].  0, or negative.
extern "C" int umma_pair_probe(const void* A, const void* B, int slabs, int fmt, int split,
                               const uint16_t* aug, float* D, unsigned* timeout_out) {
    if (slabs < 1 || slabs > MAX_SLABS || fmt < 0 || fmt > 2 || (split && (fmt == 2 || slabs % 2)))
        return -1;
    const size_t bytes = (size_t)256 * 128 * slabs, dbytes = (size_t)256 * 256 * sizeof(float);
    void *dA = nullptr, *dB = nullptr;
    uint16_t *dv = nullptr, *dg = nullptr;
    float* dD = nullptr;
    DevStatus* dst = nullptr;
    DevStatus hst = {};
    CUtensorMap ma, mb, mg;
    int rc = 0;
    const uint32_t es = fmt == 2 ? 1 : 2;
    const CUtensorMapDataType dt = fmt == 2   ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                   : fmt == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                              : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUtensorMapDataType gt = fmt == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const size_t smem = 1024 + (size_t)slabs * STAGE + 2 * AUG;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = {};
    if (cudaMalloc(&dA, bytes) || cudaMalloc(&dB, bytes) || cudaMalloc(&dD, dbytes) ||
        cudaMalloc(&dv, 256 * 64) || cudaMalloc(&dg, 256 * 64) || cudaMalloc(&dst, sizeof(DevStatus))) {
        rc = -2;
        goto done;
    }
    cudaMemcpy(dA, A, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(dB, B, bytes, cudaMemcpyHostToDevice);
    cudaMemset(dD, 0, dbytes);
    cudaMemset(dg, 0, 256 * 64);
    cudaMemset(dst, 0, sizeof(DevStatus));
    if (aug) {
        cudaMemcpy(dv, aug, 256 * 64, cudaMemcpyHostToDevice);
        aug_kernel<<<2, 128>>>(dv, dg);
    }
    if (make_tmap_2d(&ma, dA, dt, es, (uint64_t)slabs * 128 / es, 256, 128 / es, 128) ||
        make_tmap_2d(&mb, dB, dt, es, (uint64_t)slabs * 128 / es, 256, 128 / es, 128) ||
        make_tmap_2d(&mg, dg, gt, 2, 64, 128, 64, 32, false)) {
        rc = -3;
        goto done;
    }
    if (cudaFuncSetAttribute(pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) {
        rc = -4;
        goto done;
    }
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, pair_kernel, ma, mb, mg, slabs, split, aug ? 1 : 0, fmt, dD, dst) ||
        cudaDeviceSynchronize()) {
        cudaGetLastError();
        rc = -5;
        goto done;
    }
    cudaMemcpy(D, dD, dbytes, cudaMemcpyDeviceToHost);
    cudaMemcpy(&hst, dst, sizeof hst, cudaMemcpyDeviceToHost);
    if (timeout_out) *timeout_out = hst.timeout;
    if (hst.timeout) rc = -6;
done:
    cudaFree(dA);
    cudaFree(dB);
    cudaFree(dD);
    cudaFree(dv);
    cudaFree(dg);
    cudaFree(dst);
    return rc;
}
