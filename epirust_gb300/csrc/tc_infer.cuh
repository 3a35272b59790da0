// tc_infer.cuh -- the surrogate's inference products on the sm_103a tensor cores.
//
// A screen multiplies tens of thousands of rows per member.  Bias, GELU and rounding take 32
// warp instructions per 32 elements (erff most of them), 143 us of every scheduler's issue
// slots for a hidden layer of 65,536 rows x 5 members whose products are 80 us of tensor
// cores; so the products have to run under the epilogue.  k_infer is persistent, one CTA per SM:
//   warps 0..15  epilogue: a warp owns 32 rows x 32 columns of each 128 x 128 block
//   warp 16      TMA: the item's A panel (128 rows, all of K, resident for all of the item's
//                columns), and the weight blocks through a ring
//   warp 17      tcgen05.mma into two accumulators in tensor memory: a tile multiplies while
//                the one before it is in the epilogue
// An item is 128 rows of one member and a run of column blocks.  Where the rows fill the SMs it
// takes all of them, two at a time (N = 256 per MMA: half the waits and commits per product);
// otherwise (a few hundred rows, where latency counts) one block, so that more SMs share them.
// Every wait is bounded as in k_gemm; a role that gives up flags it, the others run into their
// own bounds, and the copies and MMAs still in flight are waited for before the CTA exits.
//
// Measured on one GB300, 65,536 rows x 5 members, us per launch (K = 64 -> 512, 512 -> 512,
// 512 -> 640 with the score): a tile per CTA with three CTAs per SM (k_gemm) 218, 322, 250;
// persistent with N = 128, 4 ring blocks and 16-byte stores 188, 235, 210; N = 256, 6 blocks and
// 32-byte stores 172, 206, 161.  1,024 rows x 5 members, one block per item: 12 to 14 us a
// launch.  What bounds it now: the epilogue's issue slots, 70 % busy.
#pragma once

#include "tc_gemm.cuh"

namespace epi {
namespace tc {

constexpr int kInferBN = 128;
constexpr uint32_t kInferAcc = 2u * kInferBN;  // columns of an accumulator
constexpr uint32_t kInferMaxK = 8;             // K blocks of 64 that a resident A panel may have
constexpr uint32_t kInferRing = 6;             // weight blocks in the ring (2-block stages: 3; 4 blocks 3 % slower)
constexpr int kInferEpilogueWarps = 16;
constexpr int kInferThreads = (kInferEpilogueWarps + 2) * 32;
constexpr uint32_t kInferBlock = kBM * kBK * 2;  // a 128 x 64 block of A or of the weights
constexpr uint32_t infer_smem(uint32_t nk) { return (nk + kInferRing) * kInferBlock + 1024u; }

struct InferBars {
    uint64_t a_full[kInferMaxK], a_empty[kInferMaxK];
    uint64_t b_full[kInferRing], b_empty[kInferRing];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem, a_issued, b_issued, bad;
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

// One whole 32-byte sector: lanes hold rows, so narrower stores would each write parts of 32.
__device__ __forceinline__ void store_32b(void* p, const uint32_t v[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

__device__ __forceinline__ void load_row32(const float* p, float v[32]) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float4 b = __ldg(reinterpret_cast<const float4*>(p) + q);
        v[4 * q] = b.x;
        v[4 * q + 1] = b.y;
        v[4 * q + 2] = b.z;
        v[4 * q + 3] = b.w;
    }
}

// Row m, columns n .. n + 31.
template <int EP>
__device__ __forceinline__ void infer_epilogue(const EpiArgs& a, uint32_t N, uint32_t m, uint32_t n, float x[32],
                                               const float bias[32], float& ssum) {
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] += bias[j];
    if (EP == kEpHidden) {
        __nv_bfloat16* o = a.out + (size_t)m * N + n;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            uint32_t h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const __nv_bfloat162 p = __floats2bfloat162_rn(gelu(x[16 * q + 2 * j]), gelu(x[16 * q + 2 * j + 1]));
                h[j] = *reinterpret_cast<const uint32_t*>(&p);
            }
            store_32b(o + 16 * q, h);
        }
        return;
    }
    if (a.outf && m < a.m_valid) {
        float* o = a.outf + (size_t)m * a.ld_outf + n;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (n + 8 * q < a.n_valid) store_32b(o + 8 * q, reinterpret_cast<const uint32_t*>(x + 8 * q));
    }
    if (a.score_target) {  // (padded to N: the bound only keeps the padding out of the sum)
        const float4* target = reinterpret_cast<const float4*>(a.score_target + n);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float4 t = __ldg(target + q);
            const float e[4] = {x[4 * q] - t.x, x[4 * q + 1] - t.y, x[4 * q + 2] - t.z, x[4 * q + 3] - t.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + 4 * q + j < a.n_valid) ssum += e[j] * e[j];
        }
    }
}

// Items i = blockIdx.x, + gridDim.x, ...: i = (member * M / 128 + row tile) * groups + group,
// a group being `run` column blocks, multiplied `wide` (1 or 2) at a time.  M % 128 == 0,
// N % 128 == 0, nk = K / 64 <= kInferMaxK (checked by the host).
template <int EP>
__global__ void __launch_bounds__(kInferThreads, 1)
    k_infer(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, uint32_t M, uint32_t N, uint32_t nk,
            uint32_t wide, uint32_t run, uint32_t items, const __grid_constant__ EpiArgs margs, uint32_t za, int* err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* panel = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* ring = panel + nk * kInferBlock;
    __shared__ __align__(8) InferBars b;
    const uint32_t stages = kInferRing / wide;
    const uint32_t warp = uniform_warp(), lane = threadIdx.x & 31u;
    const uint32_t row_tiles = M / kBM, blocks = N / kInferBN, groups = (blocks + run - 1) / run;

    if (threadIdx.x == 0) {
        for (uint32_t k = 0; k < kInferMaxK; ++k) {
            mbar_init(&b.a_full[k], 1);
            mbar_init(&b.a_empty[k], 1);
        }
        for (uint32_t s = 0; s < kInferRing; ++s) {
            mbar_init(&b.b_full[s], 1);
            mbar_init(&b.b_empty[s], 1);
        }
        for (int k = 0; k < 2; ++k) {
            mbar_init(&b.acc_full[k], 1);
            mbar_init(&b.acc_empty[k], kInferEpilogueWarps);
        }
        b.a_issued = b.b_issued = b.bad = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&b.tmem)),
                     "r"(2u * kInferAcc)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = b.tmem;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the inputs are the kernel before's outputs

    if (warp == kInferEpilogueWarps) {  // TMA
        asm volatile("fence.proxy.async;" ::: "memory");
        const bool lead = elect_one();
        uint32_t s = 0, round = 0, a_issued = 0, b_issued = 0;
        bool ok = true;
        for (uint32_t i = blockIdx.x, it = 0; i < items && ok; i += gridDim.x, ++it) {
            const uint32_t g = i % groups, mt = i / groups % row_tiles, e = i / groups / row_tiles;
            const uint32_t first = g * run, last = min(first + run, blocks);
            for (uint32_t t = first; t < last && ok; t += wide)
                for (uint32_t kb = 0; kb < nk && ok; ++kb) {
                    if (t == first) {  // the panel's block kb, once its last reader has gone
                        if (it > 0) ok = warp_wait(&b.a_empty[kb], (it - 1u) & 1u);
                        if (!ok) break;
                        if (lead) {
                            mbar_expect_tx(&b.a_full[kb], kInferBlock);
                            tma_load_3d(panel + kb * kInferBlock, &ta, (int32_t)(kb * kBK), (int32_t)(mt * kBM),
                                        (int32_t)(e * za), &b.a_full[kb]);
                        }
                        ++a_issued;
                    }
                    if (round > 0) ok = warp_wait(&b.b_empty[s], (round - 1u) & 1u);
                    if (!ok) break;
                    if (lead) {
                        const uint32_t w = min(wide, last - t);
                        mbar_expect_tx(&b.b_full[s], w * kInferBlock);
                        for (uint32_t q = 0; q < w; ++q)
                            tma_load_3d(ring + (s * wide + q) * kInferBlock, &tb, (int32_t)(kb * kBK),
                                        (int32_t)((t + q) * kInferBN), (int32_t)e, &b.b_full[s]);
                    }
                    ++b_issued;
                    if (++s == stages) { s = 0; ++round; }
                }
        }
        if (lead) {
            b.a_issued = a_issued;
            b.b_issued = b_issued;
            if (!ok) {
                atomicOr(err, 1);
                b.bad = 1;
            }
        }
    } else if (warp == kInferEpilogueWarps + 1) {  // MMA
        const uint64_t da = smem_desc(smem_u32(panel)), db = smem_desc(smem_u32(ring));
        const bool lead = elect_one();
        uint32_t s = 0, round = 0, tile = 0, used = 0;
        bool ok = true;
        for (uint32_t i = blockIdx.x, it = 0; i < items && ok; i += gridDim.x, ++it) {
            const uint32_t first = i % groups * run, last = min(first + run, blocks);
            for (uint32_t t = first; t < last && ok; t += wide, ++tile) {
                const uint32_t idesc = instr_desc(kBM, kInferBN * min(wide, last - t));
                const uint32_t buf = tile & 1u;
                if (tile >= 2u) ok = warp_wait(&b.acc_empty[buf], ((tile >> 1) - 1u) & 1u);
                if (!ok) break;
                tc_fence_after();
                for (uint32_t kb = 0; kb < nk; ++kb) {
                    ok = (t != first || warp_wait(&b.a_full[kb], it & 1u)) && warp_wait(&b.b_full[s], round & 1u);
                    if (!ok) break;
                    tc_fence_after();
                    if (lead) {
                        const uint64_t oa = da + (uint64_t)(kb * (kInferBlock >> 4)), ob = db + (uint64_t)(s * wide * (kInferBlock >> 4));
#pragma unroll
                        for (int j = 0; j < kBK / 16; ++j)  // K = 16 per MMA: advance 32 bytes within the swizzled row
                            mma_bf16(tmem + buf * kInferAcc, oa + 2u * j, ob + 2u * j, idesc, (kb | (uint32_t)j) != 0u);
                        mma_commit(&b.b_empty[s]);
                        if (t + wide >= last) mma_commit(&b.a_empty[kb]);
                    }
                    __syncwarp();
                    ++used;
                    if (++s == stages) { s = 0; ++round; }
                }
                if (lead && ok) mma_commit(&b.acc_full[buf]);
                __syncwarp();
            }
        }
        if (!ok && lead) {
            atomicOr(err, 1);
            b.bad = 1;
        }
        // every MMA issued has completed before the CTA goes on to free anything (bounded)
        if (used > 0) warp_wait(&b.b_empty[(used - 1u) % stages], ((used - 1u) / stages) & 1u);
    } else {  // epilogue
        const uint32_t row = (warp & 3u) * 32u, col = (warp >> 2) * 32u;
        uint32_t tile = 0;
        bool ok = true;
        for (uint32_t i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const uint32_t g = i % groups, mt = i / groups % row_tiles, e = i / groups / row_tiles;
            const EpiArgs a = member_args(margs, e);
            const uint32_t m = mt * kBM + row + lane;
            float ssum = 0.f;
            const uint32_t first = g * run, last = min(first + run, blocks);
            for (uint32_t t = first; t < last; t += wide, ++tile) {
                const uint32_t buf = tile & 1u, w = min(wide, last - t);
                float bias[32];
                load_row32(a.bias + t * kInferBN + col, bias);  // under the wait for the product
                ok = warp_wait(&b.acc_full[buf], (tile >> 1) & 1u);
                if (!ok) break;
                tc_fence_after();
                for (uint32_t q = 0; q < w; ++q) {
                    const uint32_t n = (t + q) * kInferBN + col;
                    float v[32];
                    tmem_ld32(tmem + buf * kInferAcc + (row << 16) + q * kInferBN + col, v);
                    if (q > 0) load_row32(a.bias + n, bias);
                    if (q + 1 == w) {
                        tc_fence_before();
                        if (lane == 0) mbar_arrive(&b.acc_empty[buf]);  // in registers: the tensor core may write on
                    }
                    infer_epilogue<EP>(a, N, m, n, v, bias, ssum);
                }
            }
            if (EP == kEpOut && a.score && ok && m < a.m_valid) atomicAdd(a.score + m, ssum);
        }
        if (!ok && lane == 0) {
            atomicOr(err, 2);
            b.bad = 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (b.bad && threadIdx.x == 0) {  // copies may still be in flight: wait (bounded) for the last of every block
        for (uint32_t q = b.a_issued > nk ? b.a_issued - nk : 0u; q < b.a_issued; ++q)
            mbar_wait(&b.a_full[q % nk], (q / nk) & 1u);
        for (uint32_t q = b.b_issued > stages ? b.b_issued - stages : 0u; q < b.b_issued; ++q)
            mbar_wait(&b.b_full[q % stages], (q / stages) & 1u);
    }
    __syncwarp();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * kInferAcc) : "memory");
}

}  // namespace tc
}  // namespace epi
