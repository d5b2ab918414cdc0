// 16-bit contraction for problems with few output tiles: one tile of 128 x 64 per cluster, its K range
// split over the CTAs of the cluster.
//
// The canonical problem of contraction.cuh in the row-staged output form (D[row*ldd + column], columns
// contiguous): channels-last convolutions (operand A plain or through an im2col-mode tensor map) and plain
// products with the operands exchanged. What bounds such a call is neither the tensor core nor HBM but the
// chain of one CTA: a 3x3 layer over 512 channels at 7 x 7 pixels is one row tile whose 72 k-blocks of 24 KB
// a single SM takes 270 ns each to fetch. Here S CTAs fetch num_kb / S each, every SM at its own rate; the
// fp32 partial tiles meet in distributed shared memory, where CTA r adds the S copies of rows
// r*128/S .. of the tile in rank order (the result does not depend on timing), applies alpha, beta, bias, residual
// and ReLU, and writes whole 128-byte lines. No scratch memory, no second launch.
// Measured: forward of one image through ResNet-50 594 -> 381 us (fifty such layers, 5 to 20 us each before).
//
// Roles: warps 0-3 read the accumulator (quadrant = warp), 4 TMA producer, 5 UMMA issuer and TMEM owner; all
// eight warps write the output.
#pragma once
#include "contraction.cuh"

namespace dlfb200 {

constexpr int kSplitThreads = 256;
constexpr int kSplitBN = 64;
constexpr int kSplitStageBytes = (kBM + kSplitBN) * 128;
constexpr int kSplitMaxStages = 8;
constexpr int kSplitMaxCtas = 8;                  // CTAs of a cluster (the portable limit)
constexpr int kSplitPartLd = kSplitBN + 4;        // floats between rows of the partial tile
constexpr int kSplitPartBytes = kBM * kSplitPartLd * 4;
constexpr int split_smem_bytes(int stages) {
    return 1024 + (stages * kSplitStageBytes > kSplitPartBytes ? stages * kSplitStageBytes : kSplitPartBytes);
}

namespace ptx {
__device__ __forceinline__ float4 ld_cluster_v4(uint32_t cluster_addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
    return v;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t cluster_addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
    return v;
}
__device__ __forceinline__ int ld_cluster_s32(uint32_t cluster_addr) {
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
    return v;
}
}  // namespace ptx

template <int OUT>
__global__ void __launch_bounds__(kSplitThreads, 1)
    contraction_split_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap tmA,
                             const __grid_constant__ CUtensorMap tmB, int S) {
    constexpr int BK = 64;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kSplitMaxStages];
    __shared__ __align__(8) uint64_t empty_bar[kSplitMaxStages];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int rank = S > 1 ? static_cast<int>(ptx::cluster_ctarank()) : 0;
    const uint32_t smem0 = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    const int num_kb = (p.K + BK - 1) / BK;
    const int kb0 = rank * num_kb / S, kb1 = (rank + 1) * num_kb / S;
    const int tile = blockIdx.x / S;
    const int per = p.tiles_m * p.tiles_n;
    const int b = tile / per;
    const int tn = (tile - b * per) / p.tiles_m, tm = tile - b * per - tn * p.tiles_m;
    const int m0 = tm * kBM, n0 = tn * kSplitBN;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < p.stages; ++s) {
            ptx::mbar_init(ptx::smem_u32(&full_bar[s]), 1u);
            ptx::mbar_init(ptx::smem_u32(&empty_bar[s]), 1u);
        }
        ptx::mbar_init(ptx::smem_u32(&done_bar), 1u);
        ptx::fence_mbar_init();
    }
    if (warp == 5) {
        __syncwarp();
        ptx::tmem_alloc(ptx::smem_u32(&tmem_slot), 64u);
        ptx::tmem_relinquish();
        ptx::launch_dependents();  // (in this warp, with the tensor memory in hand: see ptx.cuh)
    }
    if (warp == 4 && lane == 0) {
        ptx::tma_prefetch_desc(&tmA);
        ptx::tma_prefetch_desc(&tmB);
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
    volatile int* abort_p = &abort_flag;
    const long long wait_limit = p.wait_limit;
    // operand B (a convolution's filter bank) on its way into L2 while the kernel before this one finishes
    if (warp == 4 && ptx::elect_one()) {
        for (int kb = kb0; kb < kb1; ++kb) {
            const int bb = p.b.batch_stride ? b : 0;
            if (p.b.k_major) ptx::tma_prefetch_3d(&tmB, kb * BK, n0, bb);
            else ptx::tma_prefetch_3d(&tmB, n0, kb * BK, bb);
        }
    }
    __syncwarp();
    ptx::wait_for_dependencies();

    if (warp == 4) {
        // ------------------------------------------------------------ TMA producer
        const bool leader = ptx::elect_one();
        const int ba = p.a.batch_stride ? b : 0, bb = p.b.batch_stride ? b : 0;
        int cl_n = 0, cl_h = 0, cl_w = 0, cl_cb = 0, cl_kh = 0, cl_kw = 0;
        if (p.a_cl == 1) {  // base pixel of the tile's first filter window; tap and channel block of kb0
            cl_n = m0 / p.g.P;
            const int pp = m0 - cl_n * p.g.P;
            const int oh = pp / p.g.OW;
            cl_h = oh * p.g.sh - p.g.pad_t;
            cl_w = (pp - oh * p.g.OW) * p.g.sw - p.g.pad_l;
            const int tap = kb0 / p.cl_cblocks;
            cl_cb = kb0 - tap * p.cl_cblocks;
            cl_kh = tap / p.g.KW;
            cl_kw = tap - cl_kh * p.g.KW;
        }
        uint32_t s = 0, ph = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
            if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&empty_bar[s]), ph ^ 1u, abort_p, wait_limit))) break;
            const uint32_t bar = ptx::smem_u32(&full_bar[s]);
            const uint32_t sA = smem0 + s * kSplitStageBytes, sB = sA + kBM * 128;
            if (leader) {
                ptx::mbar_arrive_expect_tx(bar, kSplitStageBytes);
                if (p.a_cl == 1) {
                    ptx::tma_load_im2col_4d(sA, &tmA, bar, cl_cb * BK, cl_w, cl_h, cl_n,
                                            static_cast<unsigned short>(cl_kw * p.g.dw), static_cast<unsigned short>(cl_kh * p.g.dh));
                } else if (p.a.k_major) {
                    ptx::tma_load_3d(sA, &tmA, bar, kb * BK, m0, ba);
                } else {
                    ptx::tma_load_3d(sA, &tmA, bar, m0, kb * BK, ba);
                    ptx::tma_load_3d(sA + BK * 128, &tmA, bar, m0 + 64, kb * BK, ba);
                }
                if (p.b.k_major) ptx::tma_load_3d(sB, &tmB, bar, kb * BK, n0, bb);
                else ptx::tma_load_3d(sB, &tmB, bar, n0, kb * BK, bb);
            }
            __syncwarp();
            if (++cl_cb == p.cl_cblocks) {
                cl_cb = 0;
                if (++cl_kw == p.g.KW) {
                    cl_kw = 0;
                    ++cl_kh;
                }
            }
            if (++s == static_cast<uint32_t>(p.stages)) {
                s = 0;
                ph ^= 1u;
            }
        }
    } else if (warp == 5) {
        // ------------------------------------------------------------ UMMA issuer
        const uint32_t idesc = ptx::make_idesc(static_cast<uint32_t>(p.fmt), p.a.k_major ? 0u : 1u, p.b.k_major ? 0u : 1u, kBM, kSplitBN);
        const uint32_t a_step = (p.a.k_major ? 32u : 2048u) >> 4, b_step = (p.b.k_major ? 32u : 2048u) >> 4;
        const uint64_t da0 = ptx::make_smem_desc(smem0, p.a.k_major ? 16u : BK * 128u, 1024u, 2u);
        const uint64_t db0 = ptx::make_smem_desc(smem0 + kBM * 128, p.b.k_major ? 16u : BK * 128u, 1024u, 2u);
        uint32_t s = 0, ph = 0;
        bool ok = true;
        for (int kb = kb0; kb < kb1; ++kb) {
            if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&full_bar[s]), ph, abort_p, wait_limit))) {
                ok = false;
                break;
            }
            ptx::tc_fence_after();
            const uint32_t at = (s * kSplitStageBytes) >> 4;
            if (ptx::elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    ptx::umma_f16(tmem, da0 + (at + ks * a_step), db0 + (at + ks * b_step), idesc, (kb > kb0 || ks > 0) ? 1u : 0u);
                ptx::umma_commit(ptx::smem_u32(&empty_bar[s]));
            }
            __syncwarp();
            if (++s == static_cast<uint32_t>(p.stages)) {
                s = 0;
                ph ^= 1u;
            }
        }
        if (ok && !p.skip_tile_commit && ptx::elect_one()) ptx::umma_commit(ptx::smem_u32(&done_bar));
        __syncwarp();
    } else if (warp < 4) {
        // ------------------------------------------------------------ accumulator -> partial tile
        // (the operand ring is free by then: every copy into it has been consumed)
        if (__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&done_bar), 0u, abort_p, wait_limit))) {
            ptx::tc_fence_after();
            const uint32_t row = smem0 + static_cast<uint32_t>((warp * 32 + lane) * kSplitPartLd * 4);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t v[32];
                ptx::tmem_ld_32x32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + h * 32, v);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    st_shared_v4(row + (h * 32 + j) * 4, make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]));
            }
            ptx::tc_fence_before();
        }
    }
    __syncthreads();
    if (abort_flag) {
        // copies and UMMAs still in flight get time to land before shared and tensor memory are released
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        if (threadIdx.x == 0) atomicOr(p.status, DEV_STATUS_WAIT_TIMEOUT);
    }
    if (S > 1) ptx::cluster_sync();
    // (one lane per CTA of the cluster: the loads of the flags take one round trip, not S)
    int gave_up = abort_flag;
    if (S > 1) gave_up = lane < S ? ptx::ld_cluster_s32(ptx::map_to_cta(ptx::smem_u32(&abort_flag), lane)) : 0;
    const bool aborted = __any_sync(0xffffffffu, gave_up != 0);
    if (!aborted) {
        // ------------------------------------------------------------ rows rank*128/S.. : 8 columns per item
        const int r0 = rank * kBM / S, r1 = (rank + 1) * kBM / S;
        for (int id = threadIdx.x; id < (r1 - r0) * (kSplitBN / 8); id += kSplitThreads) {
            const int r = r0 + id / (kSplitBN / 8), c = (id % (kSplitBN / 8)) * 8;
            const int i = m0 + r, j = n0 + c;
            if (i >= p.M || j >= p.N) continue;
            const uint32_t at = smem0 + static_cast<uint32_t>((r * kSplitPartLd + c) * 4);
            // all copies are asked for before the first is added: a load from another SM takes several hundred clocks
            float4 lo[kSplitMaxCtas], hi[kSplitMaxCtas];
#pragma unroll
            for (int k = 0; k < kSplitMaxCtas; ++k) {
                if (k < S) {
                    const uint32_t from = S > 1 ? ptx::map_to_cta(at, k) : at;
                    lo[k] = ptx::ld_cluster_v4(from);
                    hi[k] = ptx::ld_cluster_v4(from + 16);
                }
            }
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < kSplitMaxCtas; ++k) {
                if (k < S) {
                    acc[0] += lo[k].x; acc[1] += lo[k].y; acc[2] += lo[k].z; acc[3] += lo[k].w;
                    acc[4] += hi[k].x; acc[5] += hi[k].y; acc[6] += hi[k].z; acc[7] += hi[k].w;
                }
            }
            constexpr int OES = 2;
            const long long o = static_cast<long long>(b) * p.d_batch_stride + static_cast<long long>(i) * p.ldd + j;
            char* dst = p.d + o * OES;
            uint4 cv = make_uint4(0u, 0u, 0u, 0u);
            const bool add = p.resid != nullptr || p.beta != 0.0f;
            const float beta = p.resid != nullptr ? 1.0f : p.beta;
            if (add) cv = *reinterpret_cast<const uint4*>(p.resid != nullptr ? p.resid + o * OES : dst);
            uint4 bv = make_uint4(0u, 0u, 0u, 0u);
            if (p.bias != nullptr) bv = *reinterpret_cast<const uint4*>(p.bias + static_cast<long long>(j) * OES);
            const char* cb = reinterpret_cast<const char*>(&cv);
            const char* bb = reinterpret_cast<const char*>(&bv);
            uint4 out;
            char* ob = reinterpret_cast<char*>(&out);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float v = p.alpha * acc[e];
                if (p.bias != nullptr) v += out_load<OUT>(bb + e * OES);
                if (add) v += beta * out_load<OUT>(cb + e * OES);
                if (p.relu) v = fmaxf(v, 0.0f);
                out_store<OUT>(ob + e * OES, v);
            }
            *reinterpret_cast<uint4*>(dst) = out;
        }
    }
    if (S > 1) ptx::cluster_sync();  // no CTA leaves while another still reads its partial tile
    if (warp == 5) {
        __syncwarp();
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, 64u);
    }
}

}  // namespace dlfb200
