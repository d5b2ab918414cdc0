// fp32 contraction fed by TMA on both sides (3xTF32, operand A in tensor memory).
//
// The canonical problem of contraction.cuh for fp32 operands that satisfy the TMA rules:
//     D[i + j*ldd] = alpha * sum_k Au(i,k) * Bu(j,k) + beta * D[i + j*ldd] (+ bias[j])
// Every k-block of 32 k arrives raw, by TMA, in shared memory. Four splitter warps read their row
// of A, split each value into tf32 hi (round to nearest) and lo, and put both into tensor memory;
// two converter warps write lo = x - trunc(x) beside the raw tile of B, which the tensor core reads as the
// tf32 truncation of itself. Three UMMAs per k-step accumulate lo*hi + hi*lo + hi*hi. A value of B is then known to
// 2^-21 of itself, one of A to 2^-23. Where this kernel stands in for one that rounds both parts of B too - the filters of
// 1x1 convolutions, B operands off 16-byte boundaries - it does the same: with F32_B_ROUND the converters write hi over
// the raw tile as well, with F32_B_SPLIT hi and lo are two matrices that a copy has written (pad_lines_kernel) and
// TMA fetches both. Rounding in the kernel is for launches that walk a dozen k-blocks in a row or fewer, which another
// launch would cost more (64 -> 64 channels, 64 images of 8 x 8: 5.8 us truncated, 5.9 rounded here); over more the converters are
// too slow for it (256 -> 256, 64 images of 56 x 56: 150 us truncated, 196 rounded here, 143 from two matrices).
// The tensor core truncates when it adds into its accumulator, so it gets chunks of 8 k-blocks; eight
// epilogue warps add the finished chunks with rounding to nearest, in registers (32 x 32*NB values per warp).
//
// What bounds it: the UMMA's issue interval at 64 and 128 columns (12 per k-block: 1020 and 1380 clocks), the
// shared-memory port at 192: 25 KB of B in, 49 KB through the converters, 74 KB into the tensor core and 32 KB of
// A in and out per k-block, 1400 clocks at 128 bytes each against 1152 of tensor work; 1750 measured. Running sums in
// shared memory would add 25 KB. CTA pairs (cta_group::2, half of B per CTA: 105 KB) were slower all the same,
// 200 against 233 TFLOP/s at 4096^3: the hand-shakes of two A slots across the pair take longer than a k-block.
// Measured against the general kernel: 4096^3 1000 -> 585 us (235 TFLOP/s, 0.89 of a sixth of the 16-bit peak),
// 16384^3 60.3 -> 41.0 ms, 2048^3 148 -> 91 us, 1024^3 33 -> 21 us, 512^3 14.5 -> 10.5 us. Relative error 1.9e-6 at any
// K (3.7e-6 at K = 1024 in one chunk before).
//
// Roles: warps 0-7 epilogue (two sets of columns, quadrant = warp & 3), 8-11 splitters, 12 TMA producer,
// 13 UMMA issuer and TMEM owner, 14-15 converters.
#pragma once
#include "contraction_split.cuh"
#include "contraction_ts.cuh"

namespace dlfb200 {

constexpr int kF32Threads = 512;
constexpr int kF32ChunkBlocks = 8;  // k-blocks per accumulator (256 k)
constexpr int kF32MaxStages = 6;
enum : int { F32_B_TRUNCATE = 0, F32_B_ROUND = 1, F32_B_SPLIT = 2 };  // Params::b_parts
constexpr int f32_stage_bytes(int nb) { return kBM * 128 + 2 * 64 * nb * 128; }

// Element offset of row i of D: i, or, for the rows of a convolution over the pixels of all images (out_nchw), the
// pixel's place in an NCHW tensor.
__device__ __forceinline__ long long f32_row_offset(const Params& p, int i) {
    if (!p.out_nchw) return i;
    const int img = i / p.g.P;
    return static_cast<long long>(img) * p.g.out_img_stride + (i - img * p.g.P);
}

// X (N, C, H, W) -> X' (N * OH * OW, C): the pixels a 1x1 filter's strides keep, channels contiguous, for planes or
// strides the tensor maps cannot address. HBM-bound; a 32 x 32 tile turns in shared memory.
// grid: (pixel blocks, channel blocks, images); block: 256 threads.
__global__ void __launch_bounds__(256)
    f32_pack_pixels_kernel(const float* __restrict__ x, float* __restrict__ xp, int C, long long plane, int W, int P, int OW,
                           int sh, int sw) {
    __shared__ float tile[32][33];
    ptx::launch_dependents();
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int p0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const long long img = blockIdx.z;
    const int pix = p0 + lane, oh = pix / OW;
    const float* src = x + img * C * plane + static_cast<long long>(oh) * sh * W + (pix - oh * OW) * sw;
#pragma unroll
    for (int i = 0; i < 32; i += 8)
        if (pix < P && c0 + row + i < C) tile[row + i][lane] = src[(c0 + row + i) * plane];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 32; i += 8)
        if (p0 + row + i < P && c0 + lane < C) xp[(img * P + p0 + row + i) * C + c0 + lane] = tile[lane][row + i];
}

// A CTA has tiles of 128 x 64*NB, or, split > 1, the `split` CTAs of a cluster share one tile, each with its part of the
// k-blocks: for products with few tiles. The partial tiles then meet in distributed shared memory (the operand ring,
// free by then, as [column][row]), where CTA r adds up columns r*BN/split .. in rank order and writes them.
template <int NB>
__global__ void __launch_bounds__(kF32Threads, 1)
    contraction_f32_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap tmA,
                           const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmBlo, int split) {
    constexpr int BN = 64 * NB;
    constexpr int BK = 32;
    constexpr uint32_t A_TILE = kBM * 128;
    constexpr uint32_t B_TILE = BN * 128;
    constexpr uint32_t STAGE = A_TILE + 2 * B_TILE;
    constexpr int SLOTS = NB >= 3 ? 2 : 4;  // A slots in tensor memory
    constexpr uint32_t A_COL0 = 2 * BN;
    static_assert(A_COL0 + SLOTS * 64 <= 512, "two accumulators and the A slots share 512 columns");

    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t raw_full[kF32MaxStages];   // tiles of A and B landed
    __shared__ __align__(8) uint64_t raw_empty[kF32MaxStages];  // splitters and UMMAs are done with the stage
    __shared__ __align__(8) uint64_t conv_full[kF32MaxStages];  // lo image of B written
    __shared__ __align__(8) uint64_t slot_full[SLOTS];          // hi and lo of A in tensor memory
    __shared__ __align__(8) uint64_t slot_empty[SLOTS];
    __shared__ __align__(8) uint64_t tfull_bar[2];
    __shared__ __align__(8) uint64_t tempty_bar[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int part = split == 1 ? 0 : static_cast<int>(ptx::cluster_ctarank());
    const int S = p.stages;
    const uint32_t smem0 = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    const int all_kb = (p.K + BK - 1) / BK;
    const int kb_begin = part * all_kb / split;
    const int num_kb = (part + 1) * all_kb / split - kb_begin;
    const int tile0 = blockIdx.x / split;  // (split: one tile per cluster)

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < kF32MaxStages; ++s) {
            ptx::mbar_init(ptx::smem_u32(&raw_full[s]), 1u);
            ptx::mbar_init(ptx::smem_u32(&raw_empty[s]), 4u + 1u);
            ptx::mbar_init(ptx::smem_u32(&conv_full[s]), 2u);
        }
        for (int s = 0; s < SLOTS; ++s) {
            ptx::mbar_init(ptx::smem_u32(&slot_full[s]), 4u);
            ptx::mbar_init(ptx::smem_u32(&slot_empty[s]), 1u);
        }
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(ptx::smem_u32(&tfull_bar[i]), 1u);
            ptx::mbar_init(ptx::smem_u32(&tempty_bar[i]), 8u);
        }
        ptx::fence_mbar_init();
    }
    if (warp == 13) {
        __syncwarp();
        ptx::tmem_alloc(ptx::smem_u32(&tmem_slot), 512u);
        ptx::tmem_relinquish();
        ptx::launch_dependents();  // (in this warp, with the tensor memory in hand: see ptx.cuh)
    }
    if (warp == 12 && lane == 0) {
        ptx::tma_prefetch_desc(&tmA);
        ptx::tma_prefetch_desc(&tmB);
        ptx::tma_prefetch_desc(&tmBlo);
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
    volatile int* abort_p = &abort_flag;
    const long long wait_limit = p.wait_limit;
    ptx::wait_for_dependencies();
    // the launch has 512 x 128 registers: 2 x 176 + 96 + 64 = 4 x 128
    if (warp < 8) asm volatile("setmaxnreg.inc.sync.aligned.u32 176;");
    else if (warp < 12) asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");

    if (warp < 8) {
        // ------------------------------------------------------------ epilogue
        const int q = warp & 3, set = warp >> 2;
        const int cbase = set * 32 * NB;
        const uint32_t trow = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + cbase;
        uint32_t buf = 0, tphase = 0;
        bool alive = true;
        for (int t = tile0; alive && t < p.total_tiles; t += gridDim.x) {
            int b, m0, n0;
            decode_tile(p, t, b, m0, n0);
            const int i = m0 + q * 32 + lane;
            const bool row_ok = i < p.M;
            float sum[NB][32];
            for (int kb0 = 0; kb0 < num_kb; kb0 += kF32ChunkBlocks) {
                if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&tfull_bar[buf]), tphase, abort_p, wait_limit))) {
                    alive = false;
                    break;
                }
                ptx::tc_fence_after();
#pragma unroll
                for (int blk = 0; blk < NB; ++blk) {
                    uint32_t v[32];
                    ptx::tmem_ld_32x32(trow + buf * BN + blk * 32, v);
                    ptx::tmem_ld_wait();
                    if (kb0 == 0) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) sum[blk][j] = __uint_as_float(v[j]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) sum[blk][j] += __uint_as_float(v[j]);
                    }
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&tempty_bar[buf]));
                buf ^= 1u;
                if (buf == 0) tphase ^= 1u;
            }
            if (!alive) break;
            if (split > 1) {
                const uint32_t at = smem0 + static_cast<uint32_t>((cbase * kBM + q * 32 + lane) * 4);
#pragma unroll
                for (int blk = 0; blk < NB; ++blk)
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (blk * 32 + j) * (kBM * 4)), "f"(sum[blk][j]) : "memory");
                break;
            }
            EpiExtra ex;
            ex.relu = p.relu != 0;
            ex.rdelta = p.resid ? p.resid - p.d : 0;
            const float beta = p.resid ? 1.0f : p.beta;
            const long long stride = p.ldd * 4;
            char* optr = p.d + (static_cast<long long>(b) * p.d_batch_stride + f32_row_offset(p, i) + static_cast<long long>(n0 + cbase) * p.ldd) * 4;
            const char* bias = p.bias != nullptr ? p.bias + static_cast<long long>(n0 + cbase) * 4 : nullptr;
#pragma unroll
            for (int blk = 0; blk < NB; ++blk) {
                const int ncols = min(32, p.N - n0 - cbase - blk * 32);
                if (ncols <= 0) break;
                uint32_t v[32];
                if (bias != nullptr) {
                    const float bv = lane < ncols ? reinterpret_cast<const float*>(bias)[blk * 32 + lane] : 0.0f;
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(sum[blk][j] + __shfl_sync(0xffffffffu, bv, j));  // (alpha == 1)
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(sum[blk][j]);
                }
                char* ptr = optr + blk * 32 * stride;
                if (beta != 0.0f) epilogue_chunk<OUT_F32, true, false>(v, ptr, stride, ncols, row_ok, p.alpha, beta, nullptr, lane, false, ex);
                else epilogue_chunk<OUT_F32, false, false>(v, ptr, stride, ncols, row_ok, p.alpha, beta, nullptr, lane, false, ex);
            }
        }
    } else if (warp < 12) {
        // ------------------------------------------------------------ splitters: rows of A -> tensor memory
        const int q = warp & 3;
        const int L = q * 32 + lane;
        uint32_t s = 0, ph = 0, slot = 0, sph = 0;
        bool ok = true;
        for (int t = tile0; ok && t < p.total_tiles; t += gridDim.x) {
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&raw_full[s]), ph, abort_p, wait_limit))) {
                    ok = false;
                    break;
                }
                const uint32_t sA = smem0 + s * STAGE;
                uint32_t hi[32], lo[32];
                if (p.a.k_major) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const uint4 u = ld_shared_v4(sA + L * 128u + ((c ^ (L & 7)) << 4));
                        hi[4 * c + 0] = u.x;
                        hi[4 * c + 1] = u.y;
                        hi[4 * c + 2] = u.z;
                        hi[4 * c + 3] = u.w;
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 32; ++k)
                        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(hi[k]) : "r"(sA + k * (kBM * 4) + L * 4) : "memory");
                }
                // (4096^3 7 % slower with the conversion instructions of split_tf32)
#pragma unroll
                for (int k = 0; k < 32; ++k) split_tf32_int(hi[k], hi[k], lo[k]);
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&raw_empty[s]));
                if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&slot_empty[slot]), sph ^ 1u, abort_p, wait_limit))) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                const uint32_t at = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + A_COL0 + slot * 64;
                tmem_st_32x32(at, hi);
                tmem_st_32x32(at + 32, lo);
                tmem_st_wait();
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&slot_full[slot]));
                if (++s == static_cast<uint32_t>(S)) {
                    s = 0;
                    ph ^= 1u;
                }
                if (++slot == SLOTS) {
                    slot = 0;
                    sph ^= 1u;
                }
            }
        }
    } else if (warp == 12) {
        // ------------------------------------------------------------ TMA producer
        const bool leader = ptx::elect_one();
        const bool presplit = p.b_parts == F32_B_SPLIT;
        uint32_t s = 0, ph = 0;
        bool ok = true;
        for (int t = tile0; ok && t < p.total_tiles; t += gridDim.x) {
            int b, m0, n0;
            decode_tile(p, t, b, m0, n0);
            const int ba = p.a.batch_stride ? b : 0, bb = p.b.batch_stride ? b : 0;
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&raw_empty[s]), ph ^ 1u, abort_p, wait_limit))) {
                    ok = false;
                    break;
                }
                const uint32_t bar = ptx::smem_u32(&raw_full[s]);
                const uint32_t sA = smem0 + s * STAGE, sB = sA + A_TILE;
                if (leader) {
                    ptx::mbar_arrive_expect_tx(bar, presplit ? A_TILE + 2 * B_TILE : A_TILE + B_TILE);
                    if (p.a.k_major) ptx::tma_load_3d(sA, &tmA, bar, (kb_begin + kb) * BK, m0, ba);
                    else ptx::tma_load_3d(sA, &tmA, bar, m0, (kb_begin + kb) * BK, ba);
                    for (int part_b = 0; part_b <= (presplit ? 1 : 0); ++part_b) {
                        const uint32_t to = sB + part_b * B_TILE;
                        const CUtensorMap* map = part_b ? &tmBlo : &tmB;
                        if (p.b.k_major) {
                            ptx::tma_load_3d(to, map, bar, (kb_begin + kb) * BK, n0, bb);
                        } else {
#pragma unroll
                            for (int g = 0; g < BN / 32; ++g)
                                ptx::tma_load_3d(to + g * 4096, map, bar, n0 + g * 32, (kb_begin + kb) * BK, bb);
                        }
                    }
                }
                __syncwarp();
                if (++s == static_cast<uint32_t>(S)) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp == 13) {
        // ------------------------------------------------------------ UMMA issuer
        {
            const uint32_t idesc = ptx::make_idesc(2u, 0u, p.b.k_major ? 0u : 1u, kBM, BN);
            const uint32_t b_step = (p.b.k_major ? 32u : 1024u) >> 4;
            const uint64_t db0 = ptx::make_smem_desc(smem0 + A_TILE, p.b.k_major ? 16u : BK * 128u, p.b.k_major ? 1024u : 512u,
                                                     p.b.k_major ? 2u : 1u);
            const uint64_t* b_full = p.b_parts == F32_B_SPLIT ? raw_full : conv_full;
            uint32_t s = 0, ph = 0, slot = 0, sph = 0, buf = 0, tphase = 0;
            bool ok = true;
            for (int t = tile0; ok && t < p.total_tiles; t += gridDim.x) {
                for (int kb0 = 0; ok && kb0 < num_kb; kb0 += kF32ChunkBlocks) {
                    if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&tempty_bar[buf]), tphase ^ 1u, abort_p, wait_limit))) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const uint32_t d_tmem = tmem_base + buf * BN;
                    const int kb1 = min(kb0 + kF32ChunkBlocks, num_kb);
                    for (int kb = kb0; kb < kb1; ++kb) {
                        if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&b_full[s]), ph, abort_p, wait_limit) &&
                                                         ptx::mbar_wait_bounded(ptx::smem_u32(&slot_full[slot]), sph, abort_p, wait_limit))) {
                            ok = false;
                            break;
                        }
                        ptx::tc_fence_after();
                        const uint32_t a_hi0 = tmem_base + A_COL0 + slot * 64;
                        const uint64_t dbs = db0 + ((s * STAGE) >> 4);
                        if (ptx::elect_one()) {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) {
                                const uint64_t db = dbs + ks * b_step;
                                const uint32_t a_hi = a_hi0 + ks * 8;
                                const uint32_t acc = ((kb - kb0) | ks) ? 1u : 0u;
                                umma_ts_tf32(d_tmem, a_hi + 32, db, idesc, acc);
                                umma_ts_tf32(d_tmem, a_hi, db + (B_TILE >> 4), idesc, 1u);
                                umma_ts_tf32(d_tmem, a_hi, db, idesc, 1u);
                            }
                            ptx::umma_commit(ptx::smem_u32(&slot_empty[slot]));
                            ptx::umma_commit(ptx::smem_u32(&raw_empty[s]));
                        }
                        __syncwarp();
                        if (++s == static_cast<uint32_t>(S)) {
                            s = 0;
                            ph ^= 1u;
                        }
                        if (++slot == SLOTS) {
                            slot = 0;
                            sph ^= 1u;
                        }
                    }
                    if (ok && !p.skip_tile_commit && ptx::elect_one()) ptx::umma_commit(ptx::smem_u32(&tfull_bar[buf]));
                    __syncwarp();
                    buf ^= 1u;
                    if (buf == 0) tphase ^= 1u;
                }
            }
        }
    } else if (p.b_parts != F32_B_SPLIT) {
        // ------------------------------------------------------------ converters: lo image of B
        const uint32_t ct = threadIdx.x - 14 * 32;  // 0..63
        uint32_t s = 0, ph = 0;
        bool ok = true;
        for (int t = tile0; ok && t < p.total_tiles; t += gridDim.x) {
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(ptx::smem_u32(&raw_full[s]), ph, abort_p, wait_limit))) {
                    ok = false;
                    break;
                }
                const uint32_t sB = smem0 + s * STAGE + A_TILE + ct * 16u;
                if (p.b_parts == F32_B_ROUND) {
#pragma unroll 4
                    for (uint32_t o = 0; o < B_TILE; o += 64u * 16u) {
                        const uint4 v = ld_shared_v4(sB + o);
                        uint4 hi, lo;
                        split_tf32_int(v.x, hi.x, lo.x);
                        split_tf32_int(v.y, hi.y, lo.y);
                        split_tf32_int(v.z, hi.z, lo.z);
                        split_tf32_int(v.w, hi.w, lo.w);
                        st_shared_v4(sB + o, hi);
                        st_shared_v4(sB + B_TILE + o, lo);
                    }
                } else {
#pragma unroll 4
                    for (uint32_t o = 0; o < B_TILE; o += 64u * 16u) {
                        const uint4 v = ld_shared_v4(sB + o);
                        uint4 lo;
                        lo.x = __float_as_uint(__uint_as_float(v.x) - __uint_as_float(v.x & 0xffffe000u));
                        lo.y = __float_as_uint(__uint_as_float(v.y) - __uint_as_float(v.y & 0xffffe000u));
                        lo.z = __float_as_uint(__uint_as_float(v.z) - __uint_as_float(v.z & 0xffffe000u));
                        lo.w = __float_as_uint(__uint_as_float(v.w) - __uint_as_float(v.w & 0xffffe000u));
                        st_shared_v4(sB + B_TILE + o, lo);
                    }
                }
                ptx::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&conv_full[s]));
                if (++s == static_cast<uint32_t>(S)) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    }

    // ---------------------------------------------------------------- teardown
    ptx::tc_fence_before();
    __syncthreads();
    if (*abort_p) {
        // copies and UMMAs still in flight get time to land before shared and tensor memory are released
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        if (threadIdx.x == 0) atomicOr(p.status, DEV_STATUS_WAIT_TIMEOUT);
        __syncthreads();
    }
    if (split > 1) {
        ptx::cluster_sync();
        // (only the epilogue warps go on: the other roles gave their registers away)
        int aborted = 1;
        if (warp < 8) {
            const int gave_up = lane < split ? ptx::ld_cluster_s32(ptx::map_to_cta(ptx::smem_u32(&abort_flag), lane)) : 0;
            aborted = __any_sync(0xffffffffu, gave_up != 0);
        }
        int b, m0, n0;
        decode_tile(p, tile0, b, m0, n0, kBM);
        const int row = threadIdx.x % kBM, i = m0 + row;
        const long long ro = f32_row_offset(p, i);
        const int c1 = min((part + 1) * BN / split, p.N - n0);
        const float beta = p.resid ? 1.0f : p.beta;
        if (!aborted && i < p.M) {
            // four columns at a time, all copies asked for before the first is added (a load from another SM takes
            // several hundred clocks)
            for (int c0 = part * BN / split + threadIdx.x / kBM; c0 < c1; c0 += 4 * (256 / kBM)) {
                float copy[4][8], old[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int c = c0 + u * (256 / kBM);
                    if (c >= c1) continue;
                    const uint32_t at = smem0 + static_cast<uint32_t>((c * kBM + row) * 4);
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (k < split) copy[u][k] = ptx::ld_cluster_f32(ptx::map_to_cta(at, k));
                    if (beta != 0.0f) {
                        const long long o = (static_cast<long long>(b) * p.d_batch_stride + ro + static_cast<long long>(n0 + c) * p.ldd) * 4;
                        old[u] = *reinterpret_cast<const float*>((p.resid ? p.resid : p.d) + o);
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int c = c0 + u * (256 / kBM);
                    if (c >= c1) continue;
                    float v = 0.0f;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (k < split) v += copy[u][k];
                    if (p.bias != nullptr) v += reinterpret_cast<const float*>(p.bias)[n0 + c];
                    v *= p.alpha;
                    if (beta != 0.0f) v += beta * old[u];
                    if (p.relu) v = fmaxf(v, 0.0f);
                    *reinterpret_cast<float*>(p.d + (static_cast<long long>(b) * p.d_batch_stride + ro + static_cast<long long>(n0 + c) * p.ldd) * 4) = v;
                }
            }
        }
        ptx::cluster_sync();  // no CTA leaves while another still reads its partial tile
    }
    if (warp == 13) {
        __syncwarp();
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, 512u);
    }
}

}  // namespace dlfb200
