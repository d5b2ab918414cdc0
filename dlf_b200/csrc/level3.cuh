// Helper kernels of the level-3 routines that sit on the GEMM main loop (symm, syrk, trmm, trsm).
//
// The reference's GPU versions of these routines (CLBlast-derived Xsymm / Xsyrk / Xtrmm / Xtrsm
// behind gpgpu/include/gblas.h:506-586) do the same thing this file does: the triangular or
// symmetric operand is first written out as a general square matrix, the product then runs on
// the GEMM kernel, and trsm is a blocked substitution whose off-diagonal updates are GEMMs. The
// kernels here are the memory-bound pieces of that scheme; all of them take row-major operands
// (element (i, j) at i*ld + j) - a column-major call is the row-major call with the side, the
// triangle and (syrk) the transposition flipped, which the host code does.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "contraction.cuh"
#include "ptx.cuh"

namespace dlfb200 {

template <typename T> __device__ __forceinline__ float l3_load(const T* p) { return static_cast<float>(*p); }
template <> __device__ __forceinline__ float l3_load<__half>(const __half* p) { return __half2float(*p); }
template <> __device__ __forceinline__ float l3_load<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ T l3_make(float v) { return static_cast<T>(v); }
template <> __device__ __forceinline__ __half l3_make<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 l3_make<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// dst (n x n, ld = n) = the full matrix that the `upper`/lower triangle of src stands for:
// symmetric (mirror the stored triangle) or triangular (zero elsewhere; `unit`: diagonal = 1).
template <typename T>
__global__ void l3_expand_square_kernel(T* __restrict__ dst, const T* __restrict__ src, long long ld, int n,
                                        int symmetric, int upper, int unit) {
    const long long total = static_cast<long long>(n) * n;
    for (long long id = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; id < total;
         id += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int i = static_cast<int>(id / n);
        const int j = static_cast<int>(id - static_cast<long long>(i) * n);
        const bool stored = upper ? (i <= j) : (i >= j);
        T v;
        if (i == j && unit) v = l3_make<T>(1.0f);
        else if (stored) v = src[i * ld + j];
        else if (symmetric) v = src[j * ld + i];
        else v = l3_make<T>(0.0f);
        dst[id] = v;
    }
}

// syrk: the named triangle of C = S + beta * C, S (n x n, ld = n) holding alpha * op(A) op(A)^T;
// the other triangle of C is not touched. beta == 0 does not read C.
template <typename T>
__global__ void l3_triangle_merge_kernel(T* __restrict__ c, long long ldc, const T* __restrict__ s, int n, int upper,
                                         float beta) {
    const long long total = static_cast<long long>(n) * n;
    for (long long id = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; id < total;
         id += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int i = static_cast<int>(id / n);
        const int j = static_cast<int>(id - static_cast<long long>(i) * n);
        if (!(upper ? (i <= j) : (i >= j))) continue;
        float v = l3_load(s + id);
        if (beta != 0.0f) v += beta * l3_load(c + i * ldc + j);
        c[i * ldc + j] = l3_make<T>(v);
    }
}

// B (m x n) *= alpha
template <typename T>
__global__ void l3_scale_kernel(T* __restrict__ b, long long ldb, int m, int n, float alpha) {
    const long long total = static_cast<long long>(m) * n;
    for (long long id = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; id < total;
         id += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int i = static_cast<int>(id / n);
        const int j = static_cast<int>(id - static_cast<long long>(i) * n);
        b[i * ldb + j] = l3_make<T>(alpha * l3_load(b + i * ldb + j));
    }
}

// K-split GEMM: D[i + j*ldd] = alpha * sum_s part[s][i + j*M] + beta * D[i + j*ldd] over the M x N
// window (i contiguous); `part` holds `slices` fp32 products of M*N elements each.
template <typename T>
__global__ void splitk_reduce_kernel(T* __restrict__ d, long long ldd, const float* __restrict__ part, int M, int N,
                                     int slices, float alpha, float beta) {
    const long long total = static_cast<long long>(M) * N;
    for (long long id = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; id < total;
         id += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int j = static_cast<int>(id / M);
        const int i = static_cast<int>(id - static_cast<long long>(j) * M);
        float acc = 0.0f;
        for (int s = 0; s < slices; ++s) acc += part[s * total + id];
        float v = alpha * acc;
        T* o = d + j * ldd + i;
        if (beta != 0.0f) v += beta * l3_load(o);
        *o = l3_make<T>(v);
    }
}

// Copies of matrices whose lines start anywhere (an odd leading dimension or offset) with lines on 16-byte
// boundaries, the form the tensor maps take: up to two matrices per launch (blockIdx.y). A thread writes
// one 16-byte chunk; the elements past a line's end are zero. HBM-bound (each matrix read and written once).
// fp32 lines can be written as the two tf32 parts that contraction_f32_kernel reads (operand B; F32_B_SPLIT: 2001 x 2003 x
// 2005 118 us, 110 with one part that the kernel truncates, 208 by the loader warps, which round both as this does).
// 16-bit lines that start on an odd element are read as aligned 32-bit words and shifted together.
// bf16 1111 x 1537 x 777 with both operands odd: 6 us for the copies, the product 62 -> 11 us.
struct PadLines {
    const char* src[2];
    char* dst[2];
    long long src_pitch[2], dst_pitch[2];  // bytes
    long long lines[2];
    int length[2];                         // elements of a line
    long long lo[2];                       // fp32: != 0: tf32 hi goes to dst and the rest, as tf32, this many bytes behind it
    int wait;                              // the launch is a programmatic dependent: it ends after the kernel before it
};
template <int ES>
__global__ void __launch_bounds__(256) pad_lines_kernel(const PadLines p) {
    constexpr int CPE = 16 / ES;
    const int m = blockIdx.y;
    const int len = p.length[m];
    const unsigned chunks = static_cast<unsigned>(p.dst_pitch[m] / 16), total = static_cast<unsigned>(p.lines[m]) * chunks;  // (host: below 2^31)
    ptx::launch_dependents();
    for (unsigned id = blockIdx.x * blockDim.x + threadIdx.x; id < total; id += gridDim.x * blockDim.x) {
        const unsigned line = id / chunks;
        const int e0 = static_cast<int>(id - line * chunks) * CPE;
        const char* at = p.src[m] + line * p.src_pitch[m] + static_cast<long long>(e0) * ES;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (e0 + CPE <= len) {
            if constexpr (ES == 4) {
                const uint32_t* w = reinterpret_cast<const uint32_t*>(at);
                v = make_uint4(w[0], w[1], w[2], w[3]);
            } else if ((reinterpret_cast<uintptr_t>(at) & 2u) == 0) {
                const uint32_t* w = reinterpret_cast<const uint32_t*>(at);
                v = make_uint4(w[0], w[1], w[2], w[3]);
            } else {
                // elements 0 and 7 by themselves, the six between them as three words
                const uint32_t* w = reinterpret_cast<const uint32_t*>(at + 2);
                const uint32_t first = *reinterpret_cast<const unsigned short*>(at);
                const uint32_t last = *reinterpret_cast<const unsigned short*>(at + 14);
                const uint32_t a = w[0], b = w[1], c = w[2];
                v = make_uint4(first | (a << 16), __funnelshift_r(a, b, 16), __funnelshift_r(b, c, 16), (c >> 16) | (last << 16));
            }
        } else {
            uint32_t e[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int i = 0; i < CPE; ++i) {
                if (e0 + i >= len) continue;
                if constexpr (ES == 4) e[i] = reinterpret_cast<const uint32_t*>(at)[i];
                else e[i >> 1] |= static_cast<uint32_t>(reinterpret_cast<const unsigned short*>(at)[i]) << (16 * (i & 1));
            }
            v = make_uint4(e[0], e[1], e[2], e[3]);
        }
        char* dst = p.dst[m] + line * p.dst_pitch[m] + static_cast<long long>(e0) * ES;
        if (ES == 4 && p.lo[m] != 0) {
            const uint4 x = v;
            uint4 lo;
            split_tf32_int(x.x, v.x, lo.x);
            split_tf32_int(x.y, v.y, lo.y);
            split_tf32_int(x.z, v.z, lo.z);
            split_tf32_int(x.w, v.w, lo.w);
            *reinterpret_cast<uint4*>(dst + p.lo[m]) = lo;
        }
        *reinterpret_cast<uint4*>(dst) = v;
    }
    if (p.wait) ptx::wait_for_dependencies();
}

constexpr int kTrsmOrder = 1024;   // unknowns one launch solves; longer systems are cut into blocks of this order
constexpr int kTrsmThreads = 512;  // (256 and 128: see trsm_columns in api.cu)
constexpr int kTrsmTileLd = 36;  // floats between the lines of a staged 32 x 32 tile (16-byte aligned lines)
constexpr int kTrsmTurn = 64 * 20;  // floats of a row warp's transposition buffer: 64 lines of 16 + 4 or 32 of 32 + 4

// dynamic shared memory of l3_trsm_kernel: the CTA's right-hand sides, then a transposition buffer per row warp
constexpr size_t trsm_smem_bytes(int q, int columns, bool eq_contiguous, int threads) {
    return static_cast<size_t>((q + 63) / 64 * 64) * columns * 4 + (eq_contiguous ? 0 : (threads / 32 - 3) * kTrsmTurn * 4);
}

// Substitution, whole: q <= kTrsmOrder unknowns of `nsys` independent systems, C systems per CTA, which stay
// in shared memory as fp32 from the first unknown to the last. Unknowns and equations are numbered in the order
// they are solved, so that the coefficients are lower triangular: coefficient of unknown v in equation p at
// base[p*se + v*sv], unknown p of system t at b[p*b_unknown + t*b_system] (strides negative for a backward
// substitution). EQC: equations are the contiguous direction of the stored matrix (|se| == 1), else the unknowns.
// The unused triangle, and the diagonal of a unit-triangular matrix, are not read.
//
// What bounds it is the chain of unknowns, so the block of 32 unknowns at hand is all that warp 0 works on:
// lane = equation, it takes the newest 32 solved unknowns out of the next 32 equations and solves those, the systems
// side by side to cover the latency of the shuffles (with many systems lane = system), while warps
// 1 and 2 fetch the two coefficient tiles warp 0 needs two steps later and the other warps take the newest
// unknowns out of all later equations (the solved unknowns come from shared memory, 16 bytes a lane,
// which is what sets their pace), each with its next 32 coefficients already on the way. One barrier
// per 32 unknowns. A quotient is a product with the reciprocal and one correction step (12 clocks of latency
// instead of a division's); a block with a result that is not finite is solved again with divisions.
// Measured (fp32): 1024 unknowns x 512 systems 947 us in 16 launches of one thread per system and 15 products between
// them, now 93 (equations contiguous) to 119 us (unknowns); 512 x 512 37 to 45, 128 x 512 11 to 13, 48 x 48 6 us.
template <typename T, bool EQC, int C, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS)
    l3_trsm_kernel(const T* __restrict__ base, long long se, long long sv, int unit, int q, T* __restrict__ b,
                   long long b_unknown, long long b_system, int nsys, float alpha) {
    static_assert(C % 4 == 0 && C <= 32, "a lane of warp 0 solves one system; right-hand sides move as float4");
    constexpr int kTrsmRowWarps = THREADS / 32 - 3;
    extern __shared__ __align__(16) float trsm_smem[];
    __shared__ __align__(16) float dia[2][32 * kTrsmTileLd];  // [unknown][equation] of the diagonal tile
    __shared__ __align__(16) float sub[2][32 * kTrsmTileLd];  // [unknown][equation] of the tile left of it
    __shared__ float2 pivot[2][32];                           // diagonal element and its reciprocal
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int blocks = (q + 31) / 32, rows = (q + 63) / 64 * 64;
    // Up to 8 systems: warp 0 solves them by shuffles, a row lane takes two equations. With more, a lane of warp 0
    // solves one system and a row lane has one equation (2500 x 2500: 684 us by shuffles and two
    // equations a lane, 548 so).
    constexpr bool kFew = C <= 8;
    constexpr int RPL = kFew ? 2 : 1;        // equations per row lane
    constexpr int UW = 32 / RPL;             // unknowns at a time
    constexpr int kUnroll = C <= 4 ? 8 : 4;  // short loops: unrolled in full, warp 0's code is fetched again every step
    const int groups = (q + 32 * RPL - 1) / (32 * RPL);
    float* R = trsm_smem;  // [equation][C]
    const int sys0 = blockIdx.x * C;

    // coefficients of equations p0.. and unknowns v0.. (a tile below the diagonal): one line of the tile per lane
    auto load_tile = [&](float (&v)[32], int p0, int v0) {
        const T* at = base + (EQC ? (p0 + lane) * se + v0 * sv : p0 * se + (v0 + lane) * sv);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const bool inside = EQC ? p0 + lane < q : p0 + i < q;
            v[i] = inside ? l3_load(at + i * (EQC ? sv : se)) : 0.0f;
        }
    };
    auto put_tile = [&](float* tile, const float (&v)[32]) {
        if constexpr (EQC) {
#pragma unroll
            for (int i = 0; i < 32; ++i) tile[i * kTrsmTileLd + lane] = v[i];
        } else {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
                *reinterpret_cast<float4*>(tile + lane * kTrsmTileLd + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
    };
    // warp 1: the tile left of block j's diagonal
    auto load_sub = [&](float (&v)[32], int j) { load_tile(v, j * 32, j * 32 - 32); };
    // warp 2: block j's diagonal tile (below the diagonal; zero elsewhere) and the lane's diagonal element
    auto load_dia = [&](float (&v)[32], float& d, int j) {
        const int p0 = j * 32;
        const T* at = base + (EQC ? (p0 + lane) * se + p0 * sv : p0 * se + (p0 + lane) * sv);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const int eq = EQC ? lane : i, var = EQC ? i : lane;
            v[i] = var < eq && p0 + eq < q ? l3_load(at + i * (EQC ? sv : se)) : 0.0f;
        }
        d = !unit && p0 + lane < q ? l3_load(base + (p0 + lane) * (se + sv)) : 1.0f;
    };
    auto fma4 = [](float4& a, float k, const float4& x) {
        a.x = fmaf(k, x.x, a.x);
        a.y = fmaf(k, x.y, a.y);
        a.z = fmaf(k, x.z, a.z);
        a.w = fmaf(k, x.w, a.w);
    };
    // warp 0: block j, with the unknowns of block j - 1 still in its equations (j > 0)
    auto solve_block = [&](int j) {
        const float* tile = dia[j & 1];
        const float2* piv = pivot[j & 1];
        float4* row = reinterpret_cast<float4*>(R + (j * 32 + lane) * C);
        float4 acc[C / 4];
#pragma unroll
        for (int c = 0; c < C / 4; ++c) acc[c] = row[c];
        if (j > 0) {
            const float* left = sub[j & 1];
#pragma unroll kUnroll
            for (int i = 0; i < 32; ++i) {
                const float k = -left[i * kTrsmTileLd + lane];
                const float4* x = reinterpret_cast<const float4*>(R + ((j - 1) * 32 + i) * C);
#pragma unroll
                for (int c = 0; c < C / 4; ++c) fma4(acc[c], k, x[c]);
            }
        }
        bool redo;
        if constexpr (kFew) {
            const float2 d = piv[lane];
            auto over = [&](float a) {
                const float quot = a * d.y;
                return fmaf(fmaf(-quot, d.x, a), d.y, quot);
            };
            float a[C];
#pragma unroll
            for (int c = 0; c < C / 4; ++c) {
                a[4 * c] = acc[c].x;
                a[4 * c + 1] = acc[c].y;
                a[4 * c + 2] = acc[c].z;
                a[4 * c + 3] = acc[c].w;
            }
            // (a lane's coefficients of its own and of later unknowns are zero: its right-hand sides stay)
#pragma unroll kUnroll
            for (int s = 0; s < 32; ++s) {
                const float k = -tile[s * kTrsmTileLd + lane];
#pragma unroll
                for (int c = 0; c < C; ++c) a[c] = fmaf(k, __shfl_sync(0xffffffffu, over(a[c]), s), a[c]);
            }
            float check = 0.0f;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                a[c] = over(a[c]);
                check = fmaf(0.0f, a[c], check);  // NaN if a result is not finite
            }
            redo = __any_sync(0xffffffffu, check != 0.0f);
            if (!redo) {
#pragma unroll
                for (int c = 0; c < C / 4; ++c) row[c] = make_float4(a[4 * c], a[4 * c + 1], a[4 * c + 2], a[4 * c + 3]);
            }
        } else {
#pragma unroll
            for (int c = 0; c < C / 4; ++c) row[c] = acc[c];
            __syncwarp();
            float* col = R + j * 32 * C + min(lane, C - 1);
            float a[32];
            float check = 0.0f;
#pragma unroll
            for (int r = 0; r < 32; ++r) a[r] = col[r * C];
#pragma unroll
            for (int s = 0; s < 32; ++s) {
                const float2 d = piv[s];
                const float quot = a[s] * d.y;
                const float x = fmaf(fmaf(-quot, d.x, a[s]), d.y, quot);
                a[s] = x;
                check = fmaf(0.0f, x, check);
#pragma unroll
                for (int g = (s + 1) / 4; g < 8; ++g) {
                    const float4 k = *reinterpret_cast<const float4*>(tile + s * kTrsmTileLd + g * 4);
                    if (g * 4 > s) a[g * 4] = fmaf(-k.x, x, a[g * 4]);
                    if (g * 4 + 1 > s) a[g * 4 + 1] = fmaf(-k.y, x, a[g * 4 + 1]);
                    if (g * 4 + 2 > s) a[g * 4 + 2] = fmaf(-k.z, x, a[g * 4 + 2]);
                    if (g * 4 + 3 > s) a[g * 4 + 3] = fmaf(-k.w, x, a[g * 4 + 3]);
                }
            }
            redo = __any_sync(0xffffffffu, check != 0.0f);
            if (!redo && lane < C) {
#pragma unroll
                for (int r = 0; r < 32; ++r) col[r * C] = a[r];
            }
        }
        if (redo) {
            __syncwarp();
#pragma unroll
            for (int c = 0; c < C / 4; ++c) row[c] = acc[c];
            __syncwarp();
            float* col = R + j * 32 * C + min(lane, C - 1);
#pragma unroll 1
            for (int s = 0; s < 32; ++s) {
                const float x = col[s * C] / piv[s].x;
                __syncwarp();
                if (lane < C) {
                    col[s * C] = x;
                    for (int r = s + 1; r < 32; ++r) col[r * C] = fmaf(-tile[s * kTrsmTileLd + r], x, col[r * C]);
                }
                __syncwarp();
            }
        }
        __syncwarp();
    };

    // right-hand sides in and out; threads run along the direction of b that is contiguous
    const int total = rows * C;
    const bool across = b_system == 1;
#pragma unroll 4
    for (int id = threadIdx.x; id < total; id += THREADS) {
        const int p = across ? id / C : id % rows, t = across ? id % C : id / rows;
        R[p * C + t] = p < q && sys0 + t < nsys ? alpha * l3_load(b + p * b_unknown + (sys0 + t) * b_system) : 0.0f;
    }
    // The two fetching warps run two steps ahead: what is stored for block j + 2 in step j was loaded during
    // step j - 1, so that a step does not wait for memory.
    if (warp == 0) {
        __syncthreads();
        solve_block(0);
        __syncthreads();
        for (int j = 0; j + 1 < blocks; ++j) {
            solve_block(j + 1);
            __syncthreads();
        }
    } else if (warp == 1) {
        float v[32];
        if (blocks > 1) {
            load_sub(v, 1);
            put_tile(sub[1], v);
        }
        if (blocks > 2) load_sub(v, 2);
        __syncthreads();
        __syncthreads();
        for (int j = 0; j + 1 < blocks; ++j) {
            if (j + 2 < blocks) put_tile(sub[j & 1], v);
            if (j + 3 < blocks) load_sub(v, j + 3);
            __syncthreads();
        }
    } else if (warp == 2) {
        float v[32], d = 1.0f;
        auto put_dia = [&](int j) {
            put_tile(dia[j & 1], v);
            pivot[j & 1][lane] = make_float2(d, 1.0f / d);
        };
        load_dia(v, d, 0);
        put_dia(0);
        if (blocks > 1) load_dia(v, d, 1);
        __syncthreads();
        if (blocks > 1) put_dia(1);
        if (blocks > 2) load_dia(v, d, 2);
        __syncthreads();
        for (int j = 0; j + 1 < blocks; ++j) {
            if (j + 2 < blocks) put_dia(j + 2);
            if (j + 3 < blocks) load_dia(v, d, j + 3);
            __syncthreads();
        }
    } else {
        // Groups of 32 * RPL equations, RPL per lane (32 apart): this warp's are g == w modulo kTrsmRowWarps. In step j it
        // takes block j's unknowns, UW at a time, out of those of its equations that lie behind block j + 1.
        constexpr int TLD = UW + 4;
        const int w = warp - 3;
        float* turn = trsm_smem + total + w * kTrsmTurn;
        auto first = [&](int j) {
            const int g = (j + 2) / RPL;
            return g + (w + kTrsmRowWarps - g % kTrsmRowWarps) % kTrsmRowWarps;
        };
        auto load_part = [&](float (&v)[32], int g, int j, int h) {
            const int p0 = g * 32 * RPL, v0 = j * 32 + h * UW, lo = (j + 2) * 32;
            if constexpr (EQC) {
#pragma unroll
                for (int k = 0; k < RPL; ++k) {
                    const int p = p0 + 32 * k + lane;
                    const bool inside = p >= lo && p < q;
                    const T* at = base + p * se + v0 * sv;
#pragma unroll
                    for (int i = 0; i < UW; ++i) v[UW * k + i] = inside ? l3_load(at + i * sv) : 0.0f;
                }
            } else {
                const int p1 = p0 + lane / UW;
                const T* at = base + p1 * se + (v0 + lane % UW) * sv;
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const int p = p1 + RPL * i;
                    v[i] = p >= lo && p < q ? l3_load(at + RPL * i * se) : 0.0f;
                }
            }
        };
        float v[32], next[32];
        int g = first(0), h = 0;
        if (g < groups) load_part(v, g, 0, 0);
        __syncthreads();
        __syncthreads();
        for (int j = 0; j + 1 < blocks; ++j) {
            while (g < groups) {
                // what comes next: the group's next unknowns, else the first ones of the next group or of the next step
                const bool within = h + 1 < RPL;
                const bool same = within || g + kTrsmRowWarps < groups;
                const int nh = within ? h + 1 : 0;
                const int ng = within ? g : (same ? g + kTrsmRowWarps : first(j + 1));
                if (ng < groups) load_part(next, ng, same ? j : j + 1, nh);
                float4 acc[RPL][C / 4];
#pragma unroll
                for (int k = 0; k < RPL; ++k) {
                    const float4* row = reinterpret_cast<const float4*>(R + ((g * RPL + k) * 32 + lane) * C);
#pragma unroll
                    for (int c = 0; c < C / 4; ++c) acc[k][c] = row[c];
                }
                if constexpr (!EQC) {
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 32; ++i) turn[(RPL * i + lane / UW) * TLD + lane % UW] = v[i];
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < RPL; ++k) {
#pragma unroll
                        for (int i = 0; i < UW; i += 4) {
                            const float4 e = *reinterpret_cast<const float4*>(turn + (32 * k + lane) * TLD + i);
                            v[UW * k + i] = e.x;
                            v[UW * k + i + 1] = e.y;
                            v[UW * k + i + 2] = e.z;
                            v[UW * k + i + 3] = e.w;
                        }
                    }
                }
                const float4* x = reinterpret_cast<const float4*>(R + (j * 32 + h * UW) * C);
#pragma unroll
                for (int i = 0; i < UW; ++i) {
#pragma unroll
                    for (int c = 0; c < C / 4; ++c) {
                        const float4 xv = x[i * (C / 4) + c];
#pragma unroll
                        for (int k = 0; k < RPL; ++k) fma4(acc[k][c], -v[UW * k + i], xv);
                    }
                }
                // (the first equations of a group may be block j + 1, which is warp 0's)
#pragma unroll
                for (int k = 0; k < RPL; ++k) {
                    float4* row = reinterpret_cast<float4*>(R + ((g * RPL + k) * 32 + lane) * C);
                    if (g * RPL + k >= j + 2) {
#pragma unroll
                        for (int c = 0; c < C / 4; ++c) row[c] = acc[k][c];
                    }
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = next[i];
                g = ng;
                h = nh;
                if (!same) break;
            }
            __syncthreads();
        }
    }
#pragma unroll 4
    for (int id = threadIdx.x; id < total; id += THREADS) {
        const int p = across ? id / C : id % rows, t = across ? id % C : id / rows;
        if (p < q && sys0 + t < nsys) b[p * b_unknown + (sys0 + t) * b_system] = l3_make<T>(R[p * C + t]);
    }
}

// The same for few unknowns of many systems, a thread per system; arguments as above. Bound by the chain of q * q / 2
// multiply-adds with one operand from shared memory each, and from some ten thousand systems on by their traffic.
// Q: room for that many unknowns, 32 where they fit (20 KB of shared memory a CTA, 48 KB with 64).
// Measured (fp32, in place): 4 unknowns x 100000 systems 3.3 us (l3_trsm_kernel 80), 32 x 100000 20 (90).
constexpr int kTrsmSmall = 64;
constexpr int kTrsmSmallThreads = 128;
template <typename T, int Q>
__global__ void __launch_bounds__(kTrsmSmallThreads)
    l3_trsm_small_kernel(const T* __restrict__ base, long long se, long long sv, int unit, int q, T* __restrict__ b,
                         long long b_unknown, long long b_system, int nsys, float alpha) {
    __shared__ float coef[Q][Q];  // [equation][unknown], read as a broadcast
    __shared__ float xs[Q][kTrsmSmallThreads];
    for (int id = threadIdx.x; id < q * q; id += kTrsmSmallThreads) {
        const int eq = id / q, var = id - eq * q;
        if (var <= eq) coef[eq][var] = var == eq && unit ? 1.0f : l3_load(base + eq * se + var * sv);
    }
    __syncthreads();
    const int t = blockIdx.x * kTrsmSmallThreads + threadIdx.x;
    if (t >= nsys) return;
    T* at = b + t * b_system;
    for (int p = 0; p < q; ++p) xs[p][threadIdx.x] = alpha * l3_load(at + p * b_unknown);
    for (int p = 0; p < q; ++p) {
        float acc = xs[p][threadIdx.x];
        for (int v = 0; v < p; ++v) acc = fmaf(-coef[p][v], xs[v][threadIdx.x], acc);
        acc /= coef[p][p];
        xs[p][threadIdx.x] = acc;
        at[p * b_unknown] = l3_make<T>(acc);
    }
}

}  // namespace dlfb200
