// park.cu -- Park et al. modular plaintext matrix product (Mod-PP-MM) on the GPU.
//
// park_mod_pp_mm (ccmm/park.rs:1634-1647) multiplies two u64 matrices modulo an
// arbitrary modulus q > 1: out = (lhs x rhs) mod q, lhs rows x inner, rhs
// inner x cols, row-major. Every backend of the reference
// (park_matrix_mul_{reference,transposed_rhs,wide_accumulator,parallel_wide},
// :1405-1620) returns the canonical residue of the exact integer dot product,
// and so do both device backends here.
//
// Tensor cores (default). With nb = bytes of q - 1, a = sum_i 2^(8i) a_i
// (bytes of lhs mod q) and the weights W_i = 2^(8i) (rhs mod q) mod q split into
// bytes w_ij,
//   sum_k lhs[r][k] rhs[k][c] == sum_j 2^(8j) P_j[r][c]              (mod q),
//   P_j[r][c] = sum_(k,i) a_i[r][k] w_ij[k][c],
// exact unsigned 8-bit products summed in 32 bits on tcgen05.mma.kind::i8 (an
// inner chunk keeps nb * 32 * blocks * 255^2 below 2^31; longer inner sums take
// several launches that add their residues). Two packing kernels write both
// operands as 32-byte inner steps in the canonical K-major core-matrix order
// (A: 128 rows x 32 bytes; B: nb x ct rows (j, column) x 32 bytes, ct output
// columns per tile with nb ct <= 256), so each pipeline stage is two bulk
// copies. The GEMM is a persistent kernel: one producer thread (bulk copies
// into 4 stages of 4 inner steps), one MMA thread (M = 128, N = nb ct, K = 32 per step),
// four epilogue warps (plane combine, one reduction per output); the two TMEM
// accumulator sets let a tile's epilogue overlap the next tile's MMAs.
//
// Residue system (tensor cores, moduli of 4 bytes or more below 2^62). The byte planes
// cost nb^2 products; a product modulo small coprime m_i <= 256 costs one, and the exact
// integer sum X < inner (q - 1)^2 is determined by its residues once prod m_i = M > 2 X:
// 11 products instead of 25 for a 35-bit q at inner = 4096, 17 instead of 64 for 60 bits.
// With A_i = lhs mod m_i, B_i = rhs (M / m_i)^-1 mod m_i (bytes), w_i = A_i B_i mod m_i:
//   X = sum_i w_i (M / m_i) - k M,   k = floor(sum_i w_i / m_i)  (X / M < 1/2),
// so out = sum_i w_i (M / m_i mod q) - k (M mod q) mod q, with k from 2^27-scaled integer
// reciprocals (each below the true one by under 2^-27: the sum is off by under 2^-14).
// Packing takes two byte dot products an element and modulus; the GEMM is the persistent
// kernel below with N = 256 and one accumulator, storing w_i as bytes; one kernel combines
// the n_mod bytes of an output, in slabs of the product whose workspace is bounded. Chosen by
// estimated times (worthwhile). n = 4096, 35-bit q: packing 0.17 ms, GEMM 0.54 ms (2.80 POP/s,
// 88 % of twice the bf16 rate: the tensor pipe bounds it), combining 0.12 ms; the byte planes
// took 0.26 and 1.24 ms.
//
// CUDA cores. A CTA computes a 64 x 64 block of outputs with 256 threads (4 x 4
// outputs each, strided by 16 so a warp's loads of a staged tile row are
// consecutive), staging 16-deep slices of both operands in shared memory; each
// dot product is summed exactly in 192 bits (any u64 inputs, up to 2^64 terms)
// and reduced once.
#include <algorithm>
#include <cmath>

#include "context.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int kTile = 64, kDepth = 16, kThreads = 256;

typedef unsigned __int128 u128;

struct Acc192 {
    u64 lo, mid, hi;
    __device__ __forceinline__ void add(u64 a, u64 b) {
        const u64 pl = a * b, ph = __umul64hi(a, b);
        asm("add.cc.u64 %0, %0, %3;\n\taddc.cc.u64 %1, %1, %4;\n\taddc.u64 %2, %2, 0;"
            : "+l"(lo), "+l"(mid), "+l"(hi)
            : "l"(pl), "l"(ph));
    }
};

// (hi 2^128 + mid 2^64 + lo) mod q with r64 = 2^64 mod q, r128 = 2^128 mod q
__device__ __forceinline__ u64 reduce192(const Acc192& a, u64 q, u64 r64, u64 r128) {
    const u128 Q = q;
    u128 t = (u128)(a.hi % q) * r128 % Q;
    t = (t + (u128)(a.mid % q) * r64 % Q) % Q;
    t = (t + a.lo % q) % Q;
    return (u64)t;
}

__global__ void __launch_bounds__(kThreads) k_park_mm(const u64* __restrict__ A, const u64* __restrict__ B,
                                                      u64* __restrict__ C, int rows, int inner, int cols, u64 q,
                                                      u64 r64, u64 r128) {
    __shared__ u64 sa[kDepth][kTile + 1];  // sa[k][r]: lhs[row0 + r][k0 + k]
    __shared__ u64 sb[kDepth][kTile];      // sb[k][c]: rhs[k0 + k][col0 + c]
    const int tid = threadIdx.x;
    const int tr = tid >> 4, tc = tid & 15;  // outputs (tr + 16 i, tc + 16 j)
    const int row0 = blockIdx.y * kTile, col0 = blockIdx.x * kTile;
    Acc192 acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = Acc192{0, 0, 0};
    for (int k0 = 0; k0 < inner; k0 += kDepth) {
        // stage lhs [64 x 16] (transposed) and rhs [16 x 64]; zeros outside the matrices
        for (int w = tid; w < kTile * kDepth; w += kThreads) {
            const int r = w / kDepth, k = w % kDepth;
            const int gr = row0 + r, gk = k0 + k;
            sa[k][r] = (gr < rows && gk < inner) ? A[(size_t)gr * inner + gk] : 0;
            const int kk = w / kTile, c = w % kTile;
            const int gk2 = k0 + kk, gc = col0 + c;
            sb[kk][c] = (gk2 < inner && gc < cols) ? B[(size_t)gk2 * cols + gc] : 0;
        }
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < kDepth; ++k) {
            u64 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = sa[k][tr + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = sb[k][tc + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j].add(a[i], b[j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gr = row0 + tr + 16 * i;
        if (gr >= rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gc = col0 + tc + 16 * j;
            if (gc < cols) C[(size_t)gr * cols + gc] = reduce192(acc[i][j], q, r64, r128);
        }
    }
}

// ----------------------------------------------------------------- tensor cores
namespace ptc {

using namespace tcg;

constexpr int kEpiWarps = 4, kProdWarp = 4, kMmaWarp = 5, kThreads = 32 * 6;
constexpr int kEpi = 32 * kEpiWarps, kBarEpi = 1;
#ifndef CKKS_PARK_STEPS
#define CKKS_PARK_STEPS 4
#endif
// inner steps of 32 bytes per stage (one barrier wait per kSteps MMAs), stages in 192 KB
constexpr int kSteps = CKKS_PARK_STEPS, kStages = 16 / kSteps;
static_assert(kSteps == 1 || kSteps == 2 || kSteps == 4 || kSteps == 8, "inner steps per stage");
constexpr u32 kATile = 128 * 32;        // A step: 128 rows x 32 bytes
constexpr u32 kOffB = kSteps * kATile;  // B steps after the stage's A steps (up to 256 rows x 32 bytes each)
constexpr u32 kStageBytes = kOffB + kSteps * 256 * 32;
constexpr u32 kSmemBytes = kStages * kStageBytes;  // 192 KB: one CTA per SM
constexpr u32 kTmemCols = 512;                                     // two accumulator sets of <= 256 columns
constexpr u32 kLbo = 128, kSbo = 256;  // K-major, no swizzle: K halves 128 B apart, 8-row groups 256 B

// output columns per tile for nb bytes per residue: nb * ct <= 256, a multiple of 16
constexpr int cols_per_tile(int nb) {
    return ((256 / nb) / 8 * 8 * nb) % 16 ? (256 / nb) / 8 * 8 - 8 : (256 / nb) / 8 * 8;
}
// inner 32-blocks per launch: every P_j stays below 2^31
constexpr int blocks_per_launch(int nb) { return (int)(0x7FFFFFFFull / (65025ull * (u64)nb) / 32); }

// tile order: row tiles vary fastest (CTAs that run together share column tiles of B'')
#ifndef CKKS_PARK_COLS_FIRST
#define CKKS_PARK_COLS_FIRST 0
#endif
__device__ __forceinline__ int tile_row(int t, int n_mt, int n_nt) { return CKKS_PARK_COLS_FIRST ? t / n_nt : t % n_mt; }
__device__ __forceinline__ int tile_col(int t, int n_mt, int n_nt) { return CKKS_PARK_COLS_FIRST ? t % n_nt : t / n_mt; }

__device__ __forceinline__ u32 core_off(int row, int half) { return (u32)((row >> 3) * 256 + half * 128 + (row & 7) * 16); }

// bytes `shift` .. of 16 values as one 16-byte core-matrix row
__device__ __forceinline__ uint4 pack16(const u64 (&v)[16], int shift) {
    u32 w[4];
#pragma unroll
    for (int g = 0; g < 4; ++g)
        w[g] = (u32)((v[4 * g] >> shift) & 255) | (u32)((v[4 * g + 1] >> shift) & 255) << 8 |
               (u32)((v[4 * g + 2] >> shift) & 255) << 16 | (u32)((v[4 * g + 3] >> shift) & 255) << 24;
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// A' [n_mt][n_kb][nb][128 x 32 bytes]: step (kb, i) of row tile mt holds byte i of
// lhs[128 mt + row][32 kb + k] mod q. One thread per (row, 16-deep run).
__global__ void k_pack_a(const u64* __restrict__ A, uint8_t* __restrict__ Ap, int rows, int inner, u64 q, int nb,
                         int n_mt, int n_kb) {
    const size_t runs = (size_t)2 * n_kb, total = (size_t)n_mt * 128 * runs;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int row = (int)(t / runs), h = (int)(t % runs);
        u64 v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int k = 16 * h + e;
            const u64 x = (row < rows && k < inner) ? A[(size_t)row * inner + k] : 0;
            v[e] = x < q ? x : x % q;
        }
        uint8_t* dst = Ap + ((size_t)(row >> 7) * n_kb + (h >> 1)) * nb * kATile + core_off(row & 127, h & 1);
        for (int i = 0; i < nb; ++i) *(uint4*)(dst + (size_t)i * kATile) = pack16(v, 8 * i);
    }
}

// B'' [n_nt][n_kb][nb][nb ct x 32 bytes]: step (kb, i), row j ct + c holds byte j of
// 2^(8i) (rhs[32 kb + k][ct nt + c] mod q) mod q. One thread per (column, 16-deep run).
// f256q = floor(2^72 / q): the weights step by a Shoup product with 256 when
// 256 < q <= 2^63 (f256q != 0), else by a 128-bit remainder.
__global__ void k_pack_b(const u64* __restrict__ B, uint8_t* __restrict__ Bp, int inner, int cols, u64 q, int nb,
                         int ct, int n_nt, int n_kb, u64 f256q) {
    const int cpad = n_nt * ct;
    const size_t total = (size_t)cpad * 2 * n_kb;
    const u32 b_step = (u32)(nb * ct) * 32;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t % cpad), h = (int)(t / cpad);
        const int nt = c / ct, cl = c - nt * ct;
        u64 w[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int k = 16 * h + e;
            const u64 x = (c < cols && k < inner) ? B[(size_t)k * cols + c] : 0;
            w[e] = x < q ? x : x % q;
        }
        uint8_t* base = Bp + ((size_t)nt * n_kb + (h >> 1)) * nb * b_step;
        for (int i = 0; i < nb; ++i) {
            if (i > 0 && f256q) {
#pragma unroll
                for (int e = 0; e < 16; ++e) w[e] = mul_shoup(w[e], 256, f256q, q);
            } else if (i > 0) {
#pragma unroll
                for (int e = 0; e < 16; ++e) w[e] = (u64)(((u128)w[e] << 8) % q);
            }
            for (int j = 0; j < nb; ++j)
                *(uint4*)(base + (size_t)i * b_step + core_off(j * ct + cl, h & 1)) = pack16(w, 8 * j);
        }
    }
}

// Inner blocks kb0 .. kb1 - 1 of every (row tile, column tile); accumulate: add
// the residues already in C. `err` receives the role of a timed-out wait.
template <int NB>
__global__ void __launch_bounds__(kThreads, 1)
    k_park_tc(const uint8_t* __restrict__ Ap, const uint8_t* __restrict__ Bp, u64* __restrict__ C, int rows,
              int cols, u64 q, int n_mt, int n_nt, int n_kb, int kb0, int kb1, int accumulate, int* __restrict__ err) {
    constexpr int kCt = cols_per_tile(NB), kRows = NB * kCt;
    constexpr u32 kBStep = (u32)kRows * 32;
    constexpr u32 kIdesc = idesc_i8(128, kRows, false);
    static_assert(kRows <= 256 && kRows % 16 == 0 && kCt % 8 == 0, "tile shape");
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ u32 s_tmem;
    __shared__ int s_abort;
    __shared__ __align__(8) uint64_t s_full[kStages], s_empty[kStages], s_tfull[2], s_tfree[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_tiles = n_mt * n_nt;
    const int my_tiles = (int)blockIdx.x < n_tiles ? (n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int steps = (kb1 - kb0) * NB;
    const u64 mu = ~0ull / q;
    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < kStages; ++i) {
            mbar_init(smem_u32(&s_full[i]), 1);
            mbar_init(smem_u32(&s_empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&s_tfull[i]), 1);
            mbar_init(smem_u32(&s_tfree[i]), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const u32 tmem = s_tmem, sbase = smem_u32(smem);

    if (warp == kProdWarp) {
        // ------------------------------------------------------------ producer
        if (lane == 0) {
            int g = 0;
            bool bad = false;
            for (int lt = 0; lt < my_tiles && !bad; ++lt) {
                const int t = (int)blockIdx.x + lt * (int)gridDim.x;
                const int mt = tile_row(t, n_mt, n_nt), nt = tile_col(t, n_mt, n_nt);
                const uint8_t* a = Ap + ((size_t)mt * n_kb + kb0) * NB * kATile;
                const uint8_t* b = Bp + ((size_t)nt * n_kb + kb0) * NB * kBStep;
                for (int s = 0; s < steps; s += kSteps, ++g) {
                    const int st = g % kStages;
                    const u32 n = (u32)(steps - s < kSteps ? steps - s : kSteps);
                    if ((g >= kStages && !wait_parity(smem_u32(&s_empty[st]), (u32)(((g / kStages) - 1) & 1))) ||
                        s_abort) {
                        atomicExch(err, 1);
                        s_abort = 1;
                        bad = true;
                        break;
                    }
                    const u32 bar = smem_u32(&s_full[st]), dst = sbase + (u32)st * kStageBytes;
                    expect_tx(bar, n * (kATile + kBStep));
                    bulk_g2s(dst, a + (size_t)s * kATile, n * kATile, bar);
                    bulk_g2s(dst + kOffB, b + (size_t)s * kBStep, n * kBStep, bar);
                }
            }
            // every copy issued has landed before the CTA can leave (bounded)
            for (int x = g - kStages < 0 ? 0 : g - kStages; x < g; ++x)
                wait_parity(smem_u32(&s_full[x % kStages]), (u32)((x / kStages) & 1));
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------ MMA issue
        if (lane == 0) {
            int g = 0, last = -1;
            bool bad = false;
            for (int lt = 0; lt < my_tiles && !bad; ++lt) {
                const int buf = lt & 1;
                if (lt >= 2 && !wait_parity(smem_u32(&s_tfree[buf]), (u32)(((lt >> 1) - 1) & 1))) {
                    atomicExch(err, 3);
                    s_abort = 1;
                    break;
                }
                fence_after();
                for (int s = 0; s < steps; s += kSteps, ++g) {
                    const int st = g % kStages;
                    const int n = steps - s < kSteps ? steps - s : kSteps;
                    if (!wait_parity(smem_u32(&s_full[st]), (u32)((g / kStages) & 1)) || s_abort) {
                        atomicExch(err, 2);
                        s_abort = 1;
                        bad = true;
                        break;
                    }
                    fence_after();
                    const u32 a_addr = sbase + (u32)st * kStageBytes, b_addr = a_addr + kOffB;
#pragma unroll
                    for (int u = 0; u < kSteps; ++u)
                        if (u < n)
                            mma_i8(tmem + (u32)buf * 256u, sdesc(a_addr + (u32)u * kATile, kLbo, kSbo),
                                   sdesc(b_addr + (u32)u * kBStep, kLbo, kSbo), kIdesc, (s + u) > 0 ? 1u : 0u);
                    commit(smem_u32(&s_empty[st]));
                    last = g;
                }
                if (!bad) commit(smem_u32(&s_tfull[buf]));
            }
            // the last commit covers every MMA issued
            if (last >= 0) wait_parity(smem_u32(&s_empty[last % kStages]), (u32)((last / kStages) & 1));
        }
        __syncwarp();
    } else if (warp < kEpiWarps) {
        // ------------------------------------------------------------- epilogue
        for (int lt = 0; lt < my_tiles; ++lt) {
            const int buf = lt & 1;
            const int t = (int)blockIdx.x + lt * (int)gridDim.x;
            const int mt = tile_row(t, n_mt, n_nt), nt = tile_col(t, n_mt, n_nt);
            const bool bad = !wait_parity(smem_u32(&s_tfull[buf]), (u32)((lt >> 1) & 1));
            if (group_any(kBarEpi, kEpi, bad || s_abort)) {
                if (tid == 0) {
                    atomicExch(err, 4);
                    s_abort = 1;
                }
                break;
            }
            fence_after();
            const int row = 128 * mt + 32 * warp + lane, cmax = cols - nt * kCt;
            const u32 taddr = tmem + ((u32)(32 * warp) << 16) + (u32)buf * 256u;
            u64* out = C + (size_t)row * cols + (size_t)nt * kCt;
#pragma unroll 1
            for (int c0 = 0; c0 < kCt; c0 += 8) {
                u64 r[8];
                if constexpr (NB <= 5) {  // sum_j 2^(8j) P_j < 2^63.01
                    u64 v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
                    for (int j = 0; j < NB; ++j) {
                        u32 P[8];
                        tmem_ld8(taddr + (u32)(j * kCt + c0), P);
#pragma unroll
                        for (int cc = 0; cc < 8; ++cc) v[cc] += (u64)P[cc] << (8 * j);
                    }
#pragma unroll
                    for (int cc = 0; cc < 8; ++cc) {  // v - floor(v mu / 2^64) q < 3q
                        u64 x = v[cc] - __umul64hi(v[cc], mu) * q;
                        x = x >= q ? x - q : x;
                        r[cc] = x >= q ? x - q : x;
                    }
                } else {
                    u128 v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
                    for (int j = 0; j < NB; ++j) {
                        u32 P[8];
                        tmem_ld8(taddr + (u32)(j * kCt + c0), P);
#pragma unroll
                        for (int cc = 0; cc < 8; ++cc) v[cc] += (u128)P[cc] << (8 * j);
                    }
#pragma unroll
                    for (int cc = 0; cc < 8; ++cc) r[cc] = (u64)(v[cc] % q);
                }
                if (row < rows) {
#pragma unroll
                    for (int cc = 0; cc < 8; ++cc) {
                        if (c0 + cc >= cmax) break;
                        u64 x = r[cc];
                        if (accumulate) {
                            const u64 y = x + out[c0 + cc];
                            x = (y < x || y >= q) ? y - q : y;
                        }
                        out[c0 + cc] = x;
                    }
                }
            }
            fence_before();
            named_sync(kBarEpi, kEpi);  // every lane of the set read
            if (tid == 0) arrive(smem_u32(&s_tfree[buf]));
        }
    }
    // teardown: every role has left its loop (on abort, after a bounded wait)
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == kMmaWarp) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// CUDA events around the packing and the GEMM launches of this thread's last
// tensor-core call (created per thread and device on first use)
struct Timing {
    int dev = -1;
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
    float pack_ms = -1.f, gemm_ms = -1.f;
};
thread_local Timing t_timing;

int32_t timing_events(int dev) {
    Timing& t = t_timing;
    if (t.dev == dev) return CKKS_OK;
    for (auto& e : t.ev)
        if (e) cudaEventDestroy(e), e = nullptr;
    t.dev = -1;
    for (auto& e : t.ev) CKKS_CUDA_TRY(cudaEventCreate(&e));
    t.dev = dev;
    return CKKS_OK;
}

// Runs body(err, packed): `err` a zeroed device word for the role of a timed-out wait,
// packed() called between the packing and the product; then waits and reports.
template <typename F>
int32_t timed(int dev, cudaStream_t st, F&& body) {
    {  // keep the freed packed operands cached in the device pool between calls
        cudaMemPool_t pool;
        if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
            uint64_t thr = ~0ull;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
        }
    }
    Workspace<int> err;
    int32_t rc;
    if ((rc = err.alloc(1, st))) return rc;
    CKKS_CUDA_TRY(cudaMemsetAsync(err.p, 0, sizeof(int), st));
    if ((rc = timing_events(dev))) return rc;
    t_timing.pack_ms = t_timing.gemm_ms = -1.f;
    CKKS_CUDA_TRY(cudaEventRecord(t_timing.ev[0], st));
    auto packed = [&]() -> int32_t {
        CKKS_CUDA_TRY(cudaEventRecord(t_timing.ev[1], st));
        return CKKS_OK;
    };
    if ((rc = body(err.p, packed))) return rc;
    CKKS_CUDA_TRY(cudaEventRecord(t_timing.ev[2], st));
    int h_err = 0;
    CKKS_CUDA_TRY(cudaMemcpyAsync(&h_err, err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    CKKS_CUDA_TRY(cudaStreamSynchronize(st));
    CKKS_CUDA_TRY(cudaEventElapsedTime(&t_timing.pack_ms, t_timing.ev[0], t_timing.ev[1]));
    CKKS_CUDA_TRY(cudaEventElapsedTime(&t_timing.gemm_ms, t_timing.ev[1], t_timing.ev[2]));
    if (h_err) {
        ckks_set_error("ckks_park_mod_pp_mm: a tensor-core pipeline wait timed out (role " + std::to_string(h_err) +
                       ")");
        return CKKS_ERR_TIMEOUT;
    }
    return CKKS_OK;
}

template <int NB>
int32_t launch(const u64* lhs, const u64* rhs, u64* out, u32 rows, u32 inner, u32 cols, u64 q, cudaStream_t st) {
    constexpr int kCt = cols_per_tile(NB), kRows = NB * kCt, kChunk = blocks_per_launch(NB);
    const int n_mt = (int)((rows + 127) / 128), n_nt = (int)((cols + kCt - 1) / kCt), n_kb = (int)((inner + 31) / 32);
    int dev = 0, n_sm = 0;
    CKKS_CUDA_TRY(cudaGetDevice(&dev));
    CKKS_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    return timed(dev, st, [&](int* err, auto packed) -> int32_t {
        Workspace<uint8_t> ap, bp;
        int32_t rc;
        if ((rc = ap.alloc((size_t)n_mt * n_kb * NB * kATile, st)) ||
            (rc = bp.alloc((size_t)n_nt * n_kb * NB * kRows * 32, st)))
            return rc;
        auto grid_of = [&](size_t threads) {
            const size_t g = (threads + 255) / 256, cap = (size_t)n_sm * 16;
            return (int)(g < cap ? g : cap);
        };
        k_pack_a<<<grid_of((size_t)n_mt * 128 * 2 * n_kb), 256, 0, st>>>(lhs, ap.p, (int)rows, (int)inner, q, NB, n_mt,
                                                                           n_kb);
        CKKS_CUDA_TRY(cudaGetLastError());
        const u64 f256q = (q > 256 && q <= (1ull << 63)) ? (u64)(((u128)256 << 64) / q) : 0;
        k_pack_b<<<grid_of((size_t)n_nt * kCt * 2 * n_kb), 256, 0, st>>>(rhs, bp.p, (int)inner, (int)cols, q, NB, kCt,
                                                                          n_nt, n_kb, f256q);
        CKKS_CUDA_TRY(cudaGetLastError());
        CKKS_CUDA_TRY(cudaFuncSetAttribute(k_park_tc<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
        const int n_tiles = n_mt * n_nt, grid = n_tiles < n_sm ? n_tiles : n_sm;
        if ((rc = packed())) return rc;
        for (int kb0 = 0; kb0 < n_kb; kb0 += kChunk) {
            const int kb1 = kb0 + kChunk < n_kb ? kb0 + kChunk : n_kb;
            k_park_tc<NB><<<grid, kThreads, kSmemBytes, st>>>(ap.p, bp.p, out, (int)rows, (int)cols, q, n_mt, n_nt,
                                                              n_kb, kb0, kb1, kb0 > 0 ? 1 : 0, err);
            CKKS_CUDA_TRY(cudaGetLastError());
        }
        return CKKS_OK;
    });
}

// bytes of the packed operands (the planes' workspace)
size_t packed_bytes(u32 rows, u32 inner, u32 cols, u64 q) {
    const int nb = (64 - __builtin_clzll(q - 1) + 7) / 8, ct = cols_per_tile(nb);
    return (size_t)((inner + 31) / 32) * nb * 32 *
           ((size_t)((rows + 127) / 128) * 128 + (size_t)((cols + ct - 1) / ct) * nb * ct);
}

// the tensor-core form covers every modulus; tile counts stay within int
bool supported(u32 rows, u32 cols, u64 q) {
    const int nb = (64 - __builtin_clzll(q - 1) + 7) / 8;
    const u64 n_mt = (rows + 127) / 128, n_nt = (cols + (u64)cols_per_tile(nb) - 1) / (u64)cols_per_tile(nb);
    return n_mt * n_nt < (1ull << 31);
}

int32_t run(const u64* lhs, const u64* rhs, u64* out, u32 rows, u32 inner, u32 cols, u64 q, cudaStream_t st) {
    switch ((64 - __builtin_clzll(q - 1) + 7) / 8) {
        case 1: return launch<1>(lhs, rhs, out, rows, inner, cols, q, st);
        case 2: return launch<2>(lhs, rhs, out, rows, inner, cols, q, st);
        case 3: return launch<3>(lhs, rhs, out, rows, inner, cols, q, st);
        case 4: return launch<4>(lhs, rhs, out, rows, inner, cols, q, st);
        case 5: return launch<5>(lhs, rhs, out, rows, inner, cols, q, st);
        case 6: return launch<6>(lhs, rhs, out, rows, inner, cols, q, st);
        case 7: return launch<7>(lhs, rhs, out, rows, inner, cols, q, st);
        default: return launch<8>(lhs, rhs, out, rows, inner, cols, q, st);
    }
}

}  // namespace ptc

// ------------------------------------------------------- residue number system
namespace rns {

using namespace tcg;

constexpr int kMaxMod = 20;
// pairwise coprime, descending: 256 = 2^8, 255 = 3 5 17, 253 = 11 23, 247 = 13 19, 217 = 7 31, primes
constexpr int kModuli[kMaxMod] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227,
                                  223, 217, 211, 199, 197, 193, 191, 181, 179, 173};
constexpr int kMaxInner = 33024;  // 33024 * 255^2 < 2^31
constexpr int kN = 256;           // output columns per tile
constexpr u32 kATile = 128 * 32, kBTile = kN * 32;
constexpr int kSteps = 4, kStages = 4;  // 32-byte inner steps per stage, stages
constexpr u32 kOffB = kSteps * kATile, kStageBytes = kOffB + kSteps * kBTile;
constexpr u32 kSmemBytes = kStages * kStageBytes;  // 192 KB
constexpr u32 kIdesc = idesc_i8(128, kN, false);
constexpr int kEpiWarps = 4, kProdWarp = 4, kMmaWarp = 5, kThreads = 32 * 6, kEpi = 128, kBarEpi = 1;

struct Mod {
    u32 m, mu_small, mu;      // modulus; ceil(2^32 / m) (exact quotients below 2^24), floor(2^32 / m)
    u32 a_lo, a_hi;           // bytes 2^(8j) mod m, j = 0..3, 4..7
    u32 b_lo, b_hi;           // bytes 2^(8j) (M / m)^-1 mod m
    u32 recip;                // floor(2^27 / m)
    u32 mq_lo, mq_hi;         // M / m mod q
};
struct Params {
    int n;
    Mod m[kMaxMod];
    u64 q, mu, r32, r32q;     // floor((2^64 - 1) / q), 2^32 mod q and its Shoup companion
    u32 nm_lo, nm_hi;         // q - (M mod q)
};

// x mod m from the byte dot product with 2^(8j) mod m: below 2^19 + 2^19, exact quotient
__device__ __forceinline__ u32 residue(u32 lo, u32 hi, u32 r_lo, u32 r_hi, const Mod& md) {
    const u32 s = __dp4a(lo, r_lo, __dp4a(hi, r_hi, 0u));
    return s - __umulhi(s, md.mu_small) * md.m;
}

// Both operands: per modulus 32-byte inner steps in the K-major core-matrix order.
// A' [n][n_mt][n_kb][128 x 32]: one thread per (row, 16-deep run); B' [n][n_nt][n_kb][256 x 32]:
// one thread per (column, 16-deep run). Threads [0, a_total) take A; n_mt or n_nt = 0 leaves an
// operand out. Rows of B lie ldb words apart. Neighbouring threads take neighbouring rows
// (columns), so a warp stores whole 128-byte core matrices.
__global__ void __launch_bounds__(256) k_rns_pack(const u64* __restrict__ A, const u64* __restrict__ B,
                                                  uint8_t* __restrict__ Ap, uint8_t* __restrict__ Bp, int rows,
                                                  int inner, int cols, size_t ldb, int n_mt, int n_nt, int n_kb,
                                                  bool vec_a, const __grid_constant__ Params P) {
    const size_t runs = (size_t)2 * n_kb, a_total = (size_t)n_mt * 128 * runs, b_total = (size_t)n_nt * kN * runs;
    const size_t a_plane = (size_t)n_mt * n_kb * kATile, b_plane = (size_t)n_nt * n_kb * kBTile;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < a_total + b_total;
         t += (size_t)gridDim.x * blockDim.x) {
        const bool is_a = t < a_total;
        u64 v[16];
        uint8_t* dst;
        if (is_a) {
            const int rpad = n_mt * 128, row = (int)(t % rpad), h = (int)(t / rpad);
            const u64* src = A + (size_t)row * inner + 16 * h;
            if (vec_a && row < rows && 16 * h + 16 <= inner) {
#pragma unroll
                for (int e = 0; e < 16; e += 2) {
                    const ulonglong2 x = __ldg((const ulonglong2*)(src + e));
                    v[e] = x.x, v[e + 1] = x.y;
                }
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = (row < rows && 16 * h + e < inner) ? src[e] : 0;
            }
            dst = Ap + ((size_t)(row >> 7) * n_kb + (h >> 1)) * kATile + ptc::core_off(row & 127, h & 1);
        } else {
            const size_t u = t - a_total;
            const int cpad = n_nt * kN, c = (int)(u % cpad), h = (int)(u / cpad);
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const int k = 16 * h + e;
                v[e] = (c < cols && k < inner) ? B[(size_t)k * ldb + c] : 0;
            }
            dst = Bp + ((size_t)(c / kN) * n_kb + (h >> 1)) * kBTile + ptc::core_off(c % kN, h & 1);
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = v[e] < P.q ? v[e] : v[e] % P.q;
        const size_t plane = is_a ? a_plane : b_plane;
        for (int i = 0; i < P.n; ++i, dst += plane) {
            const Mod& md = P.m[i];
            const u32 r_lo = is_a ? md.a_lo : md.b_lo, r_hi = is_a ? md.a_hi : md.b_hi;
            u32 w[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                w[g] = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    w[g] |= residue((u32)v[4 * g + e], (u32)(v[4 * g + e] >> 32), r_lo, r_hi, md) << (8 * e);
            }
            *(uint4*)dst = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// Every (modulus, row tile, column tile): w_i = A_i B_i mod m_i as bytes W [n][128 n_mt][256 n_nt].
// Roles and waits as k_park_tc; row tiles vary fastest, then column tiles, then moduli.
__global__ void __launch_bounds__(kThreads, 1)
    k_rns_gemm(const uint8_t* __restrict__ Ap, const uint8_t* __restrict__ Bp, uint8_t* __restrict__ W, int n_mt,
               int n_nt, int n_kb, const __grid_constant__ Params P, int* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ u32 s_tmem;
    __shared__ int s_abort;
    __shared__ __align__(8) uint64_t s_full[kStages], s_empty[kStages], s_tfull[2], s_tfree[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int per_mod = n_mt * n_nt, n_tiles = per_mod * P.n;
    const int my_tiles = (int)blockIdx.x < n_tiles ? (n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < kStages; ++i) {
            mbar_init(smem_u32(&s_full[i]), 1);
            mbar_init(smem_u32(&s_empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&s_tfull[i]), 1);
            mbar_init(smem_u32(&s_tfree[i]), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const u32 tmem = s_tmem, sbase = smem_u32(smem);

    if (warp == kProdWarp) {
        // ------------------------------------------------------------ producer
        if (lane == 0) {
            int g = 0;
            bool bad = false;
            for (int lt = 0; lt < my_tiles && !bad; ++lt) {
                const int t = (int)blockIdx.x + lt * (int)gridDim.x, i = t / per_mod, x = t - i * per_mod;
                const int nt = x / n_mt, mt = x - nt * n_mt;
                const uint8_t* a = Ap + ((size_t)i * n_mt + mt) * n_kb * kATile;
                const uint8_t* b = Bp + ((size_t)i * n_nt + nt) * n_kb * kBTile;
                for (int s = 0; s < n_kb; s += kSteps, ++g) {
                    const int st = g % kStages;
                    const u32 n = (u32)(n_kb - s < kSteps ? n_kb - s : kSteps);
                    if ((g >= kStages && !wait_parity(smem_u32(&s_empty[st]), (u32)(((g / kStages) - 1) & 1))) ||
                        s_abort) {
                        atomicExch(err, 1);
                        s_abort = 1;
                        bad = true;
                        break;
                    }
                    const u32 bar = smem_u32(&s_full[st]), dst = sbase + (u32)st * kStageBytes;
                    expect_tx(bar, n * (kATile + kBTile));
                    bulk_g2s(dst, a + (size_t)s * kATile, n * kATile, bar);
                    bulk_g2s(dst + kOffB, b + (size_t)s * kBTile, n * kBTile, bar);
                }
            }
            // every copy issued has landed before the CTA can leave (bounded)
            for (int x = g - kStages < 0 ? 0 : g - kStages; x < g; ++x)
                wait_parity(smem_u32(&s_full[x % kStages]), (u32)((x / kStages) & 1));
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------ MMA issue
        if (lane == 0) {
            int g = 0, last = -1;
            bool bad = false;
            for (int lt = 0; lt < my_tiles && !bad; ++lt) {
                const int buf = lt & 1;
                if (lt >= 2 && !wait_parity(smem_u32(&s_tfree[buf]), (u32)(((lt >> 1) - 1) & 1))) {
                    atomicExch(err, 3);
                    s_abort = 1;
                    break;
                }
                fence_after();
                for (int s = 0; s < n_kb; s += kSteps, ++g) {
                    const int st = g % kStages;
                    const int n = n_kb - s < kSteps ? n_kb - s : kSteps;
                    if (!wait_parity(smem_u32(&s_full[st]), (u32)((g / kStages) & 1)) || s_abort) {
                        atomicExch(err, 2);
                        s_abort = 1;
                        bad = true;
                        break;
                    }
                    fence_after();
                    const u32 a_addr = sbase + (u32)st * kStageBytes, b_addr = a_addr + kOffB;
#pragma unroll
                    for (int u = 0; u < kSteps; ++u)
                        if (u < n)
                            mma_i8(tmem + (u32)buf * 256u, sdesc(a_addr + (u32)u * kATile, ptc::kLbo, ptc::kSbo),
                                   sdesc(b_addr + (u32)u * kBTile, ptc::kLbo, ptc::kSbo), kIdesc, (s + u) > 0 ? 1u : 0u);
                    commit(smem_u32(&s_empty[st]));
                    last = g;
                }
                if (!bad) commit(smem_u32(&s_tfull[buf]));
            }
            // the last commit covers every MMA issued
            if (last >= 0) wait_parity(smem_u32(&s_empty[last % kStages]), (u32)((last / kStages) & 1));
        }
        __syncwarp();
    } else if (warp < kEpiWarps) {
        // ------------------------------------------------------------- epilogue
        for (int lt = 0; lt < my_tiles; ++lt) {
            const int buf = lt & 1;
            const int t = (int)blockIdx.x + lt * (int)gridDim.x, i = t / per_mod, x = t - i * per_mod;
            const int nt = x / n_mt, mt = x - nt * n_mt;
            const bool bad = !wait_parity(smem_u32(&s_tfull[buf]), (u32)((lt >> 1) & 1));
            if (group_any(kBarEpi, kEpi, bad || s_abort)) {
                if (tid == 0) {
                    atomicExch(err, 4);
                    s_abort = 1;
                }
                break;
            }
            fence_after();
            const u32 m = P.m[i].m, mu = P.m[i].mu;
            const u32 taddr = tmem + ((u32)(32 * warp) << 16) + (u32)buf * 256u;
            uint8_t* out = W + (((size_t)i * n_mt + mt) * 128 + 32 * warp + lane) * ((size_t)n_nt * kN) + (size_t)nt * kN;
#pragma unroll 1
            for (int c0 = 0; c0 < kN; c0 += 32) {
                u32 r[32];
                tmem_ld32(taddr + (u32)c0, r);
                u32 w[8];
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    w[g] = 0;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {  // sums below 2^31: the quotient estimate is at most one short
                        u32 v = r[4 * g + e] - __umulhi(r[4 * g + e], mu) * m;
                        v = v >= m ? v - m : v;
                        w[g] |= v << (8 * e);
                    }
                }
                *(uint4*)(out + c0) = make_uint4(w[0], w[1], w[2], w[3]);
                *(uint4*)(out + c0 + 16) = make_uint4(w[4], w[5], w[6], w[7]);
            }
            fence_before();
            named_sync(kBarEpi, kEpi);  // every lane of the set read
            if (tid == 0) arrive(smem_u32(&s_tfree[buf]));
        }
    }
    // teardown: every role has left its loop (on abort, after a bounded wait)
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == kMmaWarp) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// C [rows][cols] (rows ldc words apart) from W: a thread combines four columns, stored through
// shared memory so that a warp writes consecutive words. A block of 256 threads takes 4 X columns
// of 256 / X rows (narrow outputs several rows: 65536 x 32 x 256, 60 bits, 0.63 -> 0.44 ms).
template <int X>
__global__ void __launch_bounds__(256) k_rns_combine(const uint8_t* __restrict__ W, u64* __restrict__ C, int rows,
                                                     int cols, size_t ldc, size_t plane, size_t pitch,
                                                     const __grid_constant__ Params P) {
    __shared__ __align__(16) u64 so_[1024];
    constexpr int kRows = 256 / X;
    const int tx = threadIdx.x % X, ty = threadIdx.x / X, c0 = blockIdx.x * 4 * X, c = c0 + 4 * tx;
    u64* so = so_ + ty * 4 * X;
    for (int r0 = blockIdx.y * kRows; r0 < rows; r0 += gridDim.y * kRows) {
        const int row = r0 + ty;
        const bool on = kRows == 1 || row < rows;
        if (on && c < cols) {  // pitch is a multiple of 256: the four bytes are inside the row
            const uint8_t* src = W + (size_t)row * pitch + c;
            u32 k[4] = {0, 0, 0, 0};
            u64 lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
            constexpr int kU = 4;  // moduli whose bytes are in flight together
            for (int i0 = 0; i0 < P.n; i0 += kU, src += kU * plane) {
                u32 w4[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) w4[u] = i0 + u < P.n ? __ldcs((const u32*)(src + u * plane)) : 0u;
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const Mod& md = P.m[i0 + u];  // zeros past P.n (kMaxMod is a multiple of kU)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const u32 w = (w4[u] >> (8 * e)) & 255u;
                        k[e] += w * md.recip;
                        lo[e] += (u64)w * md.mq_lo;
                        hi[e] += (u64)w * md.mq_hi;
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const u32 kk = (k[e] + 8192u) >> 27;
                lo[e] += (u64)kk * P.nm_lo;  // lo, hi < 21 * 256 * 2^32 < 2^45
                hi[e] += (u64)kk * P.nm_hi;
                u64 x = mul_shoup_lazy(hi[e], P.r32, P.r32q, P.q) + lo[e];  // below 2 q + 2^45
                x -= __umul64hi(x, P.mu) * P.q;
                x = x >= P.q ? x - P.q : x;
                so[4 * tx + e] = x >= P.q ? x - P.q : x;
            }
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int o = tx + X * e;
            if (on && c0 + o < cols) C[(size_t)row * ldc + c0 + o] = so[o];
        }
        __syncthreads();
    }
}

// moduli whose product exceeds 2 inner (q - 1)^2 with a little to spare (0: not enough of them)
int moduli_for(u32 inner, u64 q) {
    const double need = 1.05 + std::log2((double)inner) + 2.0 * std::log2((double)(q - 1));
    double have = 0;
    for (int n = 0; n < kMaxMod; ++n) {
        have += std::log2((double)kModuli[n]);
        if (have > need) return n + 1;
    }
    return 0;
}

// Whether the residue system takes less time than the byte planes (moduli of at least 4 bytes;
// narrower ones have at most 9 products against 6 to 9 and an extra combining pass), by estimates
// (ps) fitted to both on a B200 (seven moduli of 30 to 60 bits, 46 shapes, within about 10 %).
// An output of the planes costs the epilogue of its nb accumulators or its nb^2 products,
// whichever is longer; one of the residues costs n bytes written and read back and n products,
// with columns padded to 256. Packing an element of lhs or rhs costs the planes 4 or 8 ps more,
// a call 6 us (two packing launches). ms, planes / residues: 35 bits, 4096 x inner x 4096: inner = 64
// 0.182 / 0.304, 512 0.305 / 0.345, 1024 0.470 / 0.418, 4096 1.59 / 0.92; 16384 x 64 x 16384 1.80 / 3.95;
// 60 bits, 4096 x 64 x 4096 0.40 / 0.43, 4096^3 3.68 / 1.41, 65536 x 32 x 16 0.120 / 0.335. Moduli of
// 4 bytes below 2^31 products differ by a few us either way and keep the planes.
bool worthwhile(u32 rows, u32 inner, u32 cols, u64 q) {
    if (q <= (1ull << 24) || q >= (1ull << 62) || inner > (u32)kMaxInner) return false;
    const double r = rows, k = inner, c = cols;
    if (q <= (1ull << 32) && r * k * c < 2147483648.0) return false;
    const int n = moduli_for(inner, q), nb = (64 - __builtin_clzll(q - 1) + 7) / 8, ct = ptc::cols_per_tile(nb);
    if (!n) return false;
    const u64 n_mt = (rows + 127) / 128, n_nt = (cols + kN - 1) / kN;
    if (n_mt * n_nt >= (1ull << 26)) return false;
    const double out = 128.0 * n_mt, planes_out = std::max(nb <= 5 ? 6.5 : 18.0, 0.87e-3 * nb * nb * k);
    const double planes = out * ((cols + ct - 1) / ct * ct) * planes_out + 4 * r * k + 8 * k * c + 6e6;
    return out * n_nt * kN * (2.5 + n * (0.95 + 0.55e-3 * k)) < planes;
}

Params make_params(u32 inner, u64 q) {
    Params P{};
    P.n = moduli_for(inner, q);
    u64 mq = 1 % q;  // M mod q
    for (int i = 0; i < P.n; ++i) mq = (u64)((u128)mq * (u64)kModuli[i] % q);
    for (int i = 0; i < P.n; ++i) {
        const u32 m = (u32)kModuli[i];
        Mod& md = P.m[i];
        u64 oq = 1 % q;
        u32 om = 1 % m, inv = 1;
        for (int j = 0; j < P.n; ++j)
            if (j != i) {
                oq = (u64)((u128)oq * (u64)kModuli[j] % q);
                om = om * (u32)kModuli[j] % m;
            }
        while (om * inv % m != 1) ++inv;
        md.m = m;
        md.mu_small = (u32)(((1ull << 32) + m - 1) / m);
        md.mu = (u32)((1ull << 32) / m);
        u32 ra = 1 % m, rb = inv % m;
        for (int j = 0; j < 8; ++j) {
            (j < 4 ? md.a_lo : md.a_hi) |= ra << (8 * (j & 3));
            (j < 4 ? md.b_lo : md.b_hi) |= rb << (8 * (j & 3));
            ra = ra * 256 % m;
            rb = rb * 256 % m;
        }
        md.recip = (1u << 27) / m;
        md.mq_lo = (u32)oq;
        md.mq_hi = (u32)(oq >> 32);
    }
    P.q = q;
    P.mu = ~0ull / q;
    P.r32 = (1ull << 32) % q;
    P.r32q = (u64)(((u128)P.r32 << 64) / q);
    const u64 nm = mq ? q - mq : 0;
    P.nm_lo = (u32)nm;
    P.nm_hi = (u32)(nm >> 32);
    return P;
}

// Packed operands and W take P.n bytes an element of A, B and C, which for many outputs and a
// short inner sum is far more than the planes' operands. The product is therefore made in slabs
// of rt row tiles and ct column tiles whose workspace stays within what the planes would take,
// or 2 GiB where that is less (a column slab's operand and its W for one row tile within half).
struct Slabs {
    int rt, ct;
};
Slabs slabs_for(u32 rows, u32 inner, u32 cols, u64 q, int n_mod) {
    const int n_mt = (int)((rows + 127) / 128), n_nt = (int)((cols + kN - 1) / kN);
    const size_t step = (size_t)n_mod * ((inner + 31) / 32) * 32;  // packed bytes of a row or column
    const size_t budget = std::max((size_t)2 << 30, ptc::packed_bytes(rows, inner, cols, q));
    auto even = [](int n, size_t most) {  // at most `most` (at least one) of n tiles, equal slabs
        const int k = (int)std::min<size_t>((size_t)n, std::max<size_t>(1, most)), slabs = (n + k - 1) / k;
        return (n + slabs - 1) / slabs;
    };
    Slabs s;
    s.ct = even(n_nt, budget / 2 / (kN * (step + (size_t)128 * n_mod)));
    const size_t b_bytes = (size_t)s.ct * kN * step;
    s.rt = even(n_mt, (budget - b_bytes) / (128 * (step + (size_t)n_mod * s.ct * kN)));
    return s;
}

int32_t run(const u64* lhs, const u64* rhs, u64* out, u32 rows, u32 inner, u32 cols, u64 q, cudaStream_t st) {
    const Params P = make_params(inner, q);
    const Slabs sl = slabs_for(rows, inner, cols, q, P.n);
    const int n_kb = (int)((inner + 31) / 32);
    const u32 slab_rows = (u32)sl.rt * 128, slab_cols = (u32)sl.ct * kN;
    int dev = 0, n_sm = 0;
    CKKS_CUDA_TRY(cudaGetDevice(&dev));
    CKKS_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    return ptc::timed(dev, st, [&](int* err, auto packed) -> int32_t {
        Workspace<uint8_t> ap, bp, w;
        int32_t rc;
        if ((rc = ap.alloc((size_t)P.n * sl.rt * n_kb * kATile, st)) ||
            (rc = bp.alloc((size_t)P.n * sl.ct * n_kb * kBTile, st)) ||
            (rc = w.alloc((size_t)P.n * slab_rows * slab_cols, st)))
            return rc;
        CKKS_CUDA_TRY(cudaFuncSetAttribute(k_rns_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
        bool first = true;
        for (u64 c0 = 0; c0 < cols; c0 += slab_cols)
            for (u64 r0 = 0; r0 < rows; r0 += slab_rows) {
                const u32 nr = (u32)std::min<u64>(slab_rows, rows - r0), nc = (u32)std::min<u64>(slab_cols, cols - c0);
                const int n_mt = (int)((nr + 127) / 128), n_nt = (int)((nc + kN - 1) / kN), b_nt = r0 ? 0 : n_nt;
                const u64* a = lhs + r0 * inner;
                const size_t threads = ((size_t)n_mt * 128 + (size_t)b_nt * kN) * 2 * n_kb, blocks = (threads + 255) / 256;
                const size_t cap = (size_t)n_sm * 16;
                k_rns_pack<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, st>>>(
                    a, rhs + c0, ap.p, bp.p, (int)nr, (int)inner, (int)nc, cols, n_mt, b_nt, n_kb,
                    inner % 2 == 0 && ((uintptr_t)a & 15) == 0, P);
                CKKS_CUDA_TRY(cudaGetLastError());
                if (first && (rc = packed())) return rc;
                first = false;
                const int n_tiles = n_mt * n_nt * P.n;
                k_rns_gemm<<<n_tiles < n_sm ? n_tiles : n_sm, kThreads, kSmemBytes, st>>>(ap.p, bp.p, w.p, n_mt, n_nt,
                                                                                         n_kb, P, err);
                CKKS_CUDA_TRY(cudaGetLastError());
                u32 x = 32;  // threads a row
                while (x < 256 && 4 * x < nc) x *= 2;
                const dim3 g((nc + 4 * x - 1) / (4 * x), std::min<u32>((nr * x + 255) / 256, 65535));
                auto* combine = x == 32    ? k_rns_combine<32>
                                : x == 64  ? k_rns_combine<64>
                                : x == 128 ? k_rns_combine<128>
                                           : k_rns_combine<256>;
                combine<<<g, 256, 0, st>>>(w.p, out + r0 * cols + c0, (int)nr, (int)nc, cols,
                                           (size_t)n_mt * 128 * n_nt * kN, (size_t)n_nt * kN, P);
                CKKS_CUDA_TRY(cudaGetLastError());
            }
        return CKKS_OK;
    });
}

}  // namespace rns

int32_t check_dims(uint32_t rows, uint32_t inner, uint32_t cols, uint64_t q, const char* who) {
    // the reference asserts non-empty operands and a modulus above one (ccmm/park.rs:1489-1505)
    if (rows == 0 || inner == 0 || cols == 0 || q < 2 || rows > 0x7FFFFFFFu || cols > 0x7FFFFFFFu ||
        inner > 0x7FFFFFFFu || (u64)((rows + kTile - 1) / kTile) > 65535u) {
        ckks_set_error(std::string(who) + ": empty operand, modulus below 2 or matrix too large");
        return CKKS_ERR_BAD_ARG;
    }
    return CKKS_OK;
}

}  // namespace

extern "C" {

int32_t ckks_park_mod_pp_mm_with_backend(const uint64_t* lhs, const uint64_t* rhs, uint64_t* out, uint32_t rows,
                                         uint32_t inner, uint32_t cols, uint64_t modulus, int32_t backend,
                                         void* stream) {
    if (int32_t rc = check_dims(rows, inner, cols, modulus, "ckks_park_mod_pp_mm")) return rc;
    CKKS_CHECK_ARG(lhs && rhs && out, "ckks_park_mod_pp_mm: null matrix");
    const bool tc_ok = tc_enabled() && ptc::supported(rows, cols, modulus);
    if (backend == CKKS_PARK_AUTO) backend = tc_ok ? CKKS_PARK_TENSOR_CORES : CKKS_PARK_CUDA_CORES;
    const cudaStream_t st = (cudaStream_t)stream;
    if (backend == CKKS_PARK_TENSOR_CORES) {
        CKKS_CHECK_ARG(tc_ok, "ckks_park_mod_pp_mm: the tensor-core backend needs a compute capability 10.0 device "
                              "and fewer than 2^31 output tiles");
        if (rns::worthwhile(rows, inner, cols, modulus)) {
            // out of memory before any output is written: the planes may still fit
            const int32_t rc = rns::run(lhs, rhs, out, rows, inner, cols, modulus, st);
            if (rc != CKKS_ERR_OOM) return rc;
        }
        return ptc::run(lhs, rhs, out, rows, inner, cols, modulus, st);
    }
    CKKS_CHECK_ARG(backend == CKKS_PARK_CUDA_CORES, "ckks_park_mod_pp_mm: unknown backend");
    const u64 r64 = (u64)(((u128)1 << 64) % modulus);
    const u64 r128 = (u64)((u128)r64 * r64 % modulus);
    dim3 grid((cols + kTile - 1) / kTile, (rows + kTile - 1) / kTile);
    k_park_mm<<<grid, kThreads, 0, st>>>(lhs, rhs, out, (int)rows, (int)inner, (int)cols, modulus, r64, r128);
    CKKS_CUDA_TRY(cudaGetLastError());
    return CKKS_OK;
}

int32_t ckks_park_last_timing(float* pack_ms, float* gemm_ms) {
    CKKS_CHECK_ARG(pack_ms && gemm_ms, "ckks_park_last_timing: null output");
    CKKS_CHECK_ARG(ptc::t_timing.gemm_ms >= 0.f, "ckks_park_last_timing: no tensor-core call on this thread");
    *pack_ms = ptc::t_timing.pack_ms;
    *gemm_ms = ptc::t_timing.gemm_ms;
    return CKKS_OK;
}

int32_t ckks_park_mod_pp_mm(const uint64_t* lhs, const uint64_t* rhs, uint64_t* out, uint32_t rows, uint32_t inner,
                            uint32_t cols, uint64_t modulus, void* stream) {
    return ckks_park_mod_pp_mm_with_backend(lhs, rhs, out, rows, inner, cols, modulus, CKKS_PARK_AUTO, stream);
}

int32_t ckks_park_mod_pp_mm_host(const uint64_t* lhs, const uint64_t* rhs, uint64_t* out, uint32_t rows,
                                 uint32_t inner, uint32_t cols, uint64_t modulus) {
    if (int32_t rc = check_dims(rows, inner, cols, modulus, "ckks_park_mod_pp_mm_host")) return rc;
    CKKS_CHECK_ARG(lhs && rhs && out, "ckks_park_mod_pp_mm_host: null matrix");
    const size_t na = (size_t)rows * inner, nb = (size_t)inner * cols, nc = (size_t)rows * cols;
    u64 *dA = nullptr, *dB = nullptr, *dC = nullptr;
    int32_t rc = CKKS_OK;
    if (cudaMalloc(&dA, na * 8) != cudaSuccess || cudaMalloc(&dB, nb * 8) != cudaSuccess ||
        cudaMalloc(&dC, nc * 8) != cudaSuccess) {
        cudaGetLastError();
        ckks_set_error("ckks_park_mod_pp_mm_host: out of device memory");
        rc = CKKS_ERR_OOM;
    }
    if (rc == CKKS_OK && (cudaMemcpy(dA, lhs, na * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
                          cudaMemcpy(dB, rhs, nb * 8, cudaMemcpyHostToDevice) != cudaSuccess)) {
        ckks_set_error("ckks_park_mod_pp_mm_host: copy to the device failed");
        rc = CKKS_ERR_CUDA;
    }
    if (rc == CKKS_OK) rc = ckks_park_mod_pp_mm(dA, dB, dC, rows, inner, cols, modulus, nullptr);
    if (rc == CKKS_OK && cudaMemcpy(out, dC, nc * 8, cudaMemcpyDeviceToHost) != cudaSuccess) {
        ckks_set_error(std::string("ckks_park_mod_pp_mm_host: ") + cudaGetErrorString(cudaGetLastError()));
        rc = CKKS_ERR_CUDA;
    }
    cudaFree(dA);
    cudaFree(dB);
    cudaFree(dC);
    return rc;
}

}  // extern "C"
