// mac_f64.cuh -- key-switch MAC of bounded hoisted rotations as exact sums on the
// FP64 pipe, for groups whose (ciphertext, key) pairs are few (included by
// hoisted.cu; same arguments and words as k_mac_tiled plus the base term).
//
//   acc[c][g][comp][l][s] = sum_j Y_c[j][l][s] K_g[j][l][comp][s] (+ P NTT(b_c) on b)  mod q_l
//
// Words are split into pieces whose products and sums are exact doubles, so a
// product costs one FMA per pair of pieces and no reduction:
//   P = 2 (q < 2^50): x centred in (-q/2, q/2], x = x1 + x0 with x0 in
//     [-2^24, 2^24) and x1 a multiple of 2^25, |x1| <= 2^49. Four FMAs into
//     s00 (unit 1), s01 (unit 2^25) and s11 (unit 2^50): a term adds at most
//     2^48, 2 * 2^48 and 2^48 units, so s01 is exact for 16 terms and s00, s11
//     for 32. center() of each (one FMA, exact: the result is an integer below
//     2^53) folds s01 into s00 every kFold terms and s11 every 2 kFold, which
//     leaves s00 room for the centred values it holds (bound at the fold).
//   P = 3 (q < 2^62): 21-bit pieces in [0, 2^21), nine FMAs into five sums of at
//     most 3 * 2^42 a term: exact without folding for up to 680 digits.
// Every residue is the canonical one of the same integer sum, so the words equal
// the tensor-core MAC's and the oracle's.
//
// What bounds it and why this form. The tensor-core MAC costs the same for 1 as
// for 32 keys and for 1 as for 16 ciphertexts (its cost is per item of 4 slots x
// 4 digits, about 1,380 cycles); here the FMAs follow the pairs: 4 per product at
// 64 a clock and SM. The sums take 96 registers a thread, so four warps a scheduler
// cover the FMA and shared-memory latencies: the FP64 pipe is 29 % active (34 % in the
// three-piece form), with no single stall above a third of the issue slots' wait. Leaving out the splitting (13 % of the
// time), the fetches (5 %) or the final reductions (5 %) in timing-only copies shows
// the FMA loop itself holds the rest. Two-digit unrolling (+4 %), 255 registers at
// half the warps (+35 %) and row-wise bulk copies (85 cycles a copy: 2.4x the time)
// were slower. Times by pairs: cheaper_than_tc.
//
// A CTA owns 16 T slots of one limb, every ciphertext of the group and up to 8
// keys. Rows (ciphertexts, then key components) come in by cp.async, kJs digits
// a stage and kStages stages deep; every word is split once into shared memory and
// reused by all its products; a thread sums C ciphertexts x R components of one
// slot. Four neighbouring slots and eight (ciphertext, component) groups share a
// warp, so a warp's operand loads are 64- to 256-byte broadcasts.
#pragma once

namespace macf {

constexpr int kJs = 2;        // digits per stage
constexpr int kStages = 4;    // raw stages (kStages - 1 in flight)
constexpr int kFold = 12;     // terms between folds of s01 (every second fold takes s00 and s11)
// Threads and resident CTAs: two CTAs of 256 hide each other's stage barriers (5 keys, 6
// ciphertexts: 271 -> 196 us against one CTA of 512; equal at 16 ciphertexts); the
// three-piece form keeps one CTA of 512, which splits its words once for twice the keys
// (6 keys, 16 ciphertexts, three 60-bit limbs: 2.16 against 2.55 ms). 128 registers either way.
template <int P>
constexpr int kMaxThreads = P == 2 ? 256 : 512;
constexpr int kKeysMax = 8;  // keys per CTA
constexpr int kMaxDigits = 680;
constexpr int kPitch = 20;   // split words of a 16-slot row
constexpr size_t kMaxSmem = 112 * 1024;   // up to which a CTA takes more tiles (two such CTAs fit an SM)
constexpr size_t kSmemLimit = 160 * 1024;

struct LimbList {
    unsigned char l[kMaxQ + kMaxAux];
};

__device__ __forceinline__ double magic(u32 hi, u32 lo) { return __hiloint2double((int)hi, (int)lo); }

// canonical x < q < 2^50 -> x0, x1 (above)
__device__ __forceinline__ double2 split2(u64 x, u64 q, u64 half) {
    const i64 c = (i64)(x > half ? x - q : x) + (1 << 24);
    const u32 lo = (u32)c & ((1u << 25) - 1);
    const u32 hi = (u32)(int)(c >> 25) + (1u << 25);
    return make_double2(__dsub_rn(magic(0x43300000u, lo), 4503599627370496.0 + 16777216.0),           // 2^52 + 2^24
                        __dsub_rn(magic(0x44C00000u, hi), 0x1p77 + 0x1p50));
}

struct Args {
    const u64* Y;
    size_t y_stride;
    const u64* B;  // NTT(b) [n_ct][Lq][N]
    size_t b_stride;
    const u64* const* keys;
    const u64* exps_inv;
    u64* acc;
    const NttTab* tabs;
    LimbMap lm;
    LimbList limbs;
    int n_ct, n_keys, Lq, LK, D, log_n;
    int T, CG, RG, keys_per_cta;  // 16-slot tiles a CTA, ciphertext and key groups
    const Exc* exc;
    const u32* exc_count;
    int cap;
    const u64* psi;
    const u64 *pf, *pf_q;
};

// The sparse carry corrections of the hoisted digits of one word (rare).
__device__ __noinline__ u64 corrected(const Args& A, u64 v, int c, int g, int comp, int l, u32 s, u64 q, u32 cnt) {
    const NttTab& T = A.tabs[A.lm(l)];
    const Barrett bm{q, T.mu_hi, T.mu_lo};
    const u32 n = 1u << A.log_n;
    const Exc* list = A.exc + ((size_t)c * A.n_keys + g) * A.cap;
    const u64 ps = A.psi[A.lm(l)];
    const u32 k = galois_src(s, A.exps_inv[g], A.log_n);  // unpermuted slot of s
    for (u32 e = 0; e < cnt; ++e) {
        const Exc x = list[e];
        const u64 w = pow_mod_dev(ps, ((2ull * k + 1) * x.t) & (2ull * n - 1), bm);
        u64 dm = x.delta < 0 ? (u64)(-x.delta) % q : (u64)x.delta % q;
        if (x.delta < 0 && dm) dm = q - dm;
        const size_t kofs = (((size_t)x.j * A.LK + l) * 2 + comp) << A.log_n;
        v = add_mod(v, mul_barrett(mul_barrett(w, dm, bm), A.keys[g][kofs + s], bm), q);
    }
    return v;
}

// 16 bytes of a stage: where they come from next, where their two split words go, and
// whether they belong to a key (its digits lie twice as far apart).
struct __align__(16) Piece {
    const u64* src;
    u32 w, key;
};

// A stage holds kJs digits x T tiles of 16 slots x rows; a row is one ciphertext or one
// key component: C rows for each of the CG ciphertext groups, then R rows (b and a of R / 2
// keys) for each of the RG key groups; rows past the last ciphertext or key repeat it
// (their sums are not stored). Split words have a pitch of 20 a row and 4 more after each
// group, so the groups that a warp reads together lie on different banks. Each thread
// fetches, and later splits, its own pieces of every stage.
template <int P, int C, int R>
__global__ void __launch_bounds__(kMaxThreads<P>, 512 / kMaxThreads<P>) k_mac_f64(const __grid_constant__ Args A) {
    constexpr int kSums = P == 2 ? 3 : 5;
    extern __shared__ __align__(128) u64 smem[];
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int l = A.limbs.l[blockIdx.y];
    const u32 s0 = blockIdx.x * (16 * A.T);
    const int g0 = blockIdx.z * A.keys_per_cta;
    const int kn = min(A.keys_per_cta, A.n_keys - g0);
    const int nY = A.CG * C, rows = nY + A.RG * R;
    const u64 q = A.tabs[A.lm(l)].q;
    const size_t y_step = (size_t)A.LK << A.log_n, k_step = 2 * y_step;
    // any carry corrections among this CTA's pairs (lists that overflowed are recomputed elsewhere)
    bool some = false;
    for (int i = tid; i < A.n_ct * kn; i += nthr) {
        const u32 cnt = A.exc_count[(size_t)(i / kn) * A.n_keys + g0 + i % kn];
        some |= cnt && cnt <= (u32)A.cap;
    }
    const int digit_pieces = A.T * rows * 8, n_pieces = kJs * digit_pieces;
    const int tile_words = rows * kPitch + (A.CG + A.RG) * 4, split_words = kJs * A.T * tile_words;
    Piece* piece = reinterpret_cast<Piece*>(smem);                                   // [n_pieces]
    u64* raw = smem + 2 * n_pieces;                                                  // [kStages][n_pieces][2]
    double2* dv = reinterpret_cast<double2*>(raw + 2 * kStages * n_pieces);          // [2][split_words]
    double* dz = reinterpret_cast<double*>(dv + 2 * split_words);                    // P = 3: [2][split_words]
    for (int p = tid; p < n_pieces; p += nthr) {
        int x = p >> 3;
        const int jj = x >= A.T * rows;
        x -= jj * A.T * rows;
        const int tile = x / rows, r = x - tile * rows;
        const u64* src;
        int grp;
        if (r < nY) {
            src = A.Y + (size_t)min(r, A.n_ct - 1) * A.y_stride + jj * y_step;
            grp = r / C;
        } else {
            const int x2 = r - nY, k = min(x2 >> 1, kn - 1);
            src = A.keys[g0 + k] + ((size_t)(x2 & 1) << A.log_n) + jj * k_step + ((size_t)l << A.log_n);
            grp = A.CG + x2 / R;
        }
        piece[p] = Piece{src + ((size_t)l << A.log_n) + s0 + 16 * tile + 2 * (p & 7),
                         (u32)((jj * A.T + tile) * tile_words + r * kPitch + grp * 4 + 2 * (p & 7)), r >= nY};
    }
    const int steps = (A.D + kJs - 1) / kJs;
    const u64 half = q >> 1;
    const u32 raw0 = (u32)__cvta_generic_to_shared(raw);
    auto put = [&](int buf, u32 w, u64 x) {
        if (P == 2) {
            dv[buf + w] = split2(x, q, half);
        } else {
            const double k52 = 4503599627370496.0;
            dv[buf + w] = make_double2(__dsub_rn(magic(0x43300000u, (u32)x & 0x1FFFFFu), k52),
                                       __dsub_rn(magic(0x43300000u, (u32)(x >> 21) & 0x1FFFFFu), k52));
            dz[buf + w] = __dsub_rn(magic(0x43300000u, (u32)(x >> 42)), k52);
        }
    };
    // fetch stage tf (in place of a stage that has been split) and split stage ts
    auto move = [&](int tf, int ts) {
        const bool do_fetch = tf < steps, do_split = ts >= 0 && ts < steps;
        const int n_ok = A.D - tf * kJs < kJs ? digit_pieces : n_pieces;  // past the last digit: zeros
        const u32 dst0 = raw0 + (u32)((tf % kStages) * n_pieces) * 16;
        const u64* in = raw + (ts % kStages) * n_pieces * 2;
        const int buf = (ts & 1) * split_words;
        for (int p = tid; p < n_pieces; p += nthr) {
            const Piece m = piece[p];
            if (do_split) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(in + 2 * p);
                put(buf, m.w, x.x);
                put(buf, m.w + 1, x.y);
            }
            if (do_fetch) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst0 + 16 * (u32)p),
                             "l"(p < n_ok ? m.src : A.Y), "r"(p < n_ok ? 16u : 0u)
                             : "memory");
                piece[p].src = m.src + (m.key ? kJs * k_step : kJs * y_step);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int sub = (tid >> 2) % (A.CG * A.RG), sb = (tid >> 2) / (A.CG * A.RG);
    const int cg = sub % A.CG, rg = sub / A.CG;
    const int w_y = (sb >> 2) * tile_words + cg * (C * kPitch + 4) + (sb & 3) * 4 + (tid & 3);
    const int w_k = (sb >> 2) * tile_words + nY * kPitch + A.CG * 4 + rg * (R * kPitch + 4) + (sb & 3) * 4 + (tid & 3);
    double sum[kSums][C][R];
#pragma unroll
    for (int k = 0; k < kSums; ++k)
#pragma unroll
        for (int i = 0; i < C; ++i)
#pragma unroll
            for (int r = 0; r < R; ++r) sum[k][i][r] = 0.0;
    const double qd = (double)q, qinv = 1.0 / qd;
    const bool corrections = __syncthreads_or(some);
    for (int t = 0; t < kStages - 1; ++t) move(t, -1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    move(steps, 0);
    // one stage: kJs digits
    auto step = [&](int t) {
        // this thread's pieces of stage t + 1 have landed; stage t is split; the split words of
        // stage t - 1 have been used by every thread
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 3) : "memory");
        __syncthreads();
        move(t + kStages - 1, t + 1);
#pragma unroll 1
        for (int jj = 0; jj < kJs; ++jj) {
            const int wb = (t & 1) * split_words + jj * A.T * tile_words;
            const double2 *yv = dv + wb + w_y, *kp = dv + wb + w_k;
            const double *yz = dz + wb + w_y, *kz_ = dz + wb + w_k;
            double2 kv[R];
            double kz[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                kv[r] = kp[r * kPitch];
                if constexpr (P == 3) kz[r] = kz_[r * kPitch];
            }
#pragma unroll
            for (int i = 0; i < C; ++i) {
                const double2 y = yv[i * kPitch];
                if constexpr (P == 2) {
#pragma unroll
                    for (int r = 0; r < R; ++r) sum[1][i][r] = __fma_rn(y.x, kv[r].y, sum[1][i][r]);
#pragma unroll
                    for (int r = 0; r < R; ++r) sum[0][i][r] = __fma_rn(y.x, kv[r].x, sum[0][i][r]);
#pragma unroll
                    for (int r = 0; r < R; ++r) sum[2][i][r] = __fma_rn(y.y, kv[r].y, sum[2][i][r]);
#pragma unroll
                    for (int r = 0; r < R; ++r) sum[1][i][r] = __fma_rn(y.y, kv[r].x, sum[1][i][r]);
                } else {
                    const double z = yz[i * kPitch];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        sum[0][i][r] = __fma_rn(y.x, kv[r].x, sum[0][i][r]);
                        sum[1][i][r] = __fma_rn(y.x, kv[r].y, sum[1][i][r]);
                        sum[2][i][r] = __fma_rn(y.x, kz[r], sum[2][i][r]);
                        sum[3][i][r] = __fma_rn(y.y, kz[r], sum[3][i][r]);
                        sum[4][i][r] = __fma_rn(z, kz[r], sum[4][i][r]);
                        sum[1][i][r] = __fma_rn(y.y, kv[r].x, sum[1][i][r]);
                        sum[2][i][r] = __fma_rn(y.y, kv[r].y, sum[2][i][r]);
                        sum[3][i][r] = __fma_rn(z, kv[r].y, sum[3][i][r]);
                        sum[2][i][r] = __fma_rn(z, kv[r].x, sum[2][i][r]);
                    }
                }
            }
        }
    };
    bool all = false;
    for (int t = 0;;) {
        const int t_end = P == 2 ? min(t + kFold / kJs, steps) : steps;
#pragma unroll 1
        for (; t < t_end; ++t) step(t);
        if (t >= steps) break;
        if constexpr (P == 2) {
            // s01 after kFold terms (12 * 2^49 < 2^53 units), s00 and s11 after 2 kFold: until s00 is centred
            // it holds a centred start, 24 products and the centred s01 of both folds. A centred value is at
            // most q/2 < 2 * 2^48 and the quotient's rounding (2^26 for s01): below 31 * 2^48 < 2^53.
            // center(s11): |s11| / q < 6 q < 2^52.6, so the quotient is off by under 1.8 and |r| < 2.3 q.
#pragma unroll
            for (int i = 0; i < C; ++i)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    sum[0][i][r] = __dadd_rn(sum[0][i][r], nttf::center(sum[1][i][r], qd, qinv));
                    sum[1][i][r] = 0.0;
                    if (all) {
                        sum[0][i][r] = nttf::center(sum[0][i][r], qd, qinv);
                        sum[0][i][r] = nttf::center(__dadd_rn(sum[0][i][r], nttf::center(sum[2][i][r], qd, qinv)), qd,
                                                    qinv);
                        sum[2][i][r] = 0.0;
                    }
                }
            all = !all;
        }
    }
    const u32 s = s0 + sb * 4 + (tid & 3);
    const u64 one_q = (~0ull) / q, c21 = (1ull << 21), c21q = P == 3 ? shoup_quotient_dev(c21, q) : 0;
    const bool base = l < A.Lq;
    const u64 pf = base ? __ldg(A.pf + l) : 0, pfq = base ? __ldg(A.pf_q + l) : 0;
    const size_t row_words = y_step, ct_words = (size_t)A.n_keys * 2 * row_words;
    const int c0 = cg * C, k0 = rg * (R / 2);
    u64* out = A.acc + c0 * ct_words + (size_t)(2 * (g0 + k0)) * row_words + ((size_t)l << A.log_n) + s;
    const u64* bsrc = A.B + (size_t)c0 * A.b_stride + ((size_t)l << A.log_n) + s;
#pragma unroll
    for (int i = 0; i < C; ++i, out += ct_words, bsrc += A.b_stride) {
        if (c0 + i < A.n_ct) {
            const u64 pb = base ? mul_shoup(__ldg(bsrc), pf, pfq, q) : 0;
            u64* o = out;
#pragma unroll
            for (int r = 0; r < R; ++r, o += row_words) {
                u64 v;
                if constexpr (P == 2) {
                    const double m = __dadd_rn(nttf::center(sum[1][i][r], qd, qinv), nttf::center(sum[2][i][r], qd, qinv));
                    v = nttf::to_canonical(__dadd_rn(nttf::center(sum[0][i][r], qd, qinv), m), qd, qinv);
                } else {  // Horner in 2^21 (2^21 < q): every step below 2 q + 2^53 < 2^64
                    v = (u64)__double2ll_rn(sum[4][i][r]);
#pragma unroll
                    for (int j = 3; j >= 0; --j) v = mul_shoup_lazy(v, c21, c21q, q) + (u64)__double2ll_rn(sum[j][i][r]);
                    v = reduce_2q(mul_shoup_lazy(v, 1, one_q, q), q);
                }
                if (!(r & 1) && base) v = add_mod(v, pb, q);
                const int k = k0 + (r >> 1);
                if (k < kn) {
                    if (corrections) {
                        u32 cnt = __ldg(A.exc_count + (size_t)(c0 + i) * A.n_keys + g0 + k);
                        if (cnt && cnt <= (u32)A.cap) v = corrected(A, v, c0 + i, g0 + k, r & 1, l, s, q, cnt);
                    }
                    *o = v;
                }
            }
        }
    }
}

template <int P, int C, int R>
int32_t launch_class(Args a, int n_limbs, cudaStream_t st) {
    if (!n_limbs) return CKKS_OK;
    const int kc = a.n_keys < kKeysMax ? a.n_keys : kKeysMax;
    a.CG = (a.n_ct + C - 1) / C;
    a.keys_per_cta = kc;
    a.RG = (kc + R / 2 - 1) / (R / 2);
    const int per_slot = a.CG * a.RG, n = 1 << a.log_n;
    const int rows = a.CG * C + a.RG * R;
    auto smem_of = [&](int T) {
        return (size_t)kJs * T * (rows * 8 * 16 * (1 + kStages) +
                                  2 * (P == 2 ? 16 : 24) * (rows * kPitch + (a.CG + a.RG) * 4));
    };
    a.T = 1;
    while (a.T < 4 && per_slot * 32 * a.T <= kMaxThreads<P> && 32 * a.T <= n && smem_of(2 * a.T) <= kMaxSmem) a.T *= 2;
    CKKS_CUDA_TRY(cudaFuncSetAttribute(k_mac_f64<P, C, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
    const dim3 grid(n / (16 * a.T), n_limbs, (a.n_keys + kc - 1) / kc);
    k_mac_f64<P, C, R><<<grid, per_slot * 16 * a.T, smem_of(a.T), st>>>(a);
    CKKS_CUDA_TRY(cudaGetLastError());
    return CKKS_OK;
}

// Limbs whose primes lie below 2^50 take the two-piece form, the others the
// three-piece form (half the components a thread: five sums each).
template <int C>
int32_t launch_c(const ckks_ctx* ctx, Args a, cudaStream_t st) {
    LimbList l2{}, l3{};
    int n2 = 0, n3 = 0;
    for (int l = 0; l < a.LK; ++l) {
        if (ctx->moduli[a.lm(l)] < (1ull << 50)) l2.l[n2++] = (unsigned char)l;
        else l3.l[n3++] = (unsigned char)l;
    }
    int32_t rc;
    a.limbs = l2;
    if ((rc = a.n_keys == 1 ? launch_class<2, C, 2>(a, n2, st) : launch_class<2, C, 4>(a, n2, st))) return rc;
    a.limbs = l3;
    return launch_class<3, C, 2>(a, n3, st);
}

// ciphertexts a thread sums
inline int tile_cts(int n_ct) { return n_ct == 1 ? 1 : n_ct > 8 || n_ct % 4 == 0 ? 4 : 2; }

// up to 16 ciphertexts, any number of keys, N >= 16, D <= kMaxDigits, every prime above 2^21
inline int32_t launch(const ckks_ctx* ctx, const Args& a, cudaStream_t st) {
    switch (tile_cts(a.n_ct)) {
        case 1: return launch_c<1>(ctx, a, st);
        case 2: return launch_c<2>(ctx, a, st);
        default: return launch_c<4>(ctx, a, st);
    }
}

// Whether this MAC takes less time than the tensor-core one for a group of n_ct ciphertexts, by
// estimates (us) fitted to both on a B200 (ten rings, chains and bases, 140 groups of 40 to 160 pairs).
// Tensor cores: 5.4 ns a slot and 0.67 ns more for each 4 digits (the base digit with them), for
// every 32 keys begun, whatever the ciphertexts (within 5 %; up to 20 % more for wide limbs at
// N = 2^16). This MAC: a cost a slot and digit for every 8 keys begun (fewer than 8 cost
// (keys + 2) / 10 of that), which grows with the padded ciphertexts and the pieces a prime needs.
// ms, tensor cores / FP64: N = 2^16, 24 50-bit and three 60-bit limbs, D = 38: 16 x 8 21.3 / 14.6,
// 16 x 9 21.3 / 28.7; N = 2^15, 14 60-bit limbs, D = 23: 16 x 7 4.61 / 4.57, 16 x 8 4.45 / 4.72,
// 8 x 20 4.32 / 6.46; N = 2^12, six 50-bit and a 60-bit limb, D = 10: 16 x 9 0.252 / 0.214.
// Carry corrections (-B/2 digits, D N / B of them expected a ciphertext) cost every slot 3.7 ns here
// for a ciphertext and 8 keys, 22 ns there for a ciphertext and 32 keys, whose rows share a warp:
// N = 2^15, 12 50-bit and two 60-bit limbs, base 2^20: 16 x 10 150 / 53 ms, base 2^24 18.7 / 15.2.
inline bool cheaper_than_tc(const ckks_ctx* ctx, const LimbMap& lm, int LK, int D, int base_log, int n_ct,
                            int n_keys) {
    const int tile = tile_cts(n_ct), cts = (n_ct + tile - 1) / tile * tile;
    const double two = 0.25 + 0.035 * cts;  // pieces of a prime below 2^50
    const double three = cts > 8 ? 0.1 * cts : cts == 6 ? 0.92 : 0.22 + 0.063 * cts;
    double limbs = 0;
    for (int l = 0; l < LK; ++l) limbs += ctx->moduli[lm(l)] < (1ull << 50) ? two : three;
    const int eights = (n_keys + kKeysMax - 1) / kKeysMax, chunks = (n_keys + 31) / 32;
    const double keys = n_keys < kKeysMax ? (n_keys + 2) / 10.0 : eights;
    const double slots = (double)LK * ctx->n, corrections = std::ldexp((double)D * ctx->n, -base_log) * n_ct;
    const double f64 = 10.0 + limbs * ctx->n * keys * 0.174e-3 * (D + 14) + slots * eights * 3.7e-3 * corrections;
    const double tc = 40.0 + 1e-3 * slots * chunks * (5.4 + 0.67 * (D / 4 + 1) + 22.0 * corrections);
    return f64 < tc;
}

}  // namespace macf
