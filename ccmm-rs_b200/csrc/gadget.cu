// gadget.cu -- exact gadget decompositions on the GPU.
//
// Bounded gadget (grafting/bounded_gadget.rs): per coefficient, exact CRT of
// the Q residues, centring against floor(Q/2) (wide_crt.rs:96-111), conversion to a two's complement integer of
// W 64-bit words, then balanced base-2^b digits d_j in [-2^(b-1), 2^(b-1))
// extracted as chunk_j + carry (identical to the reference loop
// residue = value mod B; digit = residue - B if residue >= B/2;
// value = (value - digit) / B, bounded_gadget.rs:75-118). The CRT sums columns of
// 25 bits on the FP64 pipe (k_*_cols); prefixes outside its limits take mixed-radix
// Garner with Shoup constants.
#include <map>
#include <type_traits>

#include "kernels.cuh"
#include "ntt_core.cuh"

namespace {

constexpr int kT = 128;

// Per Q-prefix constants: mixed-radix digits of floor(Q/2) and Q as words.
struct PrefixConst {
    u64* d_half_mr = nullptr;  // [q_limbs]
    u64* d_q_words = nullptr;  // [W]
    int W = 0;
    u32 bits = 0;
    // direct CRT (k_*_cols): columns of 25 bits. NC columns (0: the prefix is too wide);
    // d_inv [2][q_limbs]: (Q / q_i)^-1 mod q_i and its Shoup companion; d_cols [q_limbs + 2][NC]:
    // the signed columns of Q / q_i and of Q, the unsigned ones of floor(Q / 2)
    int NC = 0, pieces = 2;
    u64* d_inv = nullptr;
    double* d_cols = nullptr;
};
constexpr int kColumnSizes[] = {8, 16, 24, 32, 40, 50};

std::mutex g_prefix_mutex;
std::map<std::pair<const ckks_ctx*, u32>, PrefixConst> g_prefix;

typedef unsigned __int128 u128;

int words_for_bits(u32 bits) { return (int)(bits / 64) + 2; }
constexpr int kMaxWords = 66;  // widest k_bounded_decompose / k_crt_to_double instantiation

// Host helpers on little-endian word vectors.
void mul_small_add(std::vector<u64>& x, u64 m, u64 a) {
    u128 carry = a;
    for (auto& w : x) {
        u128 t = (u128)w * m + carry;
        w = (u64)t;
        carry = t >> 64;
    }
}

u64 mulmod_host(u64 a, u64 b, u64 q) { return (u64)((u128)a * b % q); }

// Constants of the direct CRT of a prefix (Q, floor(Q/2) as words).
int32_t column_const(ckks_ctx* ctx, u32 q_limbs, const std::vector<u64>& Q, const std::vector<u64>& half,
                     PrefixConst* pc) {
    for (int nc : kColumnSizes)
        if (!pc->NC && 25 * nc >= (int)pc->bits + 2) pc->NC = nc;
    if (!pc->NC) return CKKS_OK;
    const int NC = pc->NC;
    std::vector<u64> inv(2 * (size_t)q_limbs);
    std::vector<double> cols((size_t)(q_limbs + 2) * NC);
    auto columns = [&](const std::vector<u64>& x, double* dst, bool sgn) {
        int carry = 0;
        for (int c = 0; c < NC; ++c) {
            const int bit = 25 * c, w = bit / 64, o = bit % 64;
            u64 v = w < (int)x.size() ? x[w] >> o : 0;
            if (o > 39 && w + 1 < (int)x.size()) v |= x[w + 1] << (64 - o);
            int d = (int)(v & ((1u << 25) - 1)) + carry;
            carry = sgn && d >= (1 << 24);
            dst[c] = (double)(d - (carry << 25));
        }
    };
    pc->pieces = 2;
    for (u32 i = 0; i < q_limbs; ++i) {
        const u64 qi = ctx->moduli[i];
        if (qi >= (1ull << 50)) pc->pieces = 3;
        std::vector<u64> quo = Q;  // Q / q_i (exact)
        u128 r = 0;
        for (int w = (int)Q.size() - 1; w >= 0; --w) {
            const u128 cur = (r << 64) | quo[w];
            quo[w] = (u64)(cur / qi);
            r = cur % qi;
        }
        columns(quo, cols.data() + (size_t)i * NC, true);
        u64 m = 1 % qi, e = qi - 2, v = 1;  // (Q / q_i mod q_i)^(q_i - 2)
        for (u32 j = 0; j < q_limbs; ++j)
            if (j != i) m = mulmod_host(m, ctx->moduli[j] % qi, qi);
        for (; e; e >>= 1, m = mulmod_host(m, m, qi))
            if (e & 1) v = mulmod_host(v, m, qi);
        inv[i] = v % qi;
        inv[q_limbs + i] = shoup_quotient_host(inv[i], qi);
    }
    columns(Q, cols.data() + (size_t)q_limbs * NC, true);
    columns(half, cols.data() + (size_t)(q_limbs + 1) * NC, false);
    if (cudaMalloc(&pc->d_inv, inv.size() * 8) != cudaSuccess || cudaMalloc(&pc->d_cols, cols.size() * 8) != cudaSuccess ||
        cudaMemcpy(pc->d_inv, inv.data(), inv.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(pc->d_cols, cols.data(), cols.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(pc->d_inv);
        cudaFree(pc->d_cols);
        ckks_set_error("out of device memory for gadget constants");
        return CKKS_ERR_OOM;
    }
    return CKKS_OK;
}

int32_t prefix_const(ckks_ctx* ctx, u32 q_limbs, PrefixConst* out) {
    std::lock_guard<std::mutex> lock(g_prefix_mutex);
    auto key = std::make_pair((const ckks_ctx*)ctx, q_limbs);
    auto it = g_prefix.find(key);
    if (it != g_prefix.end()) {
        *out = it->second;
        return CKKS_OK;
    }
    double lb = 0;
    for (u32 i = 0; i < q_limbs; ++i) lb += std::log2((double)ctx->moduli[i]);
    int W = words_for_bits((u32)lb + 1);
    std::vector<u64> Q(W, 0);
    Q[0] = 1;
    for (u32 i = 0; i < q_limbs; ++i) mul_small_add(Q, ctx->moduli[i], 0);
    u32 bits = 0;
    for (int i = W - 1; i >= 0; --i)
        if (Q[i]) { bits = (u32)(64 * i + 64 - __builtin_clzll(Q[i])); break; }
    // floor(Q/2) and its mixed-radix digits: v_i in [0, q_i), value = sum v_i prod_{j<i} q_j
    std::vector<u64> half(W);
    for (int i = 0; i < W; ++i) half[i] = (Q[i] >> 1) | (i + 1 < W ? (Q[i + 1] << 63) : 0);
    std::vector<u64> mr(q_limbs), rem = half;
    for (u32 i = 0; i < q_limbs; ++i) {  // repeated division by q_i
        u128 r = 0;
        for (int w = W - 1; w >= 0; --w) {
            u128 cur = (r << 64) | rem[w];
            rem[w] = (u64)(cur / ctx->moduli[i]);
            r = cur % ctx->moduli[i];
        }
        mr[i] = (u64)r;
    }
    PrefixConst pc;
    pc.W = W;
    pc.bits = bits;
    // Q as words, zero-padded to the widest kernel instantiation (kernels of
    // width W' >= W read all W' words)
    std::vector<u64> qpad(kMaxWords, 0);
    std::copy(Q.begin(), Q.end(), qpad.begin());
    if (cudaMalloc(&pc.d_half_mr, q_limbs * sizeof(u64)) != cudaSuccess ||
        cudaMalloc(&pc.d_q_words, kMaxWords * sizeof(u64)) != cudaSuccess) {
        cudaGetLastError();
        ckks_set_error("out of device memory for gadget constants");
        return CKKS_ERR_OOM;
    }
    cudaMemcpy(pc.d_half_mr, mr.data(), q_limbs * sizeof(u64), cudaMemcpyHostToDevice);
    cudaMemcpy(pc.d_q_words, qpad.data(), kMaxWords * sizeof(u64), cudaMemcpyHostToDevice);
    if (int32_t rc = column_const(ctx, q_limbs, Q, half, &pc)) {
        cudaFree(pc.d_half_mr);
        cudaFree(pc.d_q_words);
        return rc;
    }
    g_prefix[key] = pc;
    *out = pc;
    return CKKS_OK;
}

// Exact centred CRT of one coefficient in columns of 25 bits on the FP64 pipe, without the
// mixed-radix chain: with u_i = x_i (Q / q_i)^-1 mod q_i, centred,
//   x = sum_i u_i (Q / q_i) - k Q,   k = rint(sum_i u_i / q_i).
// Columns are signed 25-bit digits (|.| <= 2^24) and u_i splits into P such pieces, so a
// product is at most 2^48 and a column of sums an exact double for kRun limbs; a carry pass
// then brings every column below 2^25. k comes from a double sum that is off by under 2^-41
// (at most 64 terms of at most 1/2): only when it lies within 2^-40 of a half is the sign
// open, and then x is compared with floor(Q/2) exactly. Costs P NC fused multiply-adds a
// limb, at four times the rate of the 32 x 32 + 64-bit integer one, against the L / 2 modular
// products and W-word steps a limb of the mixed-radix form: 24 limbs of 50 bits, N = 2^16:
// digits of 16 polynomials 918 -> 517 us, of one 79 -> 42, decode of four 225 -> 93; integer columns
// in the same form took 708, 62 and 196.
// Shared memory (stage_columns): the limbs' constants, then the columns of Q / q_i, of Q and of
// floor(Q/2) (the last unsigned). Returns x < 0 with col its two's complement columns.
struct LimbConst {
    double q, qinv, inv, inv_p;  // (Q / q_i)^-1 mod q_i and its quotient by q_i
    u64 qi, inv_i, inv_q, pad;   // the same as integers, with the Shoup companion
};
template <int NC>
__device__ __forceinline__ void stage_columns(LimbConst* lc, const NttTab* __restrict__ tabs,
                                              const u64* __restrict__ inv, const double* __restrict__ cols,
                                              int q_limbs) {
    double* sh = reinterpret_cast<double*>(lc + q_limbs);
    for (int i = threadIdx.x; i < q_limbs; i += blockDim.x) {
        const u64 q = tabs[i].q, v = inv[i];
        lc[i] = LimbConst{(double)q, 1.0 / (double)q, (double)v, (double)v / (double)q, q, v, inv[q_limbs + i], 0};
    }
    for (int i = threadIdx.x; i < (q_limbs + 2) * NC; i += blockDim.x) sh[i] = cols[i];
    __syncthreads();
}
// carries of 25-bit columns: every column to [-2^24, 2^24], the value unchanged (the last
// column keeps what is left)
template <int NC>
__device__ __forceinline__ void carry_columns(double (&acc)[NC]) {
    constexpr double kM = 6755399441055744.0 * 33554432.0;  // 1.5 * 2^(52 + 25)
#pragma unroll
    for (int c = 0; c + 1 < NC; ++c) {
        const double hi = __dsub_rn(__dadd_rn(acc[c], kM), kM);  // multiple of 2^25
        acc[c] = __dsub_rn(acc[c], hi);
        acc[c + 1] = __fma_rn(hi, 1.0 / 33554432.0, acc[c + 1]);
    }
}
template <int NC, int P>
__device__ __forceinline__ bool crt_columns(const u64* __restrict__ poly, int log_n, int q_limbs, const LimbConst* lc,
                                            u32 (&col)[NC]) {
    constexpr int kRun = P == 2 ? 14 : 9;  // 14 * 2 * 2^48 and 9 * 3 * 2^48 plus a carried column: below 2^53
    constexpr double kM25 = 6755399441055744.0 * 33554432.0, kS25 = 1.0 / 33554432.0;
    const double* sh = reinterpret_cast<const double*>(lc + q_limbs);
    double acc[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = 0.0;
    double frac = 0.0;
    u64 x[3];  // residues of the next limbs, in flight
#pragma unroll
    for (int e = 0; e < 3; ++e) x[e] = e < q_limbs ? __ldg(poly + ((size_t)e << log_n)) : 0;
    for (int i0 = 0; i0 < q_limbs; i0 += kRun) {
        const int i1 = min(i0 + kRun, q_limbs);
#pragma unroll 1
        for (int i = i0; i < i1; ++i) {
            const LimbConst& T = lc[i];
            double p[P];
            if constexpr (P == 2) {  // q below 2^50
                const double u = nttf::center(nttf::mulmod(nttf::from_u52(x[0]), T.inv, T.inv_p, T.q), T.q, T.qinv);
                frac = __fma_rn(u, T.qinv, frac);
                const double hi = __dsub_rn(__dadd_rn(u, kM25), kM25);
                p[0] = __dsub_rn(u, hi);
                p[1] = __dmul_rn(hi, kS25);
            } else {
                const u64 v = mul_shoup(x[0], T.inv_i, T.inv_q, T.qi);
                const i64 u = (i64)(v > (T.qi >> 1) ? v - T.qi : v);
                frac = __fma_rn((double)u, T.qinv, frac);
                const i64 c1 = (u + (1 << 24)) >> 25, c2 = (c1 + (1 << 24)) >> 25;
                p[0] = (double)(int)(u - (c1 << 25));
                p[1] = (double)(int)(c1 - (c2 << 25));
                p[2] = (double)(int)c2;
            }
            x[0] = x[1], x[1] = x[2];
            if (i + 3 < q_limbs) x[2] = __ldg(poly + ((size_t)(i + 3) << log_n));
            const double* Qi = sh + i * NC;
#pragma unroll
            for (int c0 = 0; c0 < NC; c0 += 2) {
                const double2 w = *reinterpret_cast<const double2*>(Qi + c0);
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int j = 0; j < P; ++j)
                        if (c0 + e + j < NC) acc[c0 + e + j] = __fma_rn(p[j], e ? w.y : w.x, acc[c0 + e + j]);
            }
        }
        if (i1 < q_limbs) carry_columns(acc);
    }
    const double k = rint(frac);
    const double *Q = sh + q_limbs * NC, *H = Q + NC;
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = __fma_rn(-k, Q[c], acc[c]);
    carry_columns(acc);
    i64 carry = 0;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const i64 v = (i64)__double2loint(__dadd_rn(acc[c], 6755399441055744.0)) + carry;
        col[c] = (u32)v & ((1u << 25) - 1);
        carry = v >> 25;
    }
    bool neg = carry < 0;
    if (fabs(fabs(__dsub_rn(frac, k)) - 0.5) < 0x1p-40) {  // sign open: |x| against floor(Q/2)
        bool over = false, decided = false;
        u32 mag[NC], cy = neg ? 1u : 0u;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const u32 t = (neg ? (~col[c] & ((1u << 25) - 1)) : col[c]) + cy;
            mag[c] = t & ((1u << 25) - 1);
            cy = t >> 25;
        }
#pragma unroll
        for (int c = NC - 1; c >= 0; --c) {
            const u32 h = (u32)H[c];
            if (!decided && mag[c] != h) {
                over = mag[c] > h;
                decided = true;
            }
        }
        if (over) {  // one Q back towards zero
            i64 cr = 0;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const i64 qc = (i64)Q[c], v = (i64)col[c] + cr + (neg ? qc : -qc);
                col[c] = (u32)v & ((1u << 25) - 1);
                cr = v >> 25;
            }
            neg = !neg;
        }
    }
    return neg;
}

// Resident CTAs asked of the register allocator: left alone it takes 209 to 255 registers by
// unrolling every column's loads ahead, and one or two CTAs an SM.
// Capped: 700-bit digits 27.5 -> 23.8 us (3 polynomials of N = 2^15), 1200-bit decode 104 ->
// 93 us (4 of N = 2^16); the 1200-bit digits are slower capped (41.6 -> 50.7 us).
constexpr int col_ctas(int nc, bool digits) { return nc <= 32 ? 4 : digits ? 0 : 3; }

// k_bounded_decompose for prefixes of up to 1248 bits and bases up to 2^39.
template <int NC, int P>
__global__ void __launch_bounds__(kT, col_ctas(NC, true)) k_bounded_decompose_cols(const u64* __restrict__ poly, i64* __restrict__ digits,
                                                               u32* __restrict__ flags, const NttTab* __restrict__ tabs,
                                                               const u64* __restrict__ inv, const double* __restrict__ cols,
                                                               int q_limbs, int log_n, int base_log, int D,
                                                               size_t poly_stride) {
    extern __shared__ __align__(16) LimbConst lc[];
    stage_columns<NC>(lc, tabs, inv, cols, q_limbs);
    const u32 n = 1u << log_n;
    const u32 c0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (c0 >= n) return;
    u32 col[NC];
    const bool neg = crt_columns<NC, P>(poly + (size_t)blockIdx.y * poly_stride + c0, log_n, q_limbs, lc, col);
    const i64 B = (i64)1 << base_log, half = B >> 1;
    i64* out = digits + ((size_t)blockIdx.y * D << log_n) + c0;
    u64 buf = 0;
    int have = 0, j = 0;
    i64 carry = 0;
    bool flag = false;
    auto emit = [&]() {
        i64 d = (i64)(buf & (u64)(B - 1)) + carry;
        buf >>= base_log;
        have -= base_log;
        carry = d >= half;
        d -= carry ? B : 0;
        flag |= d == -half;
        *out = d;
        out += n;
        ++j;
    };
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        buf |= (u64)col[c] << have;
        have += 25;
        while (have >= base_log && j < D) emit();
        if (j >= D) have = 0, buf = 0;
    }
    while (j < D) {  // sign extension
        buf |= (neg ? (u64)((1u << 25) - 1) : 0ull) << have;
        have += 25;
        while (have >= base_log && j < D) emit();
    }
    if (flags && flag) {  // list of coefficients holding a -B/2 digit: [count][indices]
        u32* fl = flags + (size_t)blockIdx.y * (n + 1);
        fl[1 + atomicAdd(fl, 1u)] = c0;
    }
}

// k_crt_to_double for prefixes of up to 1248 bits.
template <int NC, int P>
__global__ void __launch_bounds__(kT, col_ctas(NC, false)) k_crt_to_double_cols(const u64* __restrict__ poly, double* __restrict__ out,
                                                           const NttTab* __restrict__ tabs, const u64* __restrict__ inv,
                                                           const double* __restrict__ cols, int q_limbs, int log_n,
                                                           double scale) {
    extern __shared__ __align__(16) LimbConst lc[];
    stage_columns<NC>(lc, tabs, inv, cols, q_limbs);
    const u32 n = 1u << log_n;
    const u32 c0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (c0 >= n) return;
    u32 col[NC];
    const bool neg = crt_columns<NC, P>(poly + ((size_t)blockIdx.y * q_limbs << log_n) + c0, log_n, q_limbs, lc, col);
    if (neg) {  // magnitude
        u32 cy = 1;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const u32 t = (~col[c] & ((1u << 25) - 1)) + cy;
            col[c] = t & ((1u << 25) - 1);
            cy = t >> 25;
        }
    }
    // the four leading nonzero columns (at least 76 bits when they are four), the rest as a sticky bit
    u128 w = 0;
    int taken = 0, low = 0;
    bool sticky = false;
#pragma unroll
    for (int c = NC - 1; c >= 0; --c) {
        if (taken == 4) {
            sticky |= col[c] != 0;
        } else if (taken || col[c]) {
            w = (w << 25) | col[c];
            ++taken;
            low = c;
        }
    }
    double r = 0.0;
    const u64 wh = (u64)(w >> 64), wl = (u64)w;
    if (!wh && !sticky) {
        r = ldexp(__ull2double_rn(wl), 25 * low);
    } else {  // 64 leading bits plus a sticky bit round as the whole value
        const int shift = 64 - __clzll(wh);
        u64 lead = shift ? (wh << (64 - shift)) | (wl >> shift) : wl;
        sticky |= shift && (wl << (64 - shift)) != 0;
        if (sticky) lead |= 1;
        r = ldexp(__ull2double_rn(lead), 25 * low + shift);
    }
    r = neg ? -r : r;
    out[(size_t)blockIdx.y * n + c0] = __ddiv_rn(r, scale);
}

// Calls f.template operator()<NC, P>() for the prefix's column count and pieces.
template <typename F>
void with_columns(const PrefixConst& pc, F&& f) {
    auto pick = [&](auto nc) {
        constexpr int NC = decltype(nc)::value;
        if (pc.pieces == 2) f(std::integral_constant<int, NC>{}, std::integral_constant<int, 2>{});
        else f(std::integral_constant<int, NC>{}, std::integral_constant<int, 3>{});
    };
    switch (pc.NC) {
        case 8: pick(std::integral_constant<int, 8>{}); break;
        case 16: pick(std::integral_constant<int, 16>{}); break;
        case 24: pick(std::integral_constant<int, 24>{}); break;
        case 32: pick(std::integral_constant<int, 32>{}); break;
        case 40: pick(std::integral_constant<int, 40>{}); break;
        default: pick(std::integral_constant<int, 50>{});
    }
}

// bits [start, start + len) of a two's complement value, len <= 63
template <int W>
__device__ __forceinline__ u64 field(const u64 (&x)[W], u32 start, u32 len) {
    const u32 wi = start >> 6, off = start & 63;
    const u64 sign = (x[W - 1] >> 63) ? ~0ull : 0ull;
    u64 lo = wi < W ? x[wi] : sign;
    u64 hi = wi + 1 < W ? x[wi + 1] : sign;
    u64 v = off ? ((lo >> off) | (hi << (64 - off))) : lo;
    return v & ((1ull << len) - 1);
}

template <int W>
__global__ void __launch_bounds__(kT) k_bounded_decompose(const u64* __restrict__ poly, i64* __restrict__ digits,
                                                          u32* __restrict__ flags, const NttTab* __restrict__ tabs,
                                                          GarnerQ g, const u64* __restrict__ half_mr,
                                                          const u64* __restrict__ q_words, int q_limbs, int L,
                                                          int log_n, int base_log, int D, size_t poly_stride) {
    const u32 n = 1u << log_n;
    const u32 c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const size_t pbase = (size_t)blockIdx.y * poly_stride;
    // mixed radix (Garner), v kept in registers/local memory
    u64 v[kMaxQ];
    bool neg = false;
    for (int i = 0; i < q_limbs; ++i) {
        const u64 qi = tabs[i].q;
        u64 acc = 0;
        for (int j = 0; j < i; ++j) acc = add_mod(acc, mul_shoup(v[j], g.gq[i * L + j], g.gq_q[i * L + j], qi), qi);
        v[i] = mul_shoup(sub_mod(poly[pbase + ((size_t)i << log_n) + c], acc, qi), g.ginv[i], g.ginv_q[i], qi);
    }
    for (int i = q_limbs - 1; i >= 0; --i) {
        u64 h = half_mr[i];
        if (v[i] != h) { neg = v[i] > h; break; }
    }
    // binary: x = v_{L-1}; x = x * q_i + v_i
    u64 x[W];
#pragma unroll
    for (int w = 0; w < W; ++w) x[w] = 0;
    x[0] = v[q_limbs - 1];
    for (int i = q_limbs - 2; i >= 0; --i) {
        const u64 qi = tabs[i].q;
        u64 carry = v[i];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            u64 lo = x[w] * qi, hi = __umul64hi(x[w], qi);
            lo += carry;
            hi += lo < carry;
            x[w] = lo;
            carry = hi;
        }
    }
    if (neg) {  // x - Q, two's complement
        u64 borrow = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            u64 b = q_words[w] + borrow;
            u64 nb = (b < borrow) | (x[w] < b);
            x[w] -= b;
            borrow = nb;
        }
    }
    const i64 B = (i64)1 << base_log, half = B >> 1;
    i64 carry = 0;
    u32 flag = 0;
    const size_t dbase = (size_t)blockIdx.y * D << log_n;
    for (int j = 0; j < D; ++j) {
        i64 d = (i64)field<W>(x, (u32)j * base_log, base_log) + carry;
        if (d >= half) { d -= B; carry = 1; } else { carry = 0; }
        if (d == -half) flag = 1;
        digits[dbase + ((size_t)j << log_n) + c] = d;
    }
    if (flags && flag) {  // list of coefficients holding a -B/2 digit: [count][indices]
        u32* fl = flags + (size_t)blockIdx.y * (n + 1);
        u32 slot = atomicAdd(fl, 1u);
        fl[1 + slot] = c;
    }
}

// automorphism_hoisted (bounded_gadget.rs:273-312), output-driven:
// out[t] = digits of +-x[s], s = t * k^-1 mod 2N, negation re-normalised with carries.
__global__ void k_digits_automorphism(const i64* __restrict__ in, i64* __restrict__ out, int log_n, int D,
                                      int base_log, u64 k_inv) {
    const u32 n = 1u << log_n;
    const u32 t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const size_t pb = (size_t)blockIdx.y * D << log_n;
    const u64 s = ((u64)t * k_inv) & (2ull * n - 1);
    const u32 src = (u32)(s & (n - 1));
    if (s < n) {
        for (int j = 0; j < D; ++j) out[pb + ((size_t)j << log_n) + t] = in[pb + ((size_t)j << log_n) + src];
        return;
    }
    const i64 B = (i64)1 << base_log, half = B >> 1;
    i64 carry = 0;
    for (int j = 0; j < D; ++j) {
        i64 value = -in[pb + ((size_t)j << log_n) + src] + carry;
        i64 m = (value + half) & (B - 1);  // rem_euclid for a power-of-two base
        i64 normalized = m - half;
        out[pb + ((size_t)j << log_n) + t] = normalized;
        carry = (value - normalized) >> base_log;
    }
}

// Decode support (application_support/ckks.rs:106-130): per coefficient the
// exact CRT value, centred (wide_crt.rs:96-111), rounded to the nearest double
// (ties to even; 64 leading bits plus a sticky bit round exactly as the whole
// value) and divided by the scale.
template <int W>
__global__ void __launch_bounds__(kT) k_crt_to_double(const u64* __restrict__ poly, double* __restrict__ out,
                                                      const NttTab* __restrict__ tabs, GarnerQ g,
                                                      const u64* __restrict__ half_mr, const u64* __restrict__ q_words,
                                                      int q_limbs, int L, int log_n, double scale) {
    const u32 n = 1u << log_n;
    const u32 c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const size_t pbase = (size_t)blockIdx.y * q_limbs << log_n;
    u64 v[kMaxQ];
    for (int i = 0; i < q_limbs; ++i) {
        const u64 qi = tabs[i].q;
        u64 acc = 0;
        for (int j = 0; j < i; ++j) acc = add_mod(acc, mul_shoup(v[j], g.gq[i * L + j], g.gq_q[i * L + j], qi), qi);
        v[i] = mul_shoup(sub_mod(poly[pbase + ((size_t)i << log_n) + c], acc, qi), g.ginv[i], g.ginv_q[i], qi);
    }
    bool neg = false;
    for (int i = q_limbs - 1; i >= 0; --i) {
        if (v[i] != half_mr[i]) { neg = v[i] > half_mr[i]; break; }
    }
    u64 x[W];
#pragma unroll
    for (int w = 0; w < W; ++w) x[w] = 0;
    x[0] = v[q_limbs - 1];
    for (int i = q_limbs - 2; i >= 0; --i) {
        const u64 qi = tabs[i].q;
        u64 carry = v[i];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            u64 lo = x[w] * qi, hi = __umul64hi(x[w], qi);
            lo += carry;
            hi += lo < carry;
            x[w] = lo;
            carry = hi;
        }
    }
    if (neg) {  // magnitude Q - x
        u64 borrow = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            u64 b = x[w] + borrow;
            u64 nb = (b < borrow) | (q_words[w] < b);
            x[w] = q_words[w] - b;
            borrow = nb;
        }
    }
    int top = -1;
#pragma unroll
    for (int w = W - 1; w >= 0; --w)
        if (top < 0 && x[w]) top = w * 64 + 63 - __clzll(x[w]);
    double r = 0.0;
    if (top >= 0 && top < 64) {
        r = __ull2double_rn(x[0]);
    } else if (top >= 64) {
        const int shift = top - 63;
        const int wi = shift >> 6, off = shift & 63;
        u64 lead = off ? ((x[wi] >> off) | (x[wi + 1] << (64 - off))) : x[wi];
        bool sticky = off ? (x[wi] << (64 - off)) != 0 : false;
#pragma unroll
        for (int w = 0; w < W; ++w)
            if (w < wi && x[w]) sticky = true;
        if (sticky) lead |= 1;
        r = ldexp(__ull2double_rn(lead), shift);
    }
    r = neg ? -r : r;
    out[(size_t)blockIdx.y * n + c] = __ddiv_rn(r, scale);
}

u64 galois_inverse(u64 k, u32 n) {
    const u64 two_n = 2ull * n;
    k %= two_n;
    u64 r = 1, b = k, e = n - 1;
    while (e) {
        if (e & 1) r = (r * b) % two_n;
        b = (b * b) % two_n;
        e >>= 1;
    }
    return r;
}

}  // namespace

int32_t bounded_digit_count(ckks_ctx* ctx, u32 q_limbs, u32 base_log, u32* out) {
    CKKS_CHECK_ARG(base_log >= 1 && base_log <= 62, "bounded gadget base_log must be in [1, 62]");
    CKKS_CHECK_ARG(q_limbs >= 1 && q_limbs <= ctx->L, "bounded gadget: Q prefix outside the context basis");
    PrefixConst pc;
    if (int32_t rc = prefix_const(ctx, q_limbs, &pc)) return rc;
    *out = (pc.bits + 1 + base_log - 1) / base_log;  // ceil((bits(Q) + 1) / base_log), bounded_gadget.rs:24-29
    return CKKS_OK;
}

int32_t bounded_decompose_launch(ckks_ctx* ctx, const u64* poly, u32 n_polys, u32 q_limbs, u32 base_log, i64* digits,
                                 u32* flags, cudaStream_t st, size_t poly_stride) {
    if (!poly_stride) poly_stride = (size_t)q_limbs << ctx->log_n;
    u32 D;
    if (int32_t rc = bounded_digit_count(ctx, q_limbs, base_log, &D)) return rc;
    PrefixConst pc;
    if (int32_t rc = prefix_const(ctx, q_limbs, &pc)) return rc;
    if (!n_polys) return CKKS_OK;
    dim3 grid((ctx->n + kT - 1) / kT, n_polys);
    if (pc.NC && base_log <= 39) {
        const size_t smem = q_limbs * sizeof(LimbConst) + (size_t)(q_limbs + 2) * pc.NC * sizeof(double);
        with_columns(pc, [&](auto nc, auto np) {
            k_bounded_decompose_cols<decltype(nc)::value, decltype(np)::value><<<grid, kT, smem, st>>>(
                poly, digits, flags, ctx->d_tabs, pc.d_inv, pc.d_cols, (int)q_limbs, (int)ctx->log_n, (int)base_log,
                (int)D, poly_stride);
        });
        CKKS_CUDA_TRY(cudaGetLastError());
        return CKKS_OK;
    }
#define CKKS_DECOMP(WW)                                                                                          \
    k_bounded_decompose<WW><<<grid, kT, 0, st>>>(poly, digits, flags, ctx->d_tabs, ctx->garner, pc.d_half_mr,     \
                                                 pc.d_q_words, q_limbs, ctx->L, ctx->log_n, base_log, D, poly_stride)
    // wider bases and prefixes: mixed radix
    if (pc.W <= 4) CKKS_DECOMP(4);
    else if (pc.W <= 8) CKKS_DECOMP(8);
    else if (pc.W <= 16) CKKS_DECOMP(16);
    else if (pc.W <= 24) CKKS_DECOMP(24);
    else if (pc.W <= 32) CKKS_DECOMP(32);
    else if (pc.W <= 48) CKKS_DECOMP(48);
    else CKKS_DECOMP(66);
#undef CKKS_DECOMP
    CKKS_CUDA_TRY(cudaGetLastError());
    return CKKS_OK;
}

int32_t digits_automorphism_launch(ckks_ctx* ctx, const i64* in, i64* out, u32 n_polys, u32 D, u32 base_log, u64 k,
                                   cudaStream_t st) {
    CKKS_CHECK_ARG(base_log >= 1 && base_log <= 62, "bounded gadget base_log must be in [1, 62]");
    CKKS_CHECK_ARG((k & 1) == 1, "Galois exponent must be odd");
    if (!n_polys || !D) return CKKS_OK;
    dim3 grid((ctx->n + kT - 1) / kT, n_polys);
    k_digits_automorphism<<<grid, kT, 0, st>>>(in, out, ctx->log_n, D, base_log, galois_inverse(k, ctx->n));
    CKKS_CUDA_TRY(cudaGetLastError());
    return CKKS_OK;
}

int32_t crt_to_double_launch(ckks_ctx* ctx, const u64* poly, u32 n_polys, u32 q_limbs, double scale, double* out,
                             cudaStream_t st) {
    CKKS_CHECK_ARG(q_limbs >= 1 && q_limbs <= ctx->L, "decode: Q prefix outside the context basis");
    PrefixConst pc;
    if (int32_t rc = prefix_const(ctx, q_limbs, &pc)) return rc;
    if (!n_polys) return CKKS_OK;
    dim3 grid((ctx->n + kT - 1) / kT, n_polys);
    if (pc.NC) {
        const size_t smem = q_limbs * sizeof(LimbConst) + (size_t)(q_limbs + 2) * pc.NC * sizeof(double);
        with_columns(pc, [&](auto nc, auto np) {
            k_crt_to_double_cols<decltype(nc)::value, decltype(np)::value><<<grid, kT, smem, st>>>(
                poly, out, ctx->d_tabs, pc.d_inv, pc.d_cols, (int)q_limbs, (int)ctx->log_n, scale);
        });
        CKKS_CUDA_TRY(cudaGetLastError());
        return CKKS_OK;
    }
#define CKKS_CRT(WW)                                                                                                \
    k_crt_to_double<WW><<<grid, kT, 0, st>>>(poly, out, ctx->d_tabs, ctx->garner, pc.d_half_mr, pc.d_q_words,       \
                                             q_limbs, ctx->L, ctx->log_n, scale)
    if (pc.W <= 24) CKKS_CRT(24);  // prefixes beyond the columns' 1248 bits
    else if (pc.W <= 32) CKKS_CRT(32);
    else if (pc.W <= 48) CKKS_CRT(48);
    else CKKS_CRT(66);
#undef CKKS_CRT
    CKKS_CUDA_TRY(cudaGetLastError());
    return CKKS_OK;
}

// Drops the cached prefix constants of a context that is being destroyed (a
// later context may be created at the same address).
void gadget_release_ctx(const ckks_ctx* ctx) {
    std::lock_guard<std::mutex> lock(g_prefix_mutex);
    for (auto it = g_prefix.begin(); it != g_prefix.end();) {
        if (it->first.first == ctx) {
            cudaFree(it->second.d_half_mr);
            cudaFree(it->second.d_q_words);
            cudaFree(it->second.d_inv);
            cudaFree(it->second.d_cols);
            it = g_prefix.erase(it);
        } else {
            ++it;
        }
    }
}
