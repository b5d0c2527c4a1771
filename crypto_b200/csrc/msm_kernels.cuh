// Curve-templated MSM kernels.  Included by msm_bls.cu and msm_bn.cu, which
// instantiate one launcher table each (so the two curves compile in
// parallel); the host driver in msm.cu only sees MsmLaunchers.
#pragma once
#include "curve.cuh"
#include "msm_desc.cuh"
#include "msm_reduce.cuh"
#include "runtime.cuh"

namespace kb200 {


template <class C>
__global__ void k_table_to_wire(const uint32_t* __restrict__ table, uint8_t* __restrict__ wire,
                                size_t n) {
    using F = typename C::F;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t* t = table + i * 2 * F::N;
    uint8_t* o = wire + i * C::WIRE;
    if (aff_is_inf_words<F>(t)) {
        for (int k = 0; k < C::WIRE; ++k) o[k] = 0;
        return;
    }
    Affine<F> a;
    aff_load(a, t);
    Fe<F> x, y;
    fe_from_mont(x, a.x);
    fe_from_mont(y, a.y);
    fe_to_be_bytes(o, x);
    fe_to_be_bytes(o + F::BYTES, y);
}

// GLV split for BLS12-381 G1: with u = -0xd201000000010000 the curve
// parameter, lambda = u^2 - 1 (128 bits) is a cube root of unity mod r and
// phi(x, y) = (beta2 x, y), beta2 a cube root of unity mod p, acts on G1 as
// [lambda].  A scalar k < r = lambda^2 + lambda + 1 splits as
// k = k1 + k2 lambda with k1 = k mod lambda and k2 = k div lambda, both
// below 2^128, so k P = k1 P + k2 phi(P): twice the points, half the
// windows.  The quotient comes from Barrett reduction with
// mu = floor(2^384 / lambda) (exact for k < r; a correction loop covers the
// bound).  Little-endian 32-bit words.
static __constant__ uint32_t kGlvLambda[4] = {0xffffffff, 0x00000000, 0x0001a402, 0xac45a401};
static __constant__ uint32_t kGlvMu[9] = {0x896c72dd, 0xda5e4f8d, 0x268bf7a3, 0x389f49a7, 0xf6cfee30,
                                   0x63f6e522, 0xe01faadd, 0x7c6becf1, 0x00000001};
// 2^256 mod r: the reference's dropped top carry subtracts 2^256.
static __constant__ uint32_t kR256ModR[8] = {0xfffffffe, 0x00000001, 0x00034802, 0x5884b7fa,
                                      0xecbc4ff5, 0x998c4fef, 0xacc5056f, 0x1824b159};

__device__ __forceinline__ bool geq_words(const uint32_t* a, const uint32_t* b, int n) {
    for (int i = n - 1; i >= 0; --i)
        if (a[i] != b[i]) return a[i] > b[i];
    return true;
}
__device__ __forceinline__ void sub_words(uint32_t* a, const uint32_t* b, int n) {
    uint32_t br = 0;
    for (int i = 0; i < n; ++i) {
        const uint64_t d = (uint64_t)a[i] - b[i] - br;
        a[i] = (uint32_t)d;
        br = (uint32_t)(d >> 63);
    }
}

// k (8 words, < r) -> k1 = k mod lambda, k2 = k div lambda (4 words each).
static __device__ void glv_split(const uint32_t k[8], uint32_t k1[4], uint32_t k2[4]) {
    uint32_t prod[17];
    for (int i = 0; i < 17; ++i) prod[i] = 0;
    for (int i = 0; i < 8; ++i) {
        uint64_t carry = 0;
        for (int j = 0; j < 9; ++j) {
            const uint64_t t = (uint64_t)k[i] * kGlvMu[j] + prod[i + j] + carry;
            prod[i + j] = (uint32_t)t;
            carry = t >> 32;
        }
        prod[i + 9] = (uint32_t)carry;
    }
    uint32_t q[5];
    for (int i = 0; i < 5; ++i) q[i] = prod[12 + i];  // floor(k mu / 2^384)
    // rem = k - q lambda (fits: 0 <= rem < 2^129 before correction)
    uint32_t ql[9];
    for (int i = 0; i < 9; ++i) ql[i] = 0;
    for (int i = 0; i < 5; ++i) {
        uint64_t carry = 0;
        for (int j = 0; j < 4; ++j) {
            const uint64_t t = (uint64_t)q[i] * kGlvLambda[j] + ql[i + j] + carry;
            ql[i + j] = (uint32_t)t;
            carry = t >> 32;
        }
        if (i + 4 < 9) ql[i + 4] = (uint32_t)carry;
    }
    uint32_t rem[8];
    for (int i = 0; i < 8; ++i) rem[i] = k[i];
    sub_words(rem, ql, 8);
    uint32_t lam8[8] = {kGlvLambda[0], kGlvLambda[1], kGlvLambda[2], kGlvLambda[3], 0, 0, 0, 0};
    for (int guard = 0; guard < 4 && geq_words(rem, lam8, 8); ++guard) {
        sub_words(rem, lam8, 8);
        uint32_t c = 1;
        for (int i = 0; i < 5 && c; ++i) {
            q[i] += c;
            c = q[i] == 0;
        }
    }
    for (int i = 0; i < 4; ++i) {
        k1[i] = rem[i];
        k2[i] = q[i];
    }
}

// GLV split for BN254 G1 (Gallant-Lambert-Vanstone, CRYPTO 2001, with
// Babai rounding): the lattice {(x, y) : x + y lambda = 0 mod r} has the
// reduced basis v1 = (a1, -b1), v2 = (a2, b2) (extended Euclid on (r,
// lambda), det = r), a1 = b2 = 0x89d3256894d213e3,
// b1 = 0x6f4d8248eeb859fc8211bbeb7d4f1128, a2 = 0x6f4d8248eeb859fd0be4e1541221250b.
// With cA = round(k b2 / r), cB = round(k b1 / r) -- each computed as
// (k g + 2^383) >> 384, g = round(2^384 b / r) --
//   k1 = k - cA a1 - cB a2,   k2 = cA b1 - cB b2,
// so k1 + k2 lambda = k (mod r) exactly and |k1|, |k2| < 2^126 for every
// k < r.  The halves are signed: their signs go to the entries' sign bits.
static __constant__ uint32_t kBnGlvG2[7] = {0x2fafba64, 0x8fa7d32d, 0x773a6ef2, 0x6eb9c714,
                                            0xc7e0b3d7, 0xd91d232e, 0x00000002};
static __constant__ uint32_t kBnGlvG1[9] = {0x9b9bdffa, 0x86937516, 0x5eaa26d9, 0xa5e38cfb, 0x391eb18d,
                                            0x7a7bd9d4, 0xa773d2cf, 0x4ccef014, 0x00000002};
static __constant__ uint32_t kBnGlvA1[2] = {0x94d213e3, 0x89d32568};
static __constant__ uint32_t kBnGlvB1[4] = {0x7d4f1128, 0x8211bbeb, 0xeeb859fc, 0x6f4d8248};
static __constant__ uint32_t kBnGlvA2[4] = {0x1221250b, 0x0be4e154, 0xeeb859fd, 0x6f4d8248};
static __constant__ uint32_t kBnGlvB2[2] = {0x94d213e3, 0x89d32568};
// 2^256 mod r (BN254): the reference's dropped top carry subtracts 2^256.
static __constant__ uint32_t kBnR256ModR[8] = {0x4ffffffb, 0xac96341c, 0x9f60cd29, 0x36fc7695,
                                               0x7879462e, 0x666ea36f, 0x9a07df2f, 0x0e0a77c1};

// round(k g / 2^384) for k of 8 words and g of ng <= 9 words: nr words out.
static __device__ void mul_round384(const uint32_t k[8], const uint32_t* g, int ng, uint32_t* out,
                                    int nr) {
    uint32_t prod[17];
    for (int i = 0; i < 17; ++i) prod[i] = 0;
    for (int i = 0; i < 8; ++i) {
        uint64_t carry = 0;
        for (int j = 0; j < ng; ++j) {
            const uint64_t t = (uint64_t)k[i] * g[j] + prod[i + j] + carry;
            prod[i + j] = (uint32_t)t;
            carry = t >> 32;
        }
        prod[i + ng] = (uint32_t)carry;
    }
    // + 2^383 (bit 31 of word 11), then the words from 12 up
    uint64_t cy = (uint64_t)prod[11] + 0x80000000u;
    prod[11] = (uint32_t)cy;
    cy >>= 32;
    for (int i = 12; i < 17; ++i) {
        cy += prod[i];
        prod[i] = (uint32_t)cy;
        cy >>= 32;
    }
    for (int i = 0; i < nr; ++i) out[i] = prod[12 + i];
}

// acc (8 words, two's complement) += sgn * (a (na words) * b (nb words)).
static __device__ void mac_signed(uint32_t acc[8], const uint32_t* a, int na, const uint32_t* b,
                                  int nb, bool subtract) {
    uint32_t t[8];
    for (int i = 0; i < 8; ++i) t[i] = 0;
    for (int i = 0; i < na; ++i) {
        uint64_t carry = 0;
        for (int j = 0; j < nb && i + j < 8; ++j) {
            const uint64_t v = (uint64_t)a[i] * b[j] + t[i + j] + carry;
            t[i + j] = (uint32_t)v;
            carry = v >> 32;
        }
        if (i + nb < 8) t[i + nb] = (uint32_t)carry;
    }
    if (subtract) {
        sub_words(acc, t, 8);
    } else {
        uint64_t cy = 0;
        for (int i = 0; i < 8; ++i) {
            cy += (uint64_t)acc[i] + t[i];
            acc[i] = (uint32_t)cy;
            cy >>= 32;
        }
    }
}

// Two's complement (8 words) -> magnitude (4 words) and sign.
static __device__ void signed_to_mag(const uint32_t v[8], uint32_t mag[4], uint32_t& neg) {
    neg = v[7] >> 31;
    uint32_t cy = neg;
    for (int i = 0; i < 4; ++i) {
        const uint64_t x = (uint64_t)(neg ? ~v[i] : v[i]) + cy;
        mag[i] = (uint32_t)x;
        cy = (uint32_t)(x >> 32);
    }
}

// k (8 words, < r) -> |k1|, |k2| (4 words each) and their signs.
static __device__ void glv_split_bn(const uint32_t k[8], uint32_t k1[4], uint32_t k2[4],
                                    uint32_t& neg1, uint32_t& neg2) {
    uint32_t cA[2], cB[4];
    mul_round384(k, kBnGlvG2, 7, cA, 2);
    mul_round384(k, kBnGlvG1, 9, cB, 4);
    uint32_t a1[2] = {kBnGlvA1[0], kBnGlvA1[1]};
    uint32_t a2[4] = {kBnGlvA2[0], kBnGlvA2[1], kBnGlvA2[2], kBnGlvA2[3]};
    uint32_t b1[4] = {kBnGlvB1[0], kBnGlvB1[1], kBnGlvB1[2], kBnGlvB1[3]};
    uint32_t b2[2] = {kBnGlvB2[0], kBnGlvB2[1]};
    uint32_t s1[8], s2[8];
    for (int i = 0; i < 8; ++i) {
        s1[i] = k[i];
        s2[i] = 0;
    }
    mac_signed(s1, cA, 2, a1, 2, true);
    mac_signed(s1, cB, 4, a2, 4, true);
    mac_signed(s2, cA, 2, b1, 4, false);
    mac_signed(s2, cB, 4, b2, 2, true);
    signed_to_mag(s1, k1, neg1);
    signed_to_mag(s2, k2, neg2);
}

// Signed-digit recoding, one thread per scalar of the batch.  Entry (w, j)
// of item i lives at entry_base_i + w * n_i + j (GLV items: k1's digit at
// entry_base_i + w * 2 n_i + j, k2's at entry_base_i + w * 2 n_i + n_i + j).
// quirk_c: 0, or the reference window size (4 or 8) whose dropped top carry
// is reproduced by negating (s, P) -> (2^256 - s, -P) for s above the
// carry threshold 0x8888...88 (c = 4) or 0x8080...80 (c = 8).
template <class C>
__global__ void k_recode(const ItemDesc* __restrict__ items, uint32_t n_items,
                         unsigned long long first, unsigned long long count,
                         const uint32_t* __restrict__ scalars,
                         const uint32_t* __restrict__ table, uint32_t* __restrict__ keys,
                         uint32_t* __restrict__ vals) {
    using F = typename C::F;
    const unsigned long long idx = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= count) return;
    const unsigned long long g = first + idx;  // scalar index over all items
    // item: largest i with items[i].scalar_off <= g
    uint32_t lo = 0, hi = n_items;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (items[mid].scalar_off <= g)
            lo = mid;
        else
            hi = mid;
    }
    const ItemDesc it = items[lo];
    if (g < it.scalar_off || g - it.scalar_off >= it.n) return;  // gap between items
    const uint32_t j = (uint32_t)(g - it.scalar_off);
    const uint32_t row = it.point_off + j;
    // Without a table (points still in flight) infinity points get entries
    // too: every later stage skips infinity rows.
    const bool inf = table && aff_is_inf_words<F>(table + (size_t)row * 2 * F::N);
    uint32_t s[8];
    const uint4* sp = reinterpret_cast<const uint4*>(scalars + g * 8);
    const uint4 a = sp[0], b = sp[1];
    s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
    s[4] = b.x; s[5] = b.y; s[6] = b.z; s[7] = b.w;
    uint32_t neg = 0;
    bool dropped_carry = false;
    if (it.quirk_c == 4 || it.quirk_c == 8) {
        const uint32_t t = it.quirk_c == 4 ? 0x88888888u : 0x80808080u;
        int gt = 0;
#pragma unroll
        for (int k = 7; k >= 0; --k) {
            if (gt == 0) {
                if (s[k] > t) gt = 1;
                else if (s[k] < t) gt = -1;
            }
        }
        dropped_carry = gt == 1;
    }
    const int c = (int)it.c;
    const uint32_t M = it.M;
    const uint32_t mask = (1u << c) - 1u;
    // Signed digits of the nw-word scalar sc over the item's W windows; the
    // digit of window w goes to entry slot0 + w * wstride with point row prow.
    auto emit = [&](const uint32_t* sc, int nw, uint32_t prow, unsigned long long slot0,
                    unsigned long long wstride, uint32_t negbit) {
        uint32_t carry = 0;
        for (int w = 0; w < (int)it.W; ++w) {
            const int off = w * c;
            const int wd = off >> 5, sh = off & 31;
            uint32_t raw = 0;
            if (wd < nw) {
                const uint64_t lo64 = sc[wd];
                const uint64_t hi64 = (wd + 1 < nw) ? sc[wd + 1] : 0;
                raw = (uint32_t)(((hi64 << 32) | lo64) >> sh) & mask;
            }
            uint32_t d = raw + carry;
            uint32_t sign = 0;
            // a GLV half's top window stays unsigned: nothing carries past it
            if (d > M && !(it.glv && w == (int)it.W - 1)) {
                d = (1u << c) - d;
                sign = 1;
                carry = 1;
            } else {
                carry = 0;
            }
            const unsigned long long slot = slot0 + (unsigned long long)w * wstride;
            if (d == 0 || inf) {
                keys[slot] = KEY_SENTINEL;
            } else if (it.chunk_rows) {
                keys[slot] = (j / it.chunk_rows) * it.chunk_stride + it.bucket_base +
                             (uint32_t)w * M + (d - 1);
                vals[slot] = prow | ((sign ^ negbit) << 31);
            } else if (it.row_stride) {
                // shifted table: level w holds 2^(c*w) times the point, so every
                // window feeds the same buckets
                keys[slot] = it.bucket_base + (d - 1);
                vals[slot] = (prow + (uint32_t)w * it.row_stride) | ((sign ^ negbit) << 31);
            } else {
                keys[slot] = it.bucket_base + (uint32_t)w * M + (d - 1);
                vals[slot] = prow | ((sign ^ negbit) << 31);
            }
        }
    };
    if constexpr (C::CURVE_ID == 2) {
        if (it.glv) {
            // k = s mod r (s < 2^256 < 3r), minus 2^256 where the reference
            // drops its top carry
            uint32_t k[8], r8[8];
            for (int i = 0; i < 8; ++i) {
                k[i] = s[i];
                r8[i] = FrBLS::P(i);
            }
            for (int guard = 0; guard < 3 && geq_words(k, r8, 8); ++guard) sub_words(k, r8, 8);
            if (dropped_carry) {
                uint32_t t[8];
                for (int i = 0; i < 8; ++i) t[i] = kR256ModR[i];
                if (geq_words(k, t, 8)) {
                    sub_words(k, t, 8);
                } else {  // k + r - t
                    uint64_t cy = 0;
                    for (int i = 0; i < 8; ++i) {
                        cy += (uint64_t)k[i] + r8[i];
                        k[i] = (uint32_t)cy;
                        cy >>= 32;
                    }
                    sub_words(k, t, 8);
                }
            }
            uint32_t k1[4], k2[4];
            glv_split(k, k1, k2);
            const unsigned long long base = it.entry_base + j;
            emit(k1, 4, row, base, 2ull * it.n, 0u);
            emit(k2, 4, row + it.glv_off, base + it.n, 2ull * it.n, 0u);
            return;
        }
    }
    if constexpr (C::CURVE_ID == 1) {
        if (it.glv) {
            // k = s mod r (s < 2^256 < 6r), minus 2^256 where the reference
            // drops its top carry; signed halves, signs into the entries
            uint32_t k[8], r8[8];
            for (int i = 0; i < 8; ++i) {
                k[i] = s[i];
                r8[i] = FrBN::P(i);
            }
            for (int guard = 0; guard < 6 && geq_words(k, r8, 8); ++guard) sub_words(k, r8, 8);
            if (dropped_carry) {
                uint32_t t[8];
                for (int i = 0; i < 8; ++i) t[i] = kBnR256ModR[i];
                if (geq_words(k, t, 8)) {
                    sub_words(k, t, 8);
                } else {  // k + r - t
                    uint64_t cy = 0;
                    for (int i = 0; i < 8; ++i) {
                        cy += (uint64_t)k[i] + r8[i];
                        k[i] = (uint32_t)cy;
                        cy >>= 32;
                    }
                    sub_words(k, t, 8);
                }
            }
            uint32_t k1[4], k2[4], n1, n2;
            glv_split_bn(k, k1, k2, n1, n2);
            const unsigned long long base = it.entry_base + j;
            emit(k1, 4, row, base, 2ull * it.n, n1);
            emit(k2, 4, row + it.glv_off, base + it.n, 2ull * it.n, n2);
            return;
        }
    }
    if (dropped_carry) {
        uint32_t cy = 1;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint64_t v = (uint64_t)(~s[k]) + cy;
            s[k] = (uint32_t)v;
            cy = (uint32_t)(v >> 32);
        }
        neg = 1;
    }
    emit(s, 8, row, it.entry_base + j, (unsigned long long)it.n, neg);
}

// Wire points (big-endian x || y, all-zero = infinity) -> table rows, read
// in 16-byte pieces when the wire base is 16-byte aligned (rows are 64 or
// 96 bytes), byte by byte otherwise.  glv_stride: 0, or the row distance of
// the GLV rows: row i + glv_stride gets phi(P_i) = (beta x, y) (beta2 on
// BLS12-381).
template <class C, bool V16>
__global__ void k_wire_to_table(const uint8_t* __restrict__ wire, uint32_t* __restrict__ table,
                                size_t n, size_t glv_stride) {
    using F = typename C::F;
    constexpr int N = F::N;
    static_assert(C::WIRE == 8 * N, "wire row = two N-word coordinates");
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t m[2 * N];  // the row's 4-byte groups in memory order
    if constexpr (V16) {
        const uint4* s = reinterpret_cast<const uint4*>(wire + i * C::WIRE);
#pragma unroll
        for (int k = 0; k < N / 2; ++k) {
            const uint4 v = s[k];
            m[4 * k] = v.x;
            m[4 * k + 1] = v.y;
            m[4 * k + 2] = v.z;
            m[4 * k + 3] = v.w;
        }
    } else {
        const uint8_t* w = wire + i * C::WIRE;
#pragma unroll
        for (int q = 0; q < 2 * N; ++q)
            m[q] = (uint32_t)w[4 * q] | ((uint32_t)w[4 * q + 1] << 8) | ((uint32_t)w[4 * q + 2] << 16) |
                   ((uint32_t)w[4 * q + 3] << 24);
    }
    uint32_t any = 0;
#pragma unroll
    for (int q = 0; q < 2 * N; ++q) any |= m[q];
    uint32_t* dst = table + i * 2 * N;
    Fe<F> x, y;
    if (!any) {
        fe_zero(x);
        fe_zero(y);
        x.v[N - 1] = INF_FLAG;
        fe_store16(dst, x);
        fe_store16(dst + N, y);
        if (glv_stride) {
            fe_store16(dst + glv_stride * 2 * N, x);
            fe_store16(dst + glv_stride * 2 * N + N, y);
        }
        return;
    }
    // limb l (little-endian words) = the big-endian group N - 1 - l, bytes swapped
#pragma unroll
    for (int l = 0; l < N; ++l) {
        x.v[l] = __byte_perm(m[N - 1 - l], 0, 0x0123);
        y.v[l] = __byte_perm(m[2 * N - 1 - l], 0, 0x0123);
    }
    fe_to_mont(x, x);
    fe_to_mont(y, y);
    fe_store16(dst, x);
    fe_store16(dst + N, y);
    if (glv_stride) {
        Fe<F> b;
#pragma unroll
        for (int k = 0; k < N; ++k) b.v[k] = C::CURVE_ID == 2 ? kGlvBeta2Mont[k] : kBnGlvBetaMont[k % 8];
        fe_mul(x, x, b);
        fe_store16(dst + glv_stride * 2 * N, x);
        fe_store16(dst + glv_stride * 2 * N + N, y);
    }
}


template <class F>
__device__ __forceinline__ void load_table_point(Affine<F>& a, const uint32_t* table, uint32_t idx) {
    const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)idx * 2 * F::N);
    uint32_t w[2 * F::N];
#pragma unroll
    for (int k = 0; k < F::N / 2; ++k) {
        const uint4 v = src[k];
        w[4 * k] = v.x;
        w[4 * k + 1] = v.y;
        w[4 * k + 2] = v.z;
        w[4 * k + 3] = v.w;
    }
    aff_load(a, w);
}

// Bucket holding sorted entry e: the largest b with offsets[b] <= e (empty
// buckets share their successor's offset, so the largest one is the
// non-empty bucket that owns e).
__device__ __forceinline__ uint32_t bucket_of(const uint32_t* offsets, uint32_t B, uint32_t e) {
    uint32_t lo = 0, hi = B;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (offsets[mid] <= e)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// Level 1, persistent: CTAs pull units of blockDim.x chunks from *queue.
// Lane t sums chunk t = entries [tK, tK + K) of the bucket-sorted list
// with mixed XYZZ additions, flushing at bucket boundaries: the run of the
// chunk's first bucket goes to rec_first[t], the run of its last bucket (if
// different) to rec_last[t], runs of buckets strictly inside the chunk
// straight to buckets[].  Every lane does exactly K additions (the last
// chunk fewer), whatever the bucket sizes.
// The running sum lives in shared memory (SmXyzz), so registers hold only
// the formula's temporaries and more warps stay resident to hide the
// latency of the dependent multiply chains.
template <class C>
__global__ void __launch_bounds__(128, C::ACC_MIN_BLOCKS) k_accumulate(AccArgs a) {
    using F = typename C::F;
    constexpr int PW = 4 * F::N;
    __shared__ uint32_t unit;
    __shared__ uint32_t s_acc[4 * F::N * 128];
    const SmXyzz<F, 128> acc{s_acc + threadIdx.x};
    // Only non-zero digits were sorted: the list length is offsets[B].
    const uint32_t L = a.offsets[a.B];
    const uint32_t nchunks = (L + a.K - 1) / a.K;
    for (;;) {
        if (threadIdx.x == 0) unit = atomicAdd(a.queue, 1u);
        __syncthreads();
        const uint32_t base = unit * blockDim.x;
        __syncthreads();
        if (base >= nchunks) return;
        const uint32_t t = base + threadIdx.x;
        if (t < nchunks) {
            const uint32_t e0 = t * a.K;
            const uint32_t e1 = min(e0 + a.K, L);
            uint32_t b = bucket_of(a.offsets, a.B, e0);
            uint32_t bend = a.offsets[b + 1];
            uint32_t run0 = e0;
            acc.set_inf();
            uint32_t v = a.sorted ? a.sorted[e0] : e0;
            for (uint32_t e = e0; e < e1; ++e) {
                if (e == bend) {
                    // flush the finished run [run0, e) of bucket b
                    uint32_t* dst = (run0 == e0) ? a.rec_first + (size_t)t * PW
                                                 : a.buckets + (size_t)b * PW;
                    acc.to_global(dst);
                    acc.set_inf();
                    while (a.offsets[b + 1] <= e) ++b;
                    bend = a.offsets[b + 1];
                    run0 = e;
                }
                const uint32_t vn = (e + 1 < e1) ? (a.sorted ? a.sorted[e + 1] : e + 1) : 0u;
                if (e + 1 < e1) {
                    const uint32_t* nxt = a.table + (size_t)(vn & 0x7fffffffu) * 2 * F::N;
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(nxt));
                }
                const uint32_t* row = a.table + (size_t)(v & 0x7fffffffu) * 2 * F::N;
                if (!aff_is_inf_words<F>(row)) {  // pairing levels can produce infinity
                    Affine<F> p;
                    load_table_point<F>(p, a.table, v & 0x7fffffffu);
                    if (v >> 31) fe_neg(p.y, p.y);
                    xyzz_add_affine(acc, p);
                }
                v = vn;
            }
            uint32_t* dst = (run0 == e0) ? a.rec_first + (size_t)t * PW : a.rec_last + (size_t)t * PW;
            acc.to_global(dst);
        }
    }
}

// ---- Batch-affine pairing levels -------------------------------------------
// One level halves every bucket's run: slot k of bucket b adds input points
// i0 = in_off[b] + 2 (k - out_off[b]) and i0 + 1 (if still in the run) in
// affine coordinates,
//   lambda = (y1 - y0) / (x1 - x0)  (or 3 x0^2 / 2 y0 when the points are
//   equal), x3 = lambda^2 - x0 - x1, y3 = lambda (x0 - x3) - y0,
// with infinity where they cancel.  The denominators are inverted together
// (Montgomery's trick, one field inversion per block of k_inv_wide):
//   k_pair_fwd   thread t owns slots [PAIR_J t, PAIR_J t + PAIR_J): running
//                products of its denominators (prefixes to HBM), total to tot[t];
//   k_inv_wide   every total replaced by its inverse: blocks of INV_T
//                threads, each thread chaining up to INV_G totals, warp-shuffle
//                prefix/suffix products over threads and over warps, one
//                inversion per block;
//   k_pair_bwd   per thread, backwards over its slots: the slot's inverse from
//                its prefix, then the affine sum.
// Per addition: 1 product forward, 2 to recover the inverse, 3 for the sum,
// plus about 4/PAIR_J for the totals' inversion, against 10 for a mixed XYZZ
// addition.  Field
// elements in the scratch arrays are stored word-major (word q of element e
// at q * stride + e) so that consecutive threads touch consecutive words.
enum PairCase : int { PAIR_PASS0 = 0, PAIR_PASS1 = 1, PAIR_INF = 2, PAIR_ADD = 3, PAIR_DBL = 4 };

template <class F>
__device__ __forceinline__ void fe_load_wm(Fe<F>& x, const uint32_t* v, size_t stride, size_t e) {
#pragma unroll
    for (int q = 0; q < F::N; ++q) x.v[q] = v[(size_t)q * stride + e];
}
template <class F>
__device__ __forceinline__ void fe_store_wm(uint32_t* v, size_t stride, size_t e, const Fe<F>& x) {
#pragma unroll
    for (int q = 0; q < F::N; ++q) v[(size_t)q * stride + e] = x.v[q];
}

// Rows of the two operands of input position i (level 0: a table row by
// sorted index, sign in bit 31; later levels: the previous level's rows).
template <class F>
__device__ __forceinline__ const uint32_t* pair_row(const PairArgs& a, uint32_t i, bool& neg) {
    if (a.sorted) {
        const uint32_t v = a.sorted[i];
        neg = (v >> 31) != 0;
        return a.src + (size_t)(v & 0x7fffffffu) * 2 * F::N;
    }
    neg = false;
    return a.src + (size_t)i * 2 * F::N;
}

// W consecutive words (W a multiple of 4, src and dst 16-byte aligned: rows
// are 2N words and N is a multiple of 4) in 16-byte accesses.
template <int W>
__device__ __forceinline__ void ld_words16(uint32_t* w, const uint32_t* src) {
    const uint4* s = reinterpret_cast<const uint4*>(src);
#pragma unroll
    for (int k = 0; k < W / 4; ++k) {
        const uint4 v = s[k];
        w[4 * k] = v.x;
        w[4 * k + 1] = v.y;
        w[4 * k + 2] = v.z;
        w[4 * k + 3] = v.w;
    }
}
template <int W>
__device__ __forceinline__ void st_words16(uint32_t* dst, const uint32_t* w) {
    uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int k = 0; k < W / 4; ++k) d[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
}

template <class F>
__device__ __forceinline__ void pair_load(const PairArgs& a, uint32_t i, Affine<F>& P, bool& inf) {
    bool neg;
    const uint32_t* row = pair_row<F>(a, i, neg);
    uint32_t w[2 * F::N];
    ld_words16<2 * F::N>(w, row);
    inf = aff_is_inf_words<F>(w);
    aff_load(P, w);
    if (neg) fe_neg(P.y, P.y);
}

// Output row of a pairing slot: affine (x, y), or the infinity flag.
template <class F>
__device__ __forceinline__ void pair_store(uint32_t* dst, const Fe<F>& x, const Fe<F>& y) {
    uint32_t w[2 * F::N];
#pragma unroll
    for (int q = 0; q < F::N; ++q) {
        w[q] = x.v[q];
        w[F::N + q] = y.v[q];
    }
    st_words16<2 * F::N>(dst, w);
}

// Loads slot k's operands (bucket b) and classifies it; den is the
// denominator that joins the batch inversion (one for the non-additions).
template <class F>
__device__ __forceinline__ int pair_setup(const PairArgs& a, uint32_t k, uint32_t b, Affine<F>& P0,
                                          Affine<F>& P1, bool& inf0, Fe<F>& den) {
    const uint32_t i0 = a.in_off[b] + 2 * (k - a.out_off[b]);
    const bool has1 = i0 + 1 < a.in_off[b + 1];
    bool inf1 = true;
    pair_load<F>(a, i0, P0, inf0);
    if (has1) pair_load<F>(a, i0 + 1, P1, inf1);
    fe_one(den);
    if (inf1) return PAIR_PASS0;
    if (inf0) return PAIR_PASS1;
    if (!fe_eq(P0.x, P1.x)) {
        fe_sub(den, P1.x, P0.x);
        return PAIR_ADD;
    }
    if (fe_eq(P0.y, P1.y) && !fe_is_zero(P0.y)) {
        fe_dbl(den, P0.y);
        return PAIR_DBL;
    }
    return PAIR_INF;
}

// Only the denominator of slot k: the x coordinates, and the y coordinates
// when the x are equal.  Matches pair_setup's den in every case.
template <class F>
__device__ __forceinline__ void pair_den(const PairArgs& a, uint32_t k, uint32_t b, Fe<F>& den) {
    fe_one(den);
    const uint32_t i0 = a.in_off[b] + 2 * (k - a.out_off[b]);
    if (i0 + 1 >= a.in_off[b + 1]) return;
    bool n0, n1;
    const uint32_t* r0 = pair_row<F>(a, i0, n0);
    const uint32_t* r1 = pair_row<F>(a, i0 + 1, n1);
    Fe<F> x0, x1;
    ld_words16<F::N>(x0.v, r0);
    ld_words16<F::N>(x1.v, r1);
    if (aff_is_inf_words<F>(x0.v) || aff_is_inf_words<F>(x1.v)) return;
    if (!fe_eq(x0, x1)) {
        fe_sub(den, x1, x0);
        return;
    }
    Fe<F> y0, y1;
    fe_load(y0, r0 + F::N);
    fe_load(y1, r1 + F::N);
    if (n0) fe_neg(y0, y0);
    if (n1) fe_neg(y1, y1);
    if (fe_eq(y0, y1) && !fe_is_zero(y0)) fe_dbl(den, y0);
}

template <class C>
__global__ void __launch_bounds__(256) k_pair_fwd(PairArgs a, uint32_t T, uint32_t* __restrict__ pre,
                                                  uint32_t* __restrict__ tot) {
    using F = typename C::F;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const uint32_t total = a.out_off[a.B];  // slots out_off[0] .. out_off[B]
    const uint32_t k0 = a.out_off[0] + t * (uint32_t)PAIR_J;
    Fe<F> run;
    fe_one(run);
    if (k0 < total) {
        const uint32_t kend = min(k0 + (uint32_t)PAIR_J, total);
        uint32_t b = bucket_of(a.out_off, a.B, k0);
        for (uint32_t k = k0; k < kend; ++k) {
            while (a.out_off[b + 1] <= k) ++b;
            Fe<F> den;
            pair_den<F>(a, k, b, den);
            fe_mul(run, run, den);
            if (k + 1 < kend) fe_store_wm(pre + (size_t)(k - k0) * F::N * T, T, t, run);
        }
    }
    fe_store_wm(tot, T, t, run);  // one for threads without slots
}

template <class C, bool DST_OFF>
__global__ void __launch_bounds__(256, 2) k_pair_bwd(PairArgs a, uint32_t T, const uint32_t* __restrict__ pre,
                                                     const uint32_t* __restrict__ inv_tot) {
    using F = typename C::F;
    constexpr int N = F::N;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const uint32_t total = a.out_off[a.B];
    const uint32_t k0 = a.out_off[0] + t * (uint32_t)PAIR_J;
    if (k0 >= total) return;
    const uint32_t kend = min(k0 + (uint32_t)PAIR_J, total);
    Fe<F> inv_run;
    fe_load_wm(inv_run, inv_tot, T, t);
    uint32_t bend = bucket_of(a.out_off, a.B, kend - 1);
    for (int j = (int)(kend - k0) - 1; j >= 0; --j) {
        const uint32_t k = k0 + (uint32_t)j;
        while (a.out_off[bend] > k) --bend;
        Affine<F> P0, P1;
        bool inf0;
        Fe<F> den, inv;
        const int kind = pair_setup<F>(a, k, bend, P0, P1, inf0, den);
        if (j > 0) {
            fe_load_wm(inv, pre + (size_t)(j - 1) * N * T, T, t);
            // two independent products, inlined so their instruction streams
            // interleave (pair stage at 2^22: 22.65 -> 21.64 ms; inlining the
            // sum's three dependent products as well was slower, 22.47 ms)
            fe_mul_inl(inv, inv, inv_run);
            fe_mul_inl(inv_run, inv_run, den);
        } else {
            inv = inv_run;
        }
        uint32_t row = k;
        if constexpr (DST_OFF) row = a.dst_off[bend] + (k - a.out_off[bend]);
        uint32_t* dst = a.dst + (size_t)row * 2 * N;
        if (kind == PAIR_ADD || kind == PAIR_DBL) {
            Fe<F> lam, x3;
            if (kind == PAIR_ADD) {
                fe_sub(lam, P1.y, P0.y);
            } else {
                fe_sqr(lam, P0.x);
                fe_dbl(x3, lam);
                fe_add(lam, lam, x3);  // 3 x0^2
                P1.x = P0.x;
            }
            fe_mul(lam, lam, inv);
            fe_sqr(x3, lam);
            fe_sub(x3, x3, P0.x);
            fe_sub(x3, x3, P1.x);
            fe_sub(P1.y, P0.x, x3);
            fe_mul(P1.y, lam, P1.y);
            fe_sub(P1.y, P1.y, P0.y);
            pair_store<F>(dst, x3, P1.y);
        } else if (kind == PAIR_INF || (kind == PAIR_PASS0 && inf0)) {
            Fe<F> z;
            fe_zero(z);
            P0.x = z;
            P0.x.v[N - 1] = INF_FLAG;
            pair_store<F>(dst, P0.x, z);
        } else {
            const Affine<F>& R = kind == PAIR_PASS0 ? P0 : P1;
            pair_store<F>(dst, R.x, R.y);
        }
    }
}

// Inclusive prefix P and suffix S products of the warp's values.
template <class F>
__device__ __forceinline__ void warp_prefix_suffix(Fe<F>& P, Fe<F>& S, int lane) {
    Fe<F> o;
    for (int d = 1; d < 32; d <<= 1) {  // inclusive prefix P and suffix S over the warp
#pragma unroll
        for (int q = 0; q < F::N; ++q) o.v[q] = __shfl_up_sync(0xffffffffu, P.v[q], d);
        if (lane >= d) fe_mul(P, P, o);
#pragma unroll
        for (int q = 0; q < F::N; ++q) o.v[q] = __shfl_down_sync(0xffffffffu, S.v[q], d);
        if (lane + d < 32) fe_mul(S, S, o);
    }
}

// r *= P_{lane-1} * S_{lane+1}: the product of the warp's other lanes' values.
template <class F>
__device__ __forceinline__ void warp_exclude_self(Fe<F>& r, const Fe<F>& P, const Fe<F>& S, int lane) {
    Fe<F> o;
#pragma unroll
    for (int q = 0; q < F::N; ++q) o.v[q] = __shfl_up_sync(0xffffffffu, P.v[q], 1);
    if (lane > 0) fe_mul(r, r, o);
#pragma unroll
    for (int q = 0; q < F::N; ++q) o.v[q] = __shfl_down_sync(0xffffffffu, S.v[q], 1);
    if (lane < 31) fe_mul(r, r, o);
}

// The M elements of v (word-major, stride M) replaced by their inverses.
// Block b owns elements [b G INV_T, (b + 1) G INV_T); its thread t chains
// elements base + j INV_T (j < G, base = b G INV_T + t; running products in
// pre, word-major with stride TT = gridDim.x INV_T), the thread products
// combine by warp-shuffle prefix and suffix products, warp 0 repeats that over
// the warp products and inverts the block's product, so every
// thread recovers the inverse of its own product and walks its chain back.
// Elements are non-zero: every denominator is a difference of distinct x, or
// 2y with y non-zero, or one.
template <class F>
__global__ void __launch_bounds__(INV_T, 2) k_inv_wide(uint32_t* __restrict__ v, uint32_t M, uint32_t G,
                                                       uint32_t* __restrict__ pre) {
    constexpr int N = F::N;
    constexpr int NW = INV_T / 32;
    __shared__ uint32_t s_wt[NW * N];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const size_t TT = (size_t)gridDim.x * INV_T;
    const size_t gt = (size_t)blockIdx.x * INV_T + (size_t)t;
    const size_t base = (size_t)blockIdx.x * INV_T * G + (size_t)t;
    Fe<F> run, x;
    fe_one(run);
    uint32_t cnt = 0;
    for (size_t e = base; cnt < G && e < M; ++cnt, e += INV_T) {
        if (cnt) fe_store_wm(pre + (size_t)(cnt - 1) * N * TT, TT, gt, run);
        fe_load_wm(x, v, M, e);
        fe_mul(run, run, x);
    }
    Fe<F> P = run, S = run;
    warp_prefix_suffix(P, S, lane);
    if (lane == 31) fe_store(s_wt + warp * N, P);
    __syncthreads();
    if (warp == 0) {
        Fe<F> w, P2, S2, inv;
        if (lane < NW)
            fe_load(w, s_wt + lane * N);
        else
            fe_one(w);
        P2 = w;
        S2 = w;
        warp_prefix_suffix(P2, S2, lane);
        Fe<F> tot;
#pragma unroll
        for (int q = 0; q < N; ++q) tot.v[q] = __shfl_sync(0xffffffffu, P2.v[q], 31);
        fe_inv_quad(inv, tot);  // every quad of the warp inverts the same product
        warp_exclude_self(inv, P2, S2, lane);  // 1 / (warp lane's product)
        __syncwarp();
        if (lane < NW) fe_store(s_wt + lane * N, inv);
    }
    __syncthreads();
    Fe<F> r;
    fe_load(r, s_wt + warp * N);
    warp_exclude_self(r, P, S, lane);  // 1 / run
    for (int j = (int)cnt - 1; j > 0; --j) {
        const size_t e = base + (size_t)j * INV_T;
        Fe<F> p;
        fe_load_wm(x, v, M, e);
        fe_load_wm(p, pre + (size_t)(j - 1) * N * TT, TT, gt);
        fe_mul(p, p, r);  // 1 / x_j
        fe_mul(r, r, x);
        fe_store_wm(v, M, e, p);
    }
    if (cnt) fe_store_wm(v, M, base, r);
}

// Sum of each item's (already weighted) windows, then affine + wire
// (+ compressed for BLS12-381).  One block per item: quad q sums windows q,
// q + COMBINE_QUADS, ..., a tree over the quads follows, and warp 0 converts:
// one inversion by every quad (fe_inv_quad), x on the even lanes, y on the
// odd ones.  Bound by latency: 17 windows are five quad additions deep, then
// the inversion.  One item of 17 BLS12-381 windows 0.115 -> 0.083 ms, of one
// window 0.080 -> 0.057 ms, against one warp per item and one-lane conversion.
constexpr int COMBINE_THREADS = 128, COMBINE_QUADS = COMBINE_THREADS / 4;

template <class C>
__global__ void __launch_bounds__(COMBINE_THREADS)
    k_combine(const ItemDesc* __restrict__ items, const uint32_t* __restrict__ wins,
              uint8_t* __restrict__ out_wire, uint8_t* __restrict__ out_comp) {
    using F = typename C::F;
    constexpr int N = F::N, PW = 4 * N, PS = RED_PS<F>;
    __shared__ __align__(16) uint32_t s[COMBINE_QUADS * PS];
    const ItemDesc it = items[blockIdx.x];
    const uint32_t quad = threadIdx.x >> 2;
    const uint32_t W = it.n != 0 ? it.Wr : 0u;  // windows arrive weighted by 2^(c w)
    {
        uint32_t* mine = s + (size_t)quad * PS;
        const uint32_t* src = wins + (size_t)it.win_base * PW;
        if (quad < W) {
            quad_copy<F>(mine, src + (size_t)quad * PW);
            __syncwarp(0xFu << (threadIdx.x & 28));
            for (uint32_t w = quad + COMBINE_QUADS; w < W; w += COMBINE_QUADS)
                xyzz_add_quad_pt<F>(mine, src + (size_t)w * PW);
        } else {
            quad_set_inf<F>(mine);
        }
        __syncthreads();
        for (uint32_t d = COMBINE_QUADS / 2; d >= 1; d >>= 1) {
            if (quad < d && quad + d < W) xyzz_add_quad_pt<F>(mine, mine + (size_t)d * PS);
            __syncthreads();
        }
    }
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    const bool odd = (lane & 1) != 0;
    uint8_t* ow = out_wire + (size_t)it.out_index * C::WIRE;
    uint8_t* oc = out_comp && C::CURVE_ID == 2 ? out_comp + (size_t)it.out_index * 48 : nullptr;
    Fe<F> zz, zzz, t, v;
    fe_load16(zz, s + 2 * N);
    fe_load16(zzz, s + 3 * N);
    const bool fin = !fe_is_zero(zz);
    fe_mul(t, zz, zzz);
    fe_inv_quad(t, t);                      // 1 / (ZZ ZZZ)
    fe_sel(v, odd, zz, zzz);
    fe_mul(t, t, v);                        // 1 / ZZ (even), 1 / ZZZ (odd)
    fe_load16(v, s + (odd ? N : 0));
    fe_mul(v, v, t);                        // x (even), y (odd)
    fe_from_mont(v, v);                     // zero for infinity
    if (lane < 2) fe_to_be_bytes(ow + lane * F::BYTES, v);
    if (!oc) return;
    // ZCash/IETF compressed form: bit7 compressed, bit6 infinity, bit5 iff
    // y > (p-1)/2, i.e. 2y > p.
    uint32_t y2[N], cy = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        y2[k] = (v.v[k] << 1) | cy;
        cy = v.v[k] >> 31;
    }
    // 2y > p  <=>  p - 2y borrows (2y != p since p is odd)
    int64_t bw = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const int64_t d = (int64_t)F::P(k) - (int64_t)y2[k] - bw;
        bw = d < 0 ? 1 : 0;
    }
    const uint32_t sign = __shfl_sync(0xffffffffu, (uint32_t)bw, 1);
    if (lane == 0) {
        fe_to_be_bytes(oc, v);
        oc[0] |= fin ? (sign ? 0xA0 : 0x80) : 0xC0;
    }
}

template <class C>
struct MsmLaunchImpl {
    using F = typename C::F;
    static void wire_to_table(const uint8_t* w, uint32_t* t, size_t n, size_t glv_stride,
                              cudaStream_t st) {
        if (!n) return;
        if (((uintptr_t)w & 15) == 0)
            k_wire_to_table<C, true><<<ceil_div_u(n, 128), 128, 0, st>>>(w, t, n, glv_stride);
        else
            k_wire_to_table<C, false><<<ceil_div_u(n, 128), 128, 0, st>>>(w, t, n, glv_stride);
        KB_LAUNCH_CHECK();
    }
    static void table_to_wire(const uint32_t* t, uint8_t* w, size_t n, cudaStream_t st) {
        if (!n) return;
        k_table_to_wire<C><<<ceil_div_u(n, 128), 128, 0, st>>>(t, w, n);
        KB_LAUNCH_CHECK();
    }
    static void recode(const ItemDesc* items, uint32_t n_items, unsigned long long first,
                       unsigned long long count, const uint32_t* scalars, const uint32_t* table,
                       uint32_t* keys, uint32_t* vals, cudaStream_t st) {
        if (!count) return;
        k_recode<C><<<ceil_div_u(count, 256), 256, 0, st>>>(items, n_items, first, count, scalars,
                                                           table, keys, vals);
        KB_LAUNCH_CHECK();
    }
    // One pairing level over T0 = ceil(slots / PAIR_J) threads; scratch holds
    // pair_scratch_words(T0, N) words.
    static void pair_level(const PairArgs& a, uint32_t T0, uint32_t* scratch, cudaStream_t st) {
        if (!T0) return;
        constexpr int N = F::N;
        uint32_t* pre0 = scratch;
        uint32_t* tot = pre0 + (size_t)(PAIR_J - 1) * N * T0;
        k_pair_fwd<C><<<ceil_div_u(T0, 256), 256, 0, st>>>(a, T0, pre0, tot);
        KB_LAUNCH_CHECK();
        const InvGeom g = inv_geom(T0);
        k_inv_wide<F><<<g.nb, INV_T, 0, st>>>(tot, T0, g.G, tot + (size_t)N * T0);
        KB_LAUNCH_CHECK();
        if (a.dst_off)
            k_pair_bwd<C, true><<<ceil_div_u(T0, 256), 256, 0, st>>>(a, T0, pre0, tot);
        else
            k_pair_bwd<C, false><<<ceil_div_u(T0, 256), 256, 0, st>>>(a, T0, pre0, tot);
        KB_LAUNCH_CHECK();
    }
    static void accumulate(const AccArgs& a, unsigned grid, cudaStream_t st) {
        k_accumulate<C><<<grid, 128, 0, st>>>(a);
        KB_LAUNCH_CHECK();
    }
    static void fold(const FoldArgs& a, int level, const uint32_t* in, uint32_t* out,
                     unsigned grid, cudaStream_t st) {
        k_fold<C><<<grid, FOLD_THREADS, 0, st>>>(a, level, in, out);
        KB_LAUNCH_CHECK();
    }
    static void reduce(const RedArgs& a, unsigned nblk, cudaStream_t st) {
        if (!nblk) return;
        constexpr size_t smem = (size_t)(RED_TREE + RED_FINAL) * RED_PS<F> * 4;
        set_smem_attr((const void*)k_reduce<C>, smem);
        k_reduce<C><<<nblk, RED_THREADS, smem, st>>>(a);
        KB_LAUNCH_CHECK();
    }
    static void combine(const ItemDesc* items, uint32_t n_items, const uint32_t* wins,
                        uint8_t* ow, uint8_t* oc, cudaStream_t st) {
        if (!n_items) return;
        k_combine<C><<<n_items, COMBINE_THREADS, 0, st>>>(items, wins, ow, oc);
        KB_LAUNCH_CHECK();
    }
    static int accumulate_occupancy() {
        int blocks = 0;
        KB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_accumulate<C>, 128, 0));
        return blocks;
    }
    static MsmLaunchers table() {
        MsmLaunchers L;
        L.wire_to_table = &wire_to_table;
        L.table_to_wire = &table_to_wire;
        L.recode = &recode;
        L.accumulate = &accumulate;
        L.pair_level = &pair_level;
        L.fold = &fold;
        L.reduce = &reduce;
        L.combine = &combine;
        L.accumulate_occupancy = &accumulate_occupancy;
        L.point_words = 4 * F::N;
        L.table_words = 2 * F::N;
        L.wire_bytes = C::WIRE;
        return L;
    }
};

}  // namespace kb200
