// Montgomery field arithmetic on 32-bit limbs for sm_100a.
//
// Four prime fields, all with R = 2^(32N) (the same Montgomery domain as the
// reference's 64-bit-limb code, so Montgomery images are bit-identical):
//   FpBLS : BLS12-381 base field, N = 12   (bls/cpp/bls12_381_fp.hpp:83-98)
//   FrBLS : BLS12-381 scalar field, N = 8  (kzg/cpp/kzg_oracle.hpp:66-90)
//   FpBN  : BN254 base field, N = 8        (bn254/cpp/bn254_fp.hpp:75-89)
//   FrBN  : BN254 scalar field, N = 8      (bn254/cpp/bn254_fp.hpp:79-97)
//
// Multiplication (fe_mul_inl): the interleaved Montgomery product over two
// accumulators, one for even and one for odd word offsets, so that every
// partial product lands on an aligned word pair; carry chains are written as
// consecutive mad.lo.cc / madc.hi.cc instructions.  Every value is kept fully
// reduced in [0, p); all four moduli satisfy 2p < 2^(32N).
#pragma once
#include <cstdint>

#define KB_DEV __device__ __forceinline__
#define KB_HD __host__ __device__ __forceinline__

namespace kb200 {

// ---------------------------------------------------------------------------
// PTX carry-chain primitives.  volatile keeps the compiler from moving them
// relative to one another, so a chain written as consecutive calls stays a
// chain on the condition-code register.
// ---------------------------------------------------------------------------
KB_DEV uint32_t mad_lo_cc(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm volatile("mad.lo.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
KB_DEV uint32_t madc_lo_cc(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm volatile("madc.lo.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
KB_DEV uint32_t madc_hi_cc(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm volatile("madc.hi.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
KB_DEV uint32_t addc_u32(uint32_t a, uint32_t b) {
    uint32_t r;
    asm volatile("addc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
KB_DEV uint32_t add_cc(uint32_t a, uint32_t b) {
    uint32_t r;
    asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
KB_DEV uint32_t addc_cc(uint32_t a, uint32_t b) {
    uint32_t r;
    asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
KB_DEV uint32_t sub_cc(uint32_t a, uint32_t b) {
    uint32_t r;
    asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
KB_DEV uint32_t subc_cc(uint32_t a, uint32_t b) {
    uint32_t r;
    asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
KB_DEV uint32_t subc_u32(uint32_t a, uint32_t b) {
    uint32_t r;
    asm volatile("subc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// ---------------------------------------------------------------------------
// Field parameters.  Limbs are little-endian 32-bit words.
// ---------------------------------------------------------------------------
struct FpBLS {
    static constexpr int N = 12;
    static constexpr int BYTES = 48;
    static constexpr uint32_t M0 = 0xfffcfffdu;  // -p^-1 mod 2^32
    KB_HD static constexpr uint32_t P(int i) {
        constexpr uint32_t t[12] = {0xffffaaab, 0xb9feffff, 0xb153ffff, 0x1eabfffe,
                                    0xf6b0f624, 0x6730d2a0, 0xf38512bf, 0x64774b84,
                                    0x434bacd7, 0x4b1ba7b6, 0x397fe69a, 0x1a0111ea};
        return t[i];
    }
    KB_HD static constexpr uint32_t R1(int i) {
        constexpr uint32_t t[12] = {0x0002fffd, 0x76090000, 0xc40c0002, 0xebf4000b,
                                    0x53c758ba, 0x5f489857, 0x70525745, 0x77ce5853,
                                    0xa256ec6d, 0x5c071a97, 0xfa80e493, 0x15f65ec3};
        return t[i];
    }
    KB_HD static constexpr uint32_t R2(int i) {
        constexpr uint32_t t[12] = {0x1c341746, 0xf4df1f34, 0x09d104f1, 0x0a76e6a6,
                                    0x4c95b6d5, 0x8de5476c, 0x939d83c0, 0x67eb88a9,
                                    0xb519952d, 0x9a793e85, 0x92cae3aa, 0x11988fe5};
        return t[i];
    }
};

struct FrBLS {
    static constexpr int N = 8;
    static constexpr int BYTES = 32;
    static constexpr uint32_t M0 = 0xffffffffu;
    KB_HD static constexpr uint32_t P(int i) {
        constexpr uint32_t t[8] = {0x00000001, 0xffffffff, 0xfffe5bfe, 0x53bda402,
                                   0x09a1d805, 0x3339d808, 0x299d7d48, 0x73eda753};
        return t[i];
    }
    KB_HD static constexpr uint32_t R1(int i) {
        constexpr uint32_t t[8] = {0xfffffffe, 0x00000001, 0x00034802, 0x5884b7fa,
                                   0xecbc4ff5, 0x998c4fef, 0xacc5056f, 0x1824b159};
        return t[i];
    }
    KB_HD static constexpr uint32_t R2(int i) {
        constexpr uint32_t t[8] = {0xf3f29c6d, 0xc999e990, 0x87925c23, 0x2b6cedcb,
                                   0x7254398f, 0x05d31496, 0x9f59ff11, 0x0748d9d9};
        return t[i];
    }
};

struct FpBN {
    static constexpr int N = 8;
    static constexpr int BYTES = 32;
    static constexpr uint32_t M0 = 0xe4866389u;
    KB_HD static constexpr uint32_t P(int i) {
        constexpr uint32_t t[8] = {0xd87cfd47, 0x3c208c16, 0x6871ca8d, 0x97816a91,
                                   0x8181585d, 0xb85045b6, 0xe131a029, 0x30644e72};
        return t[i];
    }
    KB_HD static constexpr uint32_t R1(int i) {
        constexpr uint32_t t[8] = {0xc58f0d9d, 0xd35d438d, 0xf5c70b3d, 0x0a78eb28,
                                   0x7879462c, 0x666ea36f, 0x9a07df2f, 0x0e0a77c1};
        return t[i];
    }
    KB_HD static constexpr uint32_t R2(int i) {
        constexpr uint32_t t[8] = {0x538afa89, 0xf32cfc5b, 0xd44501fb, 0xb5e71911,
                                   0x0a417ff6, 0x47ab1eff, 0xcab8351f, 0x06d89f71};
        return t[i];
    }
};

struct FrBN {
    static constexpr int N = 8;
    static constexpr int BYTES = 32;
    static constexpr uint32_t M0 = 0xefffffffu;
    KB_HD static constexpr uint32_t P(int i) {
        constexpr uint32_t t[8] = {0xf0000001, 0x43e1f593, 0x79b97091, 0x2833e848,
                                   0x8181585d, 0xb85045b6, 0xe131a029, 0x30644e72};
        return t[i];
    }
    KB_HD static constexpr uint32_t R1(int i) {
        constexpr uint32_t t[8] = {0x4ffffffb, 0xac96341c, 0x9f60cd29, 0x36fc7695,
                                   0x7879462e, 0x666ea36f, 0x9a07df2f, 0x0e0a77c1};
        return t[i];
    }
    KB_HD static constexpr uint32_t R2(int i) {
        constexpr uint32_t t[8] = {0xae216da7, 0x1bb8e645, 0xe35c59e3, 0x53fe3ab1,
                                   0x53bb8085, 0x8c49833d, 0x7f4e44a5, 0x0216d0b1};
        return t[i];
    }
};

// ---------------------------------------------------------------------------
// Element type and arithmetic.
// ---------------------------------------------------------------------------
template <class F>
struct Fe {
    uint32_t v[F::N];
};

template <class F>
KB_DEV void fe_zero(Fe<F>& a) {
#pragma unroll
    for (int i = 0; i < F::N; ++i) a.v[i] = 0;
}
template <class F>
KB_DEV void fe_one(Fe<F>& a) {  // 1 in Montgomery form (R mod p)
#pragma unroll
    for (int i = 0; i < F::N; ++i) a.v[i] = F::R1(i);
}
template <class F>
KB_DEV bool fe_is_zero(const Fe<F>& a) {
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < F::N; ++i) acc |= a.v[i];
    return acc == 0;
}
template <class F>
KB_DEV bool fe_eq(const Fe<F>& a, const Fe<F>& b) {
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < F::N; ++i) acc |= a.v[i] ^ b.v[i];
    return acc == 0;
}

// r = t - p if t >= p else t (t < 2p, N words).
template <class F>
KB_DEV void reduce_once(Fe<F>& r, const uint32_t* t) {
    constexpr int N = F::N;
    uint32_t d[N];
    d[0] = sub_cc(t[0], F::P(0));
#pragma unroll
    for (int i = 1; i < N; ++i) d[i] = subc_cc(t[i], F::P(i));
    uint32_t borrow = subc_u32(0, 0);  // 0xffffffff if t < p
#pragma unroll
    for (int i = 0; i < N; ++i) r.v[i] = borrow ? t[i] : d[i];
}

// d[0..N) = c[0..N) + x[0], x[2], x[4], ... times b: the N/2 products as one
// carry chain over the aligned word pairs (0, 1), (2, 3), ..., each pair one
// 32 x 32 + 64 multiply-add.  The first pair takes the chain's carry in; the
// last pair's carry is left for an addc.
template <int N>
KB_DEV void mac_pairs_cin(uint32_t* d, const uint32_t* x, uint32_t b, const uint32_t* c) {
#pragma unroll
    for (int j = 0; j < N; j += 2) {
        d[j] = madc_lo_cc(x[j], b, c[j]);
        d[j + 1] = madc_hi_cc(x[j], b, c[j + 1]);
    }
}
// The same without a carry in.
template <int N>
KB_DEV void mac_pairs(uint32_t* d, const uint32_t* x, uint32_t b, const uint32_t* c) {
    d[0] = mad_lo_cc(x[0], b, c[0]);
    d[1] = madc_hi_cc(x[0], b, c[1]);
    mac_pairs_cin<N - 2>(d + 2, x + 2, b, c + 2);
}

// The reduction row of fe_mul_inl: E += m p_even, O += m p_odd with
// m = E[0] (-p^-1 mod 2^32), so E[0] becomes zero.
//
// A modulus with low words 1 and 2^32 - 1 (the BLS12-381 scalar field r)
// needs no multiply for them: m = -E[0] (as -p^-1 = 2^32 - 1), m * 1 makes
// E[0] zero with a carry iff it was not, and m (2^32 - 1) = (E[0], E[0] ?
// ~E[0] : 0) as (low, high) words: two of a row's eight pair multiply-adds
// and the multiply for m become additions.
template <class F>
KB_DEV void mont_row(uint32_t* E, uint32_t* O, const uint32_t* p) {
    constexpr int N = F::N;
    constexpr bool LOW_ONE = F::P(0) == 1u && F::P(1) == 0xffffffffu;
    if constexpr (LOW_ONE) {
        const uint32_t t = E[0], m = 0u - t, hi = t ? ~t : 0u;
        O[0] = add_cc(O[0], t);
        O[1] = addc_cc(O[1], hi);
        mac_pairs_cin<N - 2>(O + 2, p + 3, m, O + 2);
        E[0] = add_cc(t, m);
        E[1] = addc_cc(E[1], 0u);
        mac_pairs_cin<N - 2>(E + 2, p + 2, m, E + 2);
    } else {
        const uint32_t m = E[0] * F::M0;
        mac_pairs<N>(O, p + 1, m, O);
        mac_pairs<N>(E, p, m, E);
    }
    O[N - 1] = addc_u32(O[N - 1], 0);
}

// r = a * b * R^-1 mod p, R = 2^(32N); a in [0, p), b any N-word value, r in [0, p).
// Larger a up to R (1 - 2^-30) - p give r < max(p, a b / R), the same residue.
//
// Interleaved (CIOS) Montgomery product (Koc, Acar and Kaliski, "Analyzing and
// Comparing Montgomery Multiplication Algorithms", IEEE Micro 16(3), 1996) over two
// accumulators, by the parity of the word offset (the separately aligned sums of
// Emmart, Luitjens, Weems and Woolley, "Optimizing Modular Multiplication for
// NVIDIA's Maxwell GPUs", ARITH 2016): E holds words
// 0 .. N-1 and O words 1 .. N of the running sum E + 2^32 O, so the products
// of a's (and p's) even words always land on E's aligned word pairs and the
// odd ones on O's.  A word pair is one multiply-add with a 64-bit addend and
// a carry chain links the pairs, so a row of a (or p) costs N multiply-adds
// and one addc, and no word ever moves between pair alignments.  Dividing by
// 2^32 after a row swaps the roles: O becomes the new E, and E >> 64 the new
// O once E[1] has been added to the new E[0], whose carry enters the new O's
// chain.  The sum stays below (a + p) 2^32 (1 + 2^-31) < 2^(32 (N + 1)) for
// such a, whatever b is, and (a b + m p) / R < 2p for a < p: one conditional
// subtraction.
//
// What bounds it: the multiply pipe takes a 32 x 32 + 64 multiply-add in four
// cycles per warp and sub-partition, 2N^2 of them (288 for N = 12).  A single
// accumulator needs moves to realign the pairs at every row: measured on a
// B200 at 16 warps an SM (BLS12-381 Fp), 652 instructions and 1349 cycles per
// warp product with one accumulator and one Karatsuba level (252 pair
// multiply-adds), 378 instructions and 1230 cycles in this form (the pipe 97 %
// busy), i.e. 27.6 -> 30.3 G products/s; BN254 Fp 57.2 -> 65.2 G/s.
// One Karatsuba level over two accumulators (252 pair multiply-adds, 501
// instructions) ran at 1246 cycles.  Reducing the double-width product by
// double-precision multiply-adds over 24-bit limbs was exact but no gain where it
// counts: 1193 against 1232 cycles at 16 warps an SM (31.2 against 30.2 G/s; the two
// pipes share issue and register bandwidth), and though a lone warp took 1534
// instead of 1886 cycles, the kernels built on it were slower (reduction of a 2^22
// MSM 1.52 -> 1.87 ms).
template <class F>
KB_DEV void fe_mul_inl(Fe<F>& r, const Fe<F>& a, const Fe<F>& b) {
    constexpr int N = F::N;
    static_assert(N % 2 == 0, "word pairs");
    uint32_t E[N], O[N], p[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        p[j] = F::P(j);
        E[j] = O[j] = 0;
    }
    mac_pairs<N>(E, a.v, b.v[0], E);
    mac_pairs<N>(O, a.v + 1, b.v[0], O);
    mont_row<F>(E, O, p);
#pragma unroll
    for (int i = 1; i < N; ++i) {
        uint32_t X[N + 2];  // the old E, shifted into the new O
#pragma unroll
        for (int j = 0; j < N; ++j) {
            X[j] = E[j];
            E[j] = O[j];
        }
        X[N] = X[N + 1] = 0;
        E[0] = add_cc(E[0], X[1]);
        mac_pairs_cin<N>(O, a.v + 1, b.v[i], X + 2);
        mac_pairs<N>(E, a.v, b.v[i], E);
        O[N - 1] = addc_u32(O[N - 1], 0);
        mont_row<F>(E, O, p);
    }
    uint32_t U[N];
    U[0] = add_cc(O[0], E[1]);
#pragma unroll
    for (int j = 1; j < N - 1; ++j) U[j] = addc_cc(O[j], E[j + 1]);
    U[N - 1] = addc_u32(O[N - 1], 0);
    reduce_once<F>(r, U);
}

// r = a^2 R^-1 mod p, a in [0, p).  The off-diagonal products a_i a_j (i < j)
// once, in fe_mul_inl's two accumulators (words of even and of odd i + j), then
// doubled, the diagonal added, and the low half reduced row by row as there:
// N (N + 1) / 2 + N^2 pair multiply-adds instead of 2 N^2 (222 against 288 for
// N = 12).
template <class F>
KB_DEV void fe_sqr_inl(Fe<F>& r, const Fe<F>& a) {
    constexpr int N = F::N;
    uint32_t T[2 * N];
    {
        uint32_t E[2 * N], O[2 * N];
#pragma unroll
        for (int j = 0; j < 2 * N; ++j) E[j] = O[j] = 0;
#pragma unroll
        for (int i = 0; i < N - 1; ++i) {
            // a_i times a_(i+1), a_(i+3), ...: words 2i + 1, 2i + 3, ... (O, one
            // word up); times a_(i+2), a_(i+4), ...: words 2i + 2, ... (E)
            int k = 2 * i;
#pragma unroll
            for (int j = i + 1; j < N; j += 2, k += 2) {
                O[k] = j == i + 1 ? mad_lo_cc(a.v[j], a.v[i], O[k]) : madc_lo_cc(a.v[j], a.v[i], O[k]);
                O[k + 1] = madc_hi_cc(a.v[j], a.v[i], O[k + 1]);
            }
            if (i > 0 && k < 2 * N) O[k] = addc_u32(O[k], 0);
            k = 2 * i + 2;
#pragma unroll
            for (int j = i + 2; j < N; j += 2, k += 2) {
                E[k] = j == i + 2 ? mad_lo_cc(a.v[j], a.v[i], E[k]) : madc_lo_cc(a.v[j], a.v[i], E[k]);
                E[k + 1] = madc_hi_cc(a.v[j], a.v[i], E[k + 1]);
            }
            if (i > 0 && i + 2 < N && k < 2 * N) E[k] = addc_u32(E[k], 0);
        }
        // T = 2 (E + 2^32 O); words 0 and 1 of E are empty
        T[0] = 0;
        T[1] = O[0];
        T[2] = add_cc(E[2], O[1]);
#pragma unroll
        for (int k = 3; k < 2 * N - 1; ++k) T[k] = addc_cc(E[k], O[k - 1]);
        T[2 * N - 1] = addc_u32(E[2 * N - 1], O[2 * N - 2]);
    }
#pragma unroll
    for (int k = 2 * N - 1; k > 0; --k) T[k] = __funnelshift_l(T[k - 1], T[k], 1);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        T[2 * i] = i ? madc_lo_cc(a.v[i], a.v[i], T[2 * i]) : mad_lo_cc(a.v[0], a.v[0], T[0]);
        T[2 * i + 1] = madc_hi_cc(a.v[i], a.v[i], T[2 * i + 1]);
    }
    // Montgomery reduction of the low half: the rows of fe_mul_inl alone
    uint32_t E[N], O[N], p[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        p[j] = F::P(j);
        E[j] = T[j];
        O[j] = 0;
    }
    mont_row<F>(E, O, p);
#pragma unroll
    for (int i = 1; i < N; ++i) {
        uint32_t X[N + 2];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            X[j] = E[j];
            E[j] = O[j];
        }
        X[N] = X[N + 1] = 0;
        // the shifted old E joins the new O; its word 1 joins E[0], whose
        // carry enters the row's chain on O
        const uint32_t m = (E[0] + X[1]) * F::M0;
        E[0] = add_cc(E[0], X[1]);
        mac_pairs_cin<N>(O, p + 1, m, X + 2);
        mac_pairs<N>(E, p, m, E);
        O[N - 1] = addc_u32(O[N - 1], 0);
    }
    uint32_t U[N];
    U[0] = add_cc(O[0], E[1]);
#pragma unroll
    for (int j = 1; j < N - 1; ++j) U[j] = addc_cc(O[j], E[j + 1]);
    U[N - 1] = addc_u32(O[N - 1], 0);
    U[0] = add_cc(U[0], T[N]);
#pragma unroll
    for (int j = 1; j < N - 1; ++j) U[j] = addc_cc(U[j], T[N + j]);
    U[N - 1] = addc_u32(U[N - 1], T[2 * N - 1]);
    reduce_once<F>(r, U);
}

// Out-of-line copy: one instance of the product per kernel instead of one
// per call site, which keeps large kernels (bucket reduction, window combine)
// inside the instruction cache.
template <class F>
__device__ __noinline__ Fe<F> fe_mul_call(Fe<F> a, Fe<F> b) {
    Fe<F> r;
    fe_mul_inl<F>(r, a, b);
    return r;
}

template <class F>
KB_DEV void fe_mul(Fe<F>& r, const Fe<F>& a, const Fe<F>& b) {
    r = fe_mul_call<F>(a, b);
}

template <class F>
__device__ __noinline__ Fe<F> fe_sqr_call(Fe<F> a) {
    Fe<F> r;
    fe_sqr_inl<F>(r, a);
    return r;
}
template <class F>
KB_DEV void fe_sqr(Fe<F>& r, const Fe<F>& a) {
    r = fe_sqr_call<F>(a);
}

template <class F>
KB_DEV void fe_add(Fe<F>& r, const Fe<F>& a, const Fe<F>& b) {
    constexpr int N = F::N;
    uint32_t s[N];
    s[0] = add_cc(a.v[0], b.v[0]);
#pragma unroll
    for (int i = 1; i < N; ++i) s[i] = addc_cc(a.v[i], b.v[i]);
    reduce_once<F>(r, s);
}

template <class F>
KB_DEV void fe_sub(Fe<F>& r, const Fe<F>& a, const Fe<F>& b) {
    constexpr int N = F::N;
    uint32_t d[N];
    d[0] = sub_cc(a.v[0], b.v[0]);
#pragma unroll
    for (int i = 1; i < N; ++i) d[i] = subc_cc(a.v[i], b.v[i]);
    uint32_t mask = subc_u32(0, 0);
    r.v[0] = add_cc(d[0], F::P(0) & mask);
#pragma unroll
    for (int i = 1; i < N; ++i) r.v[i] = addc_cc(d[i], F::P(i) & mask);
}

template <class F>
KB_DEV void fe_neg(Fe<F>& r, const Fe<F>& a) {
    Fe<F> z;
    fe_zero(z);
    fe_sub<F>(r, z, a);
}

template <class F>
KB_DEV void fe_dbl(Fe<F>& r, const Fe<F>& a) {
    fe_add<F>(r, a, a);
}

// Conversions between canonical and Montgomery form.  to_mont accepts any
// N-word value (it need not be below p) as the product's second operand: R^2
// mod p < p keeps the product below 2p, so the result is the canonical image
// of (a mod p) -- the same reduction the reference's to_mont performs.
template <class F>
KB_DEV void fe_to_mont(Fe<F>& r, const Fe<F>& a) {
    Fe<F> r2;
#pragma unroll
    for (int i = 0; i < F::N; ++i) r2.v[i] = F::R2(i);
    fe_mul<F>(r, r2, a);
}
template <class F>
KB_DEV void fe_from_mont(Fe<F>& r, const Fe<F>& a) {
    Fe<F> one;
    fe_zero(one);
    one.v[0] = 1;
    fe_mul<F>(r, a, one);
}

// Exponent word i of p - 2, with the borrow propagated (BLS12-381 r has
// low word 1, so p - 2 borrows from word 1 there).
template <class F>
KB_HD constexpr uint32_t pm2_word(int i) {
    uint32_t borrow = 2;
    uint32_t w = 0;
    for (int k = 0; k <= i; ++k) {
        const uint32_t pk = F::P(k);
        w = pk - borrow;
        borrow = pk < borrow ? 1u : 0u;
    }
    return w;
}

// a^(p-2) by left-to-right square-and-multiply with 4-bit fixed windows:
// the reference the binary-GCD inversion is checked against on the device
// (kb200_field_inverse_check).
template <class F>
__device__ __noinline__ void fe_inv_fermat(Fe<F>& r, const Fe<F>& a) {
    Fe<F> tab[16];
    fe_one(tab[0]);
    tab[1] = a;
#pragma unroll 1
    for (int i = 2; i < 16; ++i) fe_mul<F>(tab[i], tab[i - 1], a);
    Fe<F> acc;
    fe_one(acc);
    bool started = false;
#pragma unroll 1
    for (int w = F::N * 8 - 1; w >= 0; --w) {
        const uint32_t word = pm2_word<F>(w >> 3);
        const uint32_t nib = (word >> ((w & 7) * 4)) & 15u;
        if (started) {
#pragma unroll 1
            for (int s = 0; s < 4; ++s) fe_sqr<F>(acc, acc);
        }
        if (nib) {
            if (started) {
                fe_mul<F>(acc, acc, tab[nib]);
            } else {
                acc = tab[nib];
                started = true;
            }
        }
    }
    r = acc;
}

// ---- Inversion by the optimized binary GCD ---------------------------------
// Pornin, "Optimized Binary GCD for Modular Inversion" (IACR ePrint 2020/972),
// Algorithm 2 with 32-bit words: each outer step runs 30 divsteps on 64-bit
// approximations of (a, b) (their low 31 bits and top 33 bits), collecting
// the 2x2 update (f0, g0; f1, g1) with |f| + |g| <= 2^30, then applies it to
// the full values: a <- (a f0 + b g0) / 2^30, b <- (a f1 + b g1) / 2^30 (exact
// divisions; a negative result is negated with its row of factors).  The
// companions u, v follow with the same factors and a Montgomery division by
// 2^30, so a = u y and b = v y (mod p) hold throughout; starting from u =
// R^2 the final v is (aR)^-1 R^2 = a^-1 R, the Montgomery form of the inverse.
// ceil((2 len(p) - 1) / 30) outer steps always end with a = 0 and b = 1 for
// y != 0; once a = 0 a step changes neither b nor v, so the loop ends there.
// The time depends on y (a public value, here as everywhere in this library).
//
// A single inversion is bound by the latency of its divsteps.  The factors are
// 32-bit words (30 steps instead of the 31 the approximations would allow keep
// them below 2^31); both differences are formed at once; all halvings up to
// the next odd a are one shift, 15.2 rounds on average (26 at most in 4000
// values) for 30 divsteps; a = 0 after 18.4 of 26 outer steps on average for
// BLS12-381 Fp, 12.4 of 17 for BN254; and fe_inv_quad gives each of a, b, u, v's
// full-width updates its own lane.  With 30 single steps in all of 26 (17)
// outer steps a KZG commit's k_combine took 55 us, now 41, and k_inv_wide on 240
// blocks 124, now 113.
namespace gcd_detail {

template <class F>
KB_HD constexpr int bit_length_p() {
    int top = F::N - 1;
    while (top > 0 && F::P(top) == 0) --top;
    uint32_t w = F::P(top);
    int b = 0;
    while (w) {
        ++b;
        w >>= 1;
    }
    return 32 * top + b;
}

// r (N + 2 words, two's complement) = x f + y g for non-negative N-word x, y
// and |f|, |g| <= 2^31.
template <int N>
KB_DEV void lin_comb(uint32_t (&r)[N + 2], const uint32_t (&x)[N], const uint32_t (&y)[N], int64_t f,
                     int64_t g) {
    const uint32_t fa = (uint32_t)(f < 0 ? -f : f), ga = (uint32_t)(g < 0 ? -g : g);
    const uint32_t mx = f < 0 ? 0xffffffffu : 0u, my = g < 0 ? 0xffffffffu : 0u;
    uint64_t cx = 0, cy = 0, c = (uint64_t)(mx & 1u) + (my & 1u);
#pragma unroll
    for (int i = 0; i <= N; ++i) {
        uint32_t px, py;
        if (i < N) {
            const uint64_t tx = (uint64_t)x[i] * fa + cx;
            const uint64_t ty = (uint64_t)y[i] * ga + cy;
            px = (uint32_t)tx;
            py = (uint32_t)ty;
            cx = tx >> 32;
            cy = ty >> 32;
        } else {
            px = (uint32_t)cx;
            py = (uint32_t)cy;
        }
        const uint64_t s = (uint64_t)(px ^ mx) + (py ^ my) + c;
        r[i] = (uint32_t)s;
        c = s >> 32;
    }
    r[N + 1] = mx + my + (uint32_t)c;
}

// r (N + 1 words, two's complement) = t / 2^30 for a two's-complement t of
// N + 2 words whose low 30 bits are zero.
template <int N>
KB_DEV void shr30(uint32_t (&r)[N + 1], const uint32_t (&t)[N + 2]) {
#pragma unroll
    for (int i = 0; i <= N; ++i) r[i] = (t[i] >> 30) | (t[i + 1] << 2);
}

// x <- -x for an (N + 1)-word two's-complement x if neg.
template <int N>
KB_DEV void negate_if(uint32_t (&x)[N + 1], bool neg) {
    const uint32_t m = neg ? 0xffffffffu : 0u;
    uint64_t c = neg ? 1u : 0u;
#pragma unroll
    for (int i = 0; i <= N; ++i) {
        const uint64_t s = (uint64_t)(x[i] ^ m) + c;
        x[i] = (uint32_t)s;
        c = s >> 32;
    }
}

// t (N + 2 words, two's complement) += q p for q < 2^30.
template <class F>
KB_DEV void add_qp(uint32_t (&t)[F::N + 2], uint32_t q) {
    constexpr int N = F::N;
    uint64_t c = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const uint64_t s = (uint64_t)F::P(i) * q + t[i] + c;
        t[i] = (uint32_t)s;
        c = s >> 32;
    }
    const uint64_t s = (uint64_t)t[N] + c;
    t[N] = (uint32_t)s;
    t[N + 1] += (uint32_t)(s >> 32);
}

// w (N + 1 words, two's complement, in (-2p, 2p)) into [0, p): add p while
// negative (at most twice), subtract p once if >= p.
template <class F>
KB_DEV void into_range(uint32_t (&w)[F::N + 1]) {
    constexpr int N = F::N;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t m = (w[N] >> 31) ? 0xffffffffu : 0u;
        uint64_t cc = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint64_t s = (uint64_t)w[i] + (F::P(i) & m) + cc;
            w[i] = (uint32_t)s;
            cc = s >> 32;
        }
        w[N] += (uint32_t)cc;
    }
    uint32_t d[N];
    int64_t br = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int64_t s = (int64_t)w[i] - F::P(i) + br;
        d[i] = (uint32_t)s;
        br = s >> 32;
    }
    const bool ge = (int64_t)w[N] + br >= 0;
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = ge ? d[i] : w[i];
}

// 30 divsteps on the approximations a, b (b odd): the rows (f0, g0) and
// (f1, g1) of the update, times 2^30.
KB_DEV void divsteps30(uint64_t a, uint64_t b, int32_t& f0, int32_t& g0, int32_t& f1, int32_t& g1) {
    f0 = 1, g0 = 0, f1 = 0, g1 = 1;
    int left = 30;
#pragma unroll 1
    while (true) {
        const int z = __ffs((int)((uint32_t)a | (1u << left))) - 1;  // at most left
        a >>= z;
        f1 = (int32_t)((uint32_t)f1 << z);
        g1 = (int32_t)((uint32_t)g1 << z);
        left -= z;
        if (left == 0) break;
        const bool sw = a < b;  // both odd
        const uint64_t d = a - b, e = b - a;
        const int32_t df = f0 - f1, dg = g0 - g1, ef = f1 - f0, eg = g1 - g0;
        b = sw ? a : b;
        f1 = sw ? f0 : f1;
        g1 = sw ? g0 : g1;
        a = sw ? e : d;
        f0 = sw ? ef : df;
        g0 = sw ? eg : dg;
    }
}

// Bits [s, s + 33) of the N-word x, for 31 <= s <= 32 N - 33.
template <int N>
KB_DEV uint64_t top33(const uint32_t (&x)[N], int s) {
    const int wi = s >> 5, sh = s & 31;
    uint32_t w0 = 0, w1 = 0, w2 = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        w0 = k == wi ? x[k] : w0;
        w1 = k == wi + 1 ? x[k] : w1;
        w2 = k == wi + 2 ? x[k] : w2;
    }
    uint64_t v = (((uint64_t)w1 << 32) | w0) >> sh;
    if (sh) v |= (uint64_t)w2 << (64 - sh);
    return v & ((1ull << 33) - 1);
}

// The approximations of a and b: their low 31 bits and the 33 bits below
// n = max(len a, len b, 64).
template <int N>
KB_DEV void approximate(const uint32_t (&a)[N], const uint32_t (&b)[N], uint64_t& ab, uint64_t& bb) {
    int n = 64;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const uint32_t w = a[k] | b[k];
        n = w ? max(n, 32 * k + 32 - __clz(w)) : n;
    }
    ab = (a[0] & 0x7fffffffu) | (top33<N>(a, n - 33) << 31);
    bb = (b[0] & 0x7fffffffu) | (top33<N>(b, n - 33) << 31);
}

template <class F>
KB_HD constexpr int outer_steps() {
    return (2 * bit_length_p<F>() - 1 + 29) / 30;
}

}  // namespace gcd_detail

template <class F>
__device__ __noinline__ void fe_inv_gcd(Fe<F>& r, const Fe<F>& y) {
    using namespace gcd_detail;
    constexpr int N = F::N;
    uint32_t a[N], b[N], u[N], v[N];
    uint32_t any = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        a[i] = y.v[i];
        b[i] = F::P(i);
        u[i] = F::R2(i);
        v[i] = 0;
        any |= y.v[i];
    }
#pragma unroll 1
    for (int it = 0; it < outer_steps<F>(); ++it) {
        uint64_t ab, bb;
        int32_t f0, g0, f1, g1;
        uint32_t nz = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) nz |= a[i];
        if (nz == 0) break;
        approximate<N>(a, b, ab, bb);
        divsteps30(ab, bb, f0, g0, f1, g1);
        uint32_t t[N + 2], na[N + 1], nb[N + 1];
        lin_comb<N>(t, a, b, f0, g0);
        shr30<N>(na, t);
        lin_comb<N>(t, a, b, f1, g1);
        shr30<N>(nb, t);
        const bool s0 = (na[N] >> 31) != 0, s1 = (nb[N] >> 31) != 0;
        negate_if<N>(na, s0);
        negate_if<N>(nb, s1);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            a[i] = na[i];
            b[i] = nb[i];
        }
        lin_comb<N>(t, u, v, f0, g0);
        add_qp<F>(t, (t[0] * F::M0) & 0x3fffffffu);
        shr30<N>(na, t);
        negate_if<N>(na, s0);
        into_range<F>(na);
        lin_comb<N>(t, u, v, f1, g1);
        add_qp<F>(t, (t[0] * F::M0) & 0x3fffffffu);
        shr30<N>(nb, t);
        negate_if<N>(nb, s1);
        into_range<F>(nb);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            u[i] = na[i];
            v[i] = nb[i];
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) r.v[i] = any ? v[i] : 0u;
}

// The same inversion by the four lanes of a quad, which all hold y and all
// receive the result: lanes 0 and 1 hold (a, b), lanes 2 and 3 (u, v); every
// lane runs the divsteps, each lane updates one row of its pair (even lanes
// the first), and the two rows are exchanged by shuffles.
template <class F>
__device__ __noinline__ void fe_inv_quad(Fe<F>& r, const Fe<F>& y) {
    using namespace gcd_detail;
    constexpr int N = F::N;
    const int ql = threadIdx.x & 3;
    const bool uv = ql >= 2, second = (ql & 1) != 0;
    const unsigned qm = 0xFu << (threadIdx.x & 28);
    uint32_t x[N], z[N];
    uint32_t any = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        x[i] = uv ? F::R2(i) : y.v[i];
        z[i] = uv ? 0u : F::P(i);
        any |= y.v[i];
    }
#pragma unroll 1
    for (int it = 0; it < outer_steps<F>(); ++it) {
        uint64_t ab, bb;
        int32_t f0, g0, f1, g1;
        uint32_t nz = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) nz |= x[i];
        if (__shfl_sync(qm, nz, 0, 4) == 0) break;  // lane 0's x is a
        approximate<N>(x, z, ab, bb);
        ab = __shfl_sync(qm, ab, 0, 4);
        bb = __shfl_sync(qm, bb, 0, 4);
        divsteps30(ab, bb, f0, g0, f1, g1);
        uint32_t t[N + 2], w[N + 1];
        lin_comb<N>(t, x, z, second ? f1 : f0, second ? g1 : g0);
        add_qp<F>(t, uv ? (t[0] * F::M0) & 0x3fffffffu : 0u);
        shr30<N>(w, t);
        // the sign of the row's a or b
        const bool neg = __shfl_sync(qm, (int)(w[N] >> 31), ql & 1, 4) != 0;
        negate_if<N>(w, neg);
        if (uv) into_range<F>(w);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint32_t o = __shfl_xor_sync(qm, w[i], 1, 4);
            x[i] = second ? o : w[i];
            z[i] = second ? w[i] : o;
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const uint32_t v = __shfl_sync(qm, z[i], 2, 4);
        r.v[i] = any ? v : 0u;
    }
}

// 1/a in Montgomery form (0 for 0).
template <class F>
KB_DEV void fe_inv(Fe<F>& r, const Fe<F>& a) {
    fe_inv_gcd<F>(r, a);
}

// Load / store helpers for canonical little-endian words.
template <class F>
KB_DEV void fe_load(Fe<F>& r, const uint32_t* src) {
#pragma unroll
    for (int i = 0; i < F::N; ++i) r.v[i] = src[i];
}
template <class F>
KB_DEV void fe_store(uint32_t* dst, const Fe<F>& a) {
#pragma unroll
    for (int i = 0; i < F::N; ++i) dst[i] = a.v[i];
}

// The same through 16-byte accesses: src / dst 16-byte aligned (point
// records are 2N or 4N words and N is a multiple of 4).
template <class F>
KB_DEV void fe_load16(Fe<F>& r, const uint32_t* src) {
    static_assert(F::N % 4 == 0, "16-byte field access needs N % 4 == 0");
    const uint4* s = reinterpret_cast<const uint4*>(src);
#pragma unroll
    for (int k = 0; k < F::N / 4; ++k) {
        const uint4 v = s[k];
        r.v[4 * k] = v.x;
        r.v[4 * k + 1] = v.y;
        r.v[4 * k + 2] = v.z;
        r.v[4 * k + 3] = v.w;
    }
}
template <class F>
KB_DEV void fe_store16(uint32_t* dst, const Fe<F>& a) {
    static_assert(F::N % 4 == 0, "16-byte field access needs N % 4 == 0");
    uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int k = 0; k < F::N / 4; ++k)
        d[k] = make_uint4(a.v[4 * k], a.v[4 * k + 1], a.v[4 * k + 2], a.v[4 * k + 3]);
}

// Big-endian byte string (F::BYTES long) -> little-endian words.
template <class F>
KB_DEV void fe_from_be_bytes(Fe<F>& r, const uint8_t* b) {
#pragma unroll
    for (int i = 0; i < F::N; ++i) {
        const uint8_t* q = b + F::BYTES - 4 * (i + 1);
        r.v[i] = ((uint32_t)q[0] << 24) | ((uint32_t)q[1] << 16) | ((uint32_t)q[2] << 8) |
                 (uint32_t)q[3];
    }
}
template <class F>
KB_DEV void fe_to_be_bytes(uint8_t* b, const Fe<F>& a) {
#pragma unroll
    for (int i = 0; i < F::N; ++i) {
        uint8_t* q = b + F::BYTES - 4 * (i + 1);
        q[0] = (uint8_t)(a.v[i] >> 24);
        q[1] = (uint8_t)(a.v[i] >> 16);
        q[2] = (uint8_t)(a.v[i] >> 8);
        q[3] = (uint8_t)a.v[i];
    }
}

}  // namespace kb200
