// G1 group arithmetic on device for the two a = 0 short-Weierstrass curves:
//   BLS12-381 G1 : y^2 = x^3 + 4 over FpBLS   (bls/cpp/bls12_381_g1.hpp)
//   BN254 G1     : y^2 = x^3 + 3 over FpBN    (bn254/cpp/bn254_g1.hpp)
//
// Coordinates: accumulators are extended Jacobian "XYZZ" points
// (x = X/ZZ, y = Y/ZZZ, ZZ^3 = ZZZ^2, infinity <=> ZZ = 0), using the
// published Explicit-Formulas-Database formulas madd-2008-s, add-2008-s,
// dbl-2008-s-1 and mdbl-2008-s-1 for a = 0.  Inputs are affine points in
// Montgomery form.  Exceptional cases (P = Q, P = -Q, infinity operands) are
// handled explicitly, so every result is the exact group element; the final
// affine encoding is therefore identical to the reference's Jacobian path.
#pragma once
#include "field.cuh"

namespace kb200 {

// Resident 128-thread blocks per SM requested for the bucket-accumulation
// kernel (sets its register budget: 5 -> 96 registers, 6 -> 80).
#ifndef KB_ACC_MIN_BLOCKS_BLS
#define KB_ACC_MIN_BLOCKS_BLS 5
#endif
#ifndef KB_ACC_MIN_BLOCKS_BN
#define KB_ACC_MIN_BLOCKS_BN 6
#endif

struct G1BLS {
    using F = FpBLS;
    static constexpr uint32_t B = 4;
    static constexpr int WIRE = 96;  // x || y, 48-byte big-endian each
    static constexpr int CURVE_ID = 2;
    static constexpr int ACC_MIN_BLOCKS = KB_ACC_MIN_BLOCKS_BLS;
};
// GLV endomorphism of BLS12-381 G1: phi(x, y) = (beta2 x, y) = [lambda](x, y)
// for lambda = u^2 - 1, with beta2 = 0x1a0111ea397fe699ec024086...0000aaac
// (a cube root of unity mod p), here in Montgomery form (beta2 * 2^384 mod p).
static __constant__ uint32_t kGlvBeta2Mont[12] = {0x8671f071, 0xcd03c9e4, 0x1fcda5d2, 0x5dab2246,
                                                  0xd3851b95, 0x587042af, 0x01bacb9e, 0x8eb60ebe,
                                                  0x83d050d2, 0x03f97d6e, 0x54638741, 0x18f02065};

// GLV endomorphism of BN254 G1: phi(x, y) = (beta x, y) = [lambda](x, y)
// with lambda = 0xb3c4d79d41a917585bfc41088d8daaa78b17ea66b99c90dd (a cube
// root of unity mod r) and beta = 0x59e26bcea0d48bacd4f263f1acdb5c4f5763473177fffffe
// (a cube root of unity mod p; the pair is matched on the generator), here
// in Montgomery form (beta * 2^256 mod p).  Every BN254 point has order r
// (cofactor 1), so the identity holds for every input point.
static __constant__ uint32_t kBnGlvBetaMont[8] = {0xd782e155, 0x71930c11, 0xffbe3323, 0xa6bb947c,
                                                  0xd4741444, 0xaa303344, 0x26594943, 0x2c3b3f0d};

struct G1BN {
    using F = FpBN;
    static constexpr uint32_t B = 3;
    static constexpr int WIRE = 64;  // x || y, 32-byte big-endian each
    static constexpr int CURVE_ID = 1;
    static constexpr int ACC_MIN_BLOCKS = KB_ACC_MIN_BLOCKS_BN;
};

template <class F>
struct Affine {
    Fe<F> x, y;
};
template <class F>
struct Xyzz {
    Fe<F> X, Y, ZZ, ZZZ;
};

// Internal affine table entries are 2N words (x then y, Montgomery form).
// The top bit of x's most significant word flags the point at infinity; it
// is free because every modulus here is below 2^(32N - 1).
constexpr uint32_t INF_FLAG = 0x80000000u;

template <class F>
KB_DEV bool aff_is_inf_words(const uint32_t* w) {
    return (w[F::N - 1] & INF_FLAG) != 0;
}

template <class F>
KB_DEV void xyzz_set_inf(Xyzz<F>& p) {
    fe_zero(p.X);
    fe_zero(p.Y);
    fe_zero(p.ZZ);
    fe_zero(p.ZZZ);
}
template <class F>
KB_DEV bool xyzz_is_inf(const Xyzz<F>& p) {
    return fe_is_zero(p.ZZ);
}
template <class F>
KB_DEV void xyzz_from_affine(Xyzz<F>& p, const Affine<F>& a) {
    p.X = a.x;
    p.Y = a.y;
    fe_one(p.ZZ);
    fe_one(p.ZZZ);
}

// dbl-2008-s-1 with a = 0.
template <class F>
KB_DEV void xyzz_dbl(Xyzz<F>& r, const Xyzz<F>& p) {
    Fe<F> U, V, W, S, M, t;
    fe_dbl(U, p.Y);
    fe_sqr(V, U);
    fe_mul(W, U, V);
    fe_mul(S, p.X, V);
    fe_sqr(t, p.X);
    fe_dbl(M, t);
    fe_add(M, M, t);
    Fe<F> X3, Y3;
    fe_sqr(X3, M);
    fe_sub(X3, X3, S);
    fe_sub(X3, X3, S);
    fe_sub(t, S, X3);
    fe_mul(Y3, M, t);
    fe_mul(t, W, p.Y);
    fe_sub(Y3, Y3, t);
    fe_mul(r.ZZ, V, p.ZZ);
    fe_mul(r.ZZZ, W, p.ZZZ);
    r.X = X3;
    r.Y = Y3;
}

// r = c ? a : b.
template <class F>
KB_DEV void fe_sel(Fe<F>& r, bool c, const Fe<F>& a, const Fe<F>& b) {
#pragma unroll
    for (int i = 0; i < F::N; ++i) r.v[i] = c ? a.v[i] : b.v[i];
}

// r = a + b without reduction (the sum below 2^(32N)).
template <class F>
KB_DEV void fe_add_raw(Fe<F>& r, const Fe<F>& a, const Fe<F>& b) {
    constexpr int N = F::N;
    r.v[0] = add_cc(a.v[0], b.v[0]);
#pragma unroll
    for (int i = 1; i < N - 1; ++i) r.v[i] = addc_cc(a.v[i], b.v[i]);
    r.v[N - 1] = addc_u32(a.v[N - 1], b.v[N - 1]);
}
// r = p - a for a in [0, p].
template <class F>
KB_DEV void fe_compl(Fe<F>& r, const Fe<F>& a) {
    constexpr int N = F::N;
    r.v[0] = sub_cc(F::P(0), a.v[0]);
#pragma unroll
    for (int i = 1; i < N - 1; ++i) r.v[i] = subc_cc(F::P(i), a.v[i]);
    r.v[N - 1] = subc_u32(F::P(N - 1), a.v[N - 1]);
}
// r = a 2^S without reduction.
template <int S, class F>
KB_DEV void fe_shl(Fe<F>& r, const Fe<F>& a) {
#pragma unroll
    for (int i = F::N - 1; i > 0; --i) r.v[i] = __funnelshift_l(a.v[i - 1], a.v[i], S);
    r.v[0] = a.v[0] << S;
}

// k >= 0 doublings of a point in shared memory (4N words: X, Y, ZZ, ZZZ)
// with the coordinates dbl-2008-s-1 gives, two product levels per doubling
// instead of three: the chain carries X^2, C = 3X^3 and D = 2Y^2 beside the
// point.  With t = C - D and u = 3C - 4D (= 9X^3 - 8Y^2), the Jacobian
// doubling for a = 0 (X' = 9X^4 - 8XY^2, Y' = 36X^3Y^2 - 27X^6 - 8Y^4,
// Z' = 2YZ, with ZZ = Z^2 and ZZZ = Z^3) reads
//   X' = X u,  Y' = 2 (D t) - C u,  ZZ' = ZZ 2D,  ZZZ' = ZZZ 4 (Y D),
//   X'^2 = X^2 u^2,  C' = (C u) u^2,  D' = Y' 2Y',
// level 1 on lanes 0..5 (X u, u^2, C u, D t, Y D, ZZ 2D), level 2 on lanes
// 0..3.  Eight lanes per point, four points to a warp, each with its own p, k
// and tmp (8N words of shared scratch); p and tmp 16-byte aligned.  All 32
// lanes call it.
//
// Bound by latency: two dependent products per doubling and what lies between
// them, so the sums between them are not reduced.  A product's second operand
// may be any N-word value and its first any below 2^(32N) - p; the result is
// below p + ab / 2^(32N), and one conditional subtraction makes it canonical
// if that is below 2p.  p / 2^(32N) is 0.102 for BLS12-381 and 0.189 for BN254:
//   BLS12-381: t < 2p, u = 3C + 4 (p - D) < 7p; u^2 < 6p stays unreduced (it is
//     a second operand next); Y' = 2 (D t) + (p - C u) less p once, < 2p, and
//     Y' 2Y' < 1.9p.
//   BN254: t canonical, u = 3t + (p - D) < 4p, u^2 < 4.1p; Y' canonical.
// Measured: 3.3 -> 2.45 us a doubling (BLS12-381) against canonical sums.
template <class F>
__device__ __noinline__ void xyzz_dbl_chain_oct(uint32_t* p, uint32_t k, uint32_t* tmp) {
    constexpr int N = F::N;
    constexpr bool WIDE = F::N == 12;  // 2^(32N) > 9p
    const int lane = threadIdx.x & 7;
    uint32_t kmax = k;
#pragma unroll
    for (int d = 16; d >= 8; d >>= 1) kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, d));
    if (kmax == 0) return;
    uint32_t* pX = p;
    uint32_t* pY = p + N;
    uint32_t* pZZ = p + 2 * N;
    uint32_t* pZZZ = p + 3 * N;
    uint32_t* tX2 = tmp;          // X^2
    uint32_t* tC = tmp + N;       // 3 X^3
    uint32_t* tD = tmp + 2 * N;   // 2 Y^2
    uint32_t* tXn = tmp + 3 * N;  // X u = X'
    uint32_t* tU2 = tmp + 4 * N;  // u^2
    uint32_t* tCU = tmp + 5 * N;  // 3 X^3 u
    uint32_t* tT = tmp + 6 * N;   // 2 Y^2 t
    uint32_t* tYD = tmp + 7 * N;  // Y 2Y^2
    Fe<F> a, b, r, c;
    // set-up: X^2 (lane 0), Y^2 (lane 1); then X X^2 (lane 0)
    fe_load16(a, lane == 1 ? pY : pX);
    fe_mul_inl(r, a, a);
    if (lane == 0) fe_store16(tX2, r);
    if (lane == 1) {
        fe_dbl(r, r);
        fe_store16(tD, r);
    }
    __syncwarp();
    fe_load16(a, pX);
    fe_load16(b, tX2);
    fe_mul_inl(r, a, b);
    if (lane == 0) {
        fe_dbl(c, r);
        fe_add(r, c, r);
        fe_store16(tC, r);
    }
    __syncwarp();
    // first operands from memory (lanes that compute nothing read tC or tCU,
    // which no lane writes at that level)
    const uint32_t* a1 = lane == 0 ? pX : (lane == 3 ? tD : (lane == 4 ? pY : (lane == 5 ? pZZ : tC)));
    const uint32_t* a2 = lane == 0 ? tX2 : (lane == 3 ? pZZZ : tCU);
    const uint32_t* b2 = lane == 3 ? tYD : tU2;
    uint32_t* o1 = lane == 0 ? tXn : (lane == 1 ? tU2 : (lane == 2 ? tCU : (lane == 3 ? tT : (lane == 4 ? tYD : pZZ))));
    uint32_t* o2 = lane == 0 ? tX2 : (lane == 1 ? tC : (lane == 2 ? tD : pZZZ));
    for (uint32_t it = 0; it < kmax; ++it) {
        const bool on = it < k;  // uniform over the point's eight lanes
        Fe<F> t, u, d, n;
        fe_load16(c, tC);
        fe_load16(d, tD);
        fe_load16(a, a1);
        fe_compl(n, d);        // p - D
        fe_add_raw(t, c, n);   // C - D + p
        if constexpr (WIDE) {
            fe_shl<1>(u, c);
            fe_add_raw(u, u, c);
            fe_shl<2>(n, n);
        } else {
            reduce_once<F>(t, t.v);
            fe_shl<1>(u, t);
            fe_add_raw(u, u, t);
        }
        fe_add_raw(u, u, n);
        fe_shl<1>(n, d);       // 2D
        fe_sel(a, lane == 1, u, a);
        fe_sel(b, lane == 3, t, d);
        fe_sel(b, lane == 5, n, b);
        fe_sel(b, lane <= 2, u, b);
        fe_mul_inl(r, a, b);
        if (on && lane < 6) fe_store16(o1, r);
        __syncwarp();
        Fe<F> yn;
        fe_load16(yn, tT);
        fe_load16(c, tCU);
        fe_load16(a, a2);
        fe_load16(b, b2);
        fe_shl<1>(yn, yn);
        fe_compl(c, c);
        fe_add_raw(yn, yn, c);  // 2 (D t) - C u + p
        reduce_once<F>(yn, yn.v);
        if constexpr (!WIDE) reduce_once<F>(yn, yn.v);
        fe_shl<2>(t, b);
        fe_sel(b, lane == 3, t, b);
        fe_shl<1>(t, yn);
        fe_sel(a, lane == 2, yn, a);
        fe_sel(b, lane == 2, t, b);
        fe_mul_inl(r, a, b);
        if (on && lane < 4) fe_store16(o2, r);
        if (on && lane == 4) {
            fe_load16(c, tXn);
            fe_store16(pX, c);
        }
        if (on && lane == 5) fe_store16(pY, yn);
        __syncwarp();
    }
    if constexpr (WIDE) {
        if (lane == 0) {
            fe_load16(c, pY);
            reduce_once<F>(c, c.v);
            fe_store16(pY, c);
        }
        __syncwarp();
    }
}

// mdbl-2008-s-1: r = 2 * (affine a).
template <class F>
KB_DEV void xyzz_mdbl(Xyzz<F>& r, const Affine<F>& a) {
    Fe<F> U, V, W, S, M, t;
    fe_dbl(U, a.y);
    fe_sqr(V, U);
    fe_mul(W, U, V);
    fe_mul(S, a.x, V);
    fe_sqr(t, a.x);
    fe_dbl(M, t);
    fe_add(M, M, t);
    fe_sqr(r.X, M);
    fe_sub(r.X, r.X, S);
    fe_sub(r.X, r.X, S);
    fe_sub(t, S, r.X);
    fe_mul(r.Y, M, t);
    fe_mul(t, W, a.y);
    fe_sub(r.Y, r.Y, t);
    r.ZZ = V;
    r.ZZZ = W;
}

// madd-2008-s: p += a, with a a finite affine point.  Temporaries are
// reused so that at most five field elements are live besides p and a.
template <class F>
KB_DEV void xyzz_add_affine(Xyzz<F>& p, const Affine<F>& a) {
    if (xyzz_is_inf(p)) {
        xyzz_from_affine(p, a);
        return;
    }
    Fe<F> P, R, t;
    fe_mul(P, a.x, p.ZZ);
    fe_sub(P, P, p.X);          // P = x2*ZZ1 - X1
    fe_mul(R, a.y, p.ZZZ);
    fe_sub(R, R, p.Y);          // R = y2*ZZZ1 - Y1
    if (fe_is_zero(P)) {
        if (fe_is_zero(R))
            xyzz_mdbl(p, a);
        else
            xyzz_set_inf(p);
        return;
    }
    Fe<F> PP, Q;
    fe_sqr(PP, P);              // PP
    fe_mul(Q, p.X, PP);         // Q = X1*PP
    fe_mul(p.ZZ, p.ZZ, PP);     // ZZ3 = ZZ1*PP
    fe_mul(PP, P, PP);          // PP <- PPP = P*PP
    fe_mul(p.ZZZ, p.ZZZ, PP);   // ZZZ3 = ZZZ1*PPP
    fe_mul(t, p.Y, PP);         // Y1*PPP
    fe_sqr(p.X, R);
    fe_sub(p.X, p.X, PP);
    fe_sub(p.X, p.X, Q);
    fe_sub(p.X, p.X, Q);        // X3 = R^2 - PPP - 2Q
    fe_sub(Q, Q, p.X);
    fe_mul(Q, R, Q);
    fe_sub(p.Y, Q, t);          // Y3 = R(Q - X3) - Y1*PPP
}

// add-2008-s: p += q, both XYZZ (either may be infinity).
template <class F>
KB_DEV void xyzz_add(Xyzz<F>& p, const Xyzz<F>& q) {
    if (xyzz_is_inf(q)) return;
    if (xyzz_is_inf(p)) {
        p = q;
        return;
    }
    Fe<F> U1, S1, P, R;
    fe_mul(U1, p.X, q.ZZ);
    fe_mul(P, q.X, p.ZZ);
    fe_sub(P, P, U1);           // P = U2 - U1
    fe_mul(S1, p.Y, q.ZZZ);
    fe_mul(R, q.Y, p.ZZZ);
    fe_sub(R, R, S1);           // R = S2 - S1
    if (fe_is_zero(P)) {
        if (fe_is_zero(R))
            xyzz_dbl(p, p);
        else
            xyzz_set_inf(p);
        return;
    }
    Fe<F> PP;
    fe_sqr(PP, P);
    fe_mul(p.ZZ, p.ZZ, q.ZZ);
    fe_mul(p.ZZ, p.ZZ, PP);     // ZZ3 = ZZ1*ZZ2*PP
    fe_mul(U1, U1, PP);         // U1 <- Q = U1*PP
    fe_mul(PP, P, PP);          // PP <- PPP = P*PP
    fe_mul(p.ZZZ, p.ZZZ, q.ZZZ);
    fe_mul(p.ZZZ, p.ZZZ, PP);   // ZZZ3 = ZZZ1*ZZZ2*PPP
    fe_mul(S1, S1, PP);         // S1*PPP
    fe_sqr(p.X, R);
    fe_sub(p.X, p.X, PP);
    fe_sub(p.X, p.X, U1);
    fe_sub(p.X, p.X, U1);       // X3 = R^2 - PPP - 2Q
    fe_sub(U1, U1, p.X);
    fe_mul(U1, R, U1);
    fe_sub(p.Y, U1, S1);        // Y3 = R(Q - X3) - S1*PPP
}

// Affine result (Montgomery form); returns false for infinity.
template <class F>
KB_DEV bool xyzz_to_affine(Affine<F>& a, const Xyzz<F>& p) {
    if (xyzz_is_inf(p)) return false;
    Fe<F> t, inv;
    fe_mul(t, p.ZZ, p.ZZZ);
    fe_inv(inv, t);           // 1 / (ZZ * ZZZ)
    Fe<F> izz, izzz;
    fe_mul(izz, inv, p.ZZZ);  // 1 / ZZ
    fe_mul(izzz, inv, p.ZZ);  // 1 / ZZZ
    fe_mul(a.x, p.X, izz);
    fe_mul(a.y, p.Y, izzz);
    return true;
}


// Memory helpers for XYZZ points stored as 4N consecutive words.
template <class F>
KB_DEV void xyzz_load(Xyzz<F>& p, const uint32_t* w) {  // w 16-byte aligned
    fe_load16(p.X, w);
    fe_load16(p.Y, w + F::N);
    fe_load16(p.ZZ, w + 2 * F::N);
    fe_load16(p.ZZZ, w + 3 * F::N);
}
template <class F>
KB_DEV void xyzz_store(uint32_t* w, const Xyzz<F>& p) {  // w 16-byte aligned
    fe_store16(w, p.X);
    fe_store16(w + F::N, p.Y);
    fe_store16(w + 2 * F::N, p.ZZ);
    fe_store16(w + 3 * F::N, p.ZZZ);
}

// An XYZZ point held in shared memory, word-major over a block of STRIDE
// threads: coordinate f (0 = X, 1 = Y, 2 = ZZ, 3 = ZZZ), word k of this
// thread at base[(f * N + k) * STRIDE].  Consecutive threads hit consecutive
// banks.  An accumulator kept here rather than in registers leaves only the
// temporaries of the formula in registers, which raises the resident warps
// per SM of the latency-bound addition kernels.
template <class F, int STRIDE>
struct SmXyzz {
    uint32_t* base;  // shared array + threadIdx.x
    KB_DEV void get(int f, Fe<F>& r) const {
#pragma unroll
        for (int k = 0; k < F::N; ++k) r.v[k] = base[(f * F::N + k) * STRIDE];
    }
    KB_DEV void put(int f, const Fe<F>& r) const {
#pragma unroll
        for (int k = 0; k < F::N; ++k) base[(f * F::N + k) * STRIDE] = r.v[k];
    }
    KB_DEV void set_inf() const {
#pragma unroll
        for (int k = 0; k < 4 * F::N; ++k) base[k * STRIDE] = 0;
    }
    KB_DEV void to_global(uint32_t* w) const {  // w 16-byte aligned
        uint4* d = reinterpret_cast<uint4*>(w);
#pragma unroll
        for (int k = 0; k < F::N; ++k)
            d[k] = make_uint4(base[(4 * k) * STRIDE], base[(4 * k + 1) * STRIDE],
                              base[(4 * k + 2) * STRIDE], base[(4 * k + 3) * STRIDE]);
    }
};

// dbl-2008-s-1 in place on a shared-memory point.
template <class F, int S>
KB_DEV void xyzz_dbl(const SmXyzz<F, S>& p) {
    Fe<F> U, V, W, t;
    p.get(1, t);
    fe_dbl(U, t);
    fe_sqr(V, U);
    fe_mul(W, U, V);
    p.get(2, t);
    fe_mul(t, V, t);
    p.put(2, t);                // ZZ3 = V*ZZ1
    p.get(0, t);
    fe_mul(U, t, V);            // U <- S = X1*V
    p.get(3, t);
    fe_mul(t, W, t);
    p.put(3, t);                // ZZZ3 = W*ZZZ1
    p.get(1, t);
    fe_mul(W, W, t);            // W <- W*Y1
    p.get(0, t);
    fe_sqr(V, t);
    fe_dbl(t, V);
    fe_add(V, V, t);            // V <- M = 3 X1^2
    fe_sqr(t, V);
    fe_sub(t, t, U);
    fe_sub(t, t, U);            // X3 = M^2 - 2S
    p.put(0, t);
    fe_sub(U, U, t);
    fe_mul(U, V, U);
    fe_sub(U, U, W);            // Y3 = M(S - X3) - W*Y1
    p.put(1, U);
}

// W consecutive words (W a multiple of 4), both 16-byte aligned.
template <int W>
KB_DEV void ld_st_words16(uint32_t* dst, const uint32_t* src) {
    uint4* d = reinterpret_cast<uint4*>(dst);
    const uint4* s = reinterpret_cast<const uint4*>(src);
#pragma unroll
    for (int k = 0; k < W / 4; ++k) d[k] = s[k];
}

// Whether a point of 4N consecutive words (16-byte aligned) is infinity.
template <class F>
KB_DEV bool point_is_inf(const uint32_t* p) {
    Fe<F> z;
    fe_load16(z, p + 2 * F::N);
    return fe_is_zero(z);
}

// Exchange with lane (own ^ 1) or from lane k of this thread's quad.
template <class F>
KB_DEV void fe_qxor1(Fe<F>& r, const Fe<F>& a, unsigned qm) {
#pragma unroll
    for (int i = 0; i < F::N; ++i) r.v[i] = __shfl_xor_sync(qm, a.v[i], 1, 4);
}
template <class F>
KB_DEV void fe_qget(Fe<F>& r, const Fe<F>& a, int k, unsigned qm) {
#pragma unroll
    for (int i = 0; i < F::N; ++i) r.v[i] = __shfl_sync(qm, a.v[i], k, 4);
}
// p += q (add-2008-s) by the four lanes of a quad, for points of 4N
// consecutive words (X, Y, ZZ, ZZZ; 16-byte aligned, p in shared memory, q
// anywhere, not aliasing p).  The 14 products fall into four dependent levels
// of at most four, so the addition is four product latencies deep; each lane
// loads only its own operands and passes the products the others need by
// quad shuffles (six field elements in all), so no lane holds a point:
//   level 1: U1 = X1 ZZ2 (0), U2 = X2 ZZ1 (1), S1 = Y1 ZZZ2 (2), S2 = Y2 ZZZ1 (3)
//   level 2: PP = P^2 (0), ZZ1 ZZ2 (1), RR = R^2 (2), ZZZ1 ZZZ2 (3)
//   level 3: PPP = P PP (0), ZZ3 = ZZ1 ZZ2 PP (1), Q = U1 PP (2)
//   level 4: S1 PPP (1), R (Q - X3) (2), ZZZ3 = ZZZ1 ZZZ2 PPP (3)
// with P = U2 - U1, R = S2 - S1, X3 = RR - PPP - 2Q.  All four lanes of the
// quad call it with the same arguments; branches are uniform in the quad.
template <class F>
__device__ __noinline__ void xyzz_add_quad_pt(uint32_t* p, const uint32_t* q) {
    constexpr int N = F::N;
    const int ql = threadIdx.x & 3, hb = ql >> 1;
    const unsigned qsh = threadIdx.x & 28, qm = 0xFu << qsh;
    const bool odd = (ql & 1) != 0;
    Fe<F> a, b, r1, r2, r, d, o;
    fe_load16(a, (odd ? q : p) + hb * N);
    fe_load16(b, (odd ? p : q) + (2 + hb) * N);
    // lane 0 holds ZZ2, lane 1 ZZ1: zero for infinity
    const unsigned inf = __ballot_sync(qm, fe_is_zero(b)) >> qsh;
    if (inf & 1u) return;
    if (inf & 2u) {
        ld_st_words16<N>(p + ql * N, q + ql * N);
        __syncwarp(qm);
        return;
    }
    fe_mul_inl(r1, a, b);
    fe_qxor1(o, r1, qm);
    fe_sel(a, odd, r1, o);
    fe_sel(o, odd, o, r1);
    fe_sub(d, a, o);  // lanes 0, 1: P; lanes 2, 3: R
    const unsigned zero = __ballot_sync(qm, fe_is_zero(d)) >> qsh;
    if (zero & 1u) {  // the same x: P = Q or P = -Q
        if (ql == 0) {
            const SmXyzz<F, 1> s{p};
            if (zero & 4u)
                xyzz_dbl(s);
            else
                s.set_inf();
        }
        __syncwarp(qm);
        return;
    }
    fe_load16(a, q + (2 + hb) * N);
    fe_sel(a, odd, a, d);
    fe_sel(b, odd, b, d);
    fe_mul_inl(r2, a, b);
    fe_qget(b, r2, 0, qm);   // PP
    fe_qget(o, r1, 0, qm);   // U1
    fe_sel(a, odd, r2, o);
    fe_sel(a, ql == 0, d, a);
    fe_mul_inl(r, a, b);     // PPP (0), ZZ3 (1), Q (2)
    if (ql == 1) fe_store16(p + 2 * N, r);
    fe_qget(b, r, 0, qm);    // PPP
    fe_qget(o, r1, 2, qm);   // S1
    // lane 2: X3 = RR - PPP - 2Q, then Q - X3
    Fe<F> x3;
    fe_sub(x3, r2, b);
    fe_sub(x3, x3, r);
    fe_sub(x3, x3, r);
    fe_sub(a, r, x3);
    fe_sel(b, ql == 2, d, b);
    fe_sel(a, odd, r2, a);   // lane 3: ZZZ1 ZZZ2
    fe_sel(a, ql == 1, o, a);
    fe_mul_inl(r, a, b);     // S1 PPP (1), R (Q - X3) (2), ZZZ3 (3)
    fe_qget(o, r, 1, qm);
    fe_sub(a, r, o);         // lane 2: Y3 = R (Q - X3) - S1 PPP
    if (ql == 3) fe_store16(p + 3 * N, r);
    if (ql == 2) {
        fe_store16(p, x3);
        fe_store16(p + N, a);
    }
    __syncwarp(qm);
}

// The same sum by eight lanes, three product latencies deep instead of four with
// 17 products instead of 14: with P, R, U1, S1 as above and E = R - S1,
//   Y3 = R (Q - X3) - S1 PPP = PP (3 R U1 + E P) - R RR,
// so nothing waits for X3:
//   level 1: U1 (0), U2 (1), S1 (2), S2 (3), ZZ1 ZZ2 (4), ZZZ1 ZZZ2 (5)
//   level 2: PP (0), RR (1), R U1 (2), E P (3), ZZZ1 ZZZ2 P (5)
//   level 3: PPP (0), R RR (1), Q (2), PP (3 R U1 + E P) (3), ZZ3 (4), ZZZ3 (5)
// 3 R U1 + E P < 4p stays unreduced as a second operand: the product is below
// p + 4p p / 2^(32N) < 1.8p.  For rounds of so few additions that quads leave
// most of an SM's warps idle: KZG commit of 4096 442 -> 408 us, of 64 279 -> 260,
// MSM of 1000 points in G1 574 -> 550.
template <class F>
__device__ __noinline__ void xyzz_add_oct_pt(uint32_t* p, const uint32_t* q) {
    constexpr int N = F::N;
    const int ol = threadIdx.x & 7;
    const unsigned osh = threadIdx.x & 24, om = 0xFFu << osh;
    auto get = [&](Fe<F>& r, const Fe<F>& a, int k) {
#pragma unroll
        for (int i = 0; i < N; ++i) r.v[i] = __shfl_sync(om, a.v[i], k, 8);
    };
    Fe<F> a, b, r1, r2, r, P, R, u1, pp, o;
    {
        // coordinates of the operands: X1 ZZ2, X2 ZZ1, Y1 ZZZ2, Y2 ZZZ1, ZZ1 ZZ2, ZZZ1 ZZZ2
        const int ca = ol < 2 || ol > 5 ? 0 : (ol < 4 ? 1 : ol - 2);
        const int cb = ol == 2 || ol == 3 || ol == 5 ? 3 : 2;
        const bool second = ol == 1 || ol == 3;
        fe_load16(a, (second ? q : p) + ca * N);
        fe_load16(b, (second ? p : q) + cb * N);
    }
    // lane 0 holds ZZ2, lane 1 ZZ1: zero for infinity
    const unsigned inf = __ballot_sync(om, fe_is_zero(b)) >> osh;
    if (inf & 1u) return;
    if (inf & 2u) {
        if (ol < 4) ld_st_words16<N>(p + ol * N, q + ol * N);
        __syncwarp(om);
        return;
    }
    fe_mul_inl(r1, a, b);
    get(u1, r1, 0);
    get(P, r1, 1);
    fe_sub(P, P, u1);
    get(o, r1, 2);  // S1
    get(R, r1, 3);
    fe_sub(R, R, o);
    if (fe_is_zero(P)) {  // the same x: P = Q or P = -Q; uniform in the eight lanes
        if (ol == 0) {
            const SmXyzz<F, 1> s{p};
            if (fe_is_zero(R))
                xyzz_dbl(s);
            else
                s.set_inf();
        }
        __syncwarp(om);
        return;
    }
    fe_sub(o, R, o);  // E
    fe_sel(a, ol == 0, P, R);
    fe_sel(a, ol == 3, o, a);
    fe_sel(a, ol == 5, r1, a);
    fe_sel(b, ol == 1, R, P);
    fe_sel(b, ol == 2, u1, b);
    fe_mul_inl(r2, a, b);
    get(pp, r2, 0);
    get(o, r2, 2);  // R U1
    fe_shl<1>(b, o);
    fe_add_raw(o, o, b);
    fe_add_raw(o, o, r2);  // lane 3: 3 R U1 + E P
    fe_sel(b, ol == 3, o, pp);
    fe_sel(b, ol == 1, r2, b);
    fe_sel(a, ol == 0, P, R);
    fe_sel(a, ol == 2, u1, a);
    fe_sel(a, ol == 3, pp, a);
    fe_sel(a, ol == 4, r1, a);
    fe_sel(a, ol == 5, r2, a);
    fe_mul_inl(r, a, b);
    get(P, r, 0);   // PPP
    get(u1, r, 2);  // Q
    get(o, r, 1);   // R RR
    fe_sub(a, r2, P);
    fe_sub(a, a, u1);
    fe_sub(a, a, u1);  // lane 1: X3 = RR - PPP - 2Q
    fe_sub(b, r, o);   // lane 3: Y3
    if (ol == 1) fe_store16(p, a);
    if (ol == 3) fe_store16(p + N, b);
    if (ol == 4 || ol == 5) fe_store16(p + (ol - 2) * N, r);
    __syncwarp(om);
}

// mdbl-2008-s-1 into a shared-memory point: p = 2 * (affine a).
template <class F, int S>
KB_DEV void xyzz_mdbl_sm(const SmXyzz<F, S>& p, const Affine<F>& a) {
    Fe<F> U, V, W, t;
    fe_dbl(U, a.y);
    fe_sqr(V, U);
    fe_mul(W, U, V);
    p.put(3, W);                // ZZZ3 = W
    fe_mul(U, a.x, V);          // U <- S = x*V
    p.put(2, V);                // ZZ3 = V
    fe_sqr(t, a.x);
    fe_dbl(V, t);
    fe_add(V, V, t);            // V <- M = 3x^2
    fe_sqr(t, V);
    fe_sub(t, t, U);
    fe_sub(t, t, U);            // X3 = M^2 - 2S
    p.put(0, t);
    fe_sub(U, U, t);
    fe_mul(U, V, U);            // M(S - X3)
    fe_mul(W, W, a.y);
    fe_sub(U, U, W);            // Y3 = M(S - X3) - W*y
    p.put(1, U);
}

// madd-2008-s on a shared-memory accumulator: p += a, a finite affine
// point.  At most five field elements are live in registers besides a.
template <class F, int S>
KB_DEV void xyzz_add_affine(const SmXyzz<F, S>& p, const Affine<F>& a) {
    Fe<F> P, R, t;
    p.get(2, t);
    if (fe_is_zero(t)) {
        p.put(0, a.x);
        p.put(1, a.y);
        fe_one(t);
        p.put(2, t);
        p.put(3, t);
        return;
    }
    {
        // the two independent products inlined so they interleave
        // (accumulation at 2^22: 2.14 -> 2.02 ms)
        Fe<F> t3;
        p.get(3, t3);
        fe_mul_inl(P, a.x, t);
        fe_mul_inl(R, a.y, t3);
    }
    p.get(0, t);
    fe_sub(P, P, t);            // P = x2*ZZ1 - X1
    p.get(1, t);
    fe_sub(R, R, t);            // R = y2*ZZZ1 - Y1
    if (fe_is_zero(P)) {
        if (fe_is_zero(R))
            xyzz_mdbl_sm(p, a);
        else
            p.set_inf();
        return;
    }
    Fe<F> PP, Q;
    fe_sqr(PP, P);              // PP
    p.get(0, t);
    fe_mul(Q, t, PP);           // Q = X1*PP
    p.get(2, t);
    fe_mul(t, t, PP);
    p.put(2, t);                // ZZ3 = ZZ1*PP
    fe_mul(PP, P, PP);          // PP <- PPP
    p.get(3, t);
    fe_mul(t, t, PP);
    p.put(3, t);                // ZZZ3 = ZZZ1*PPP
    p.get(1, t);
    fe_mul(P, t, PP);           // P <- Y1*PPP
    fe_sqr(t, R);
    fe_sub(t, t, PP);
    fe_sub(t, t, Q);
    fe_sub(t, t, Q);            // X3 = R^2 - PPP - 2Q
    p.put(0, t);
    fe_sub(Q, Q, t);
    fe_mul(Q, R, Q);
    fe_sub(Q, Q, P);            // Y3 = R(Q - X3) - Y1*PPP
    p.put(1, Q);
}

// Affine table entry (2N words) -> Affine<F>; the infinity flag is masked.
template <class F>
KB_DEV void aff_load(Affine<F>& a, const uint32_t* w) {
    fe_load(a.x, w);
    a.x.v[F::N - 1] &= ~INF_FLAG;
    fe_load(a.y, w + F::N);
}

// Wire (big-endian x || y, all-zero = infinity) -> internal table entry.
template <class C>
KB_DEV void wire_to_table(uint32_t* dst, const uint8_t* wire) {
    using F = typename C::F;
    uint32_t any = 0;
    for (int i = 0; i < C::WIRE; ++i) any |= wire[i];
    if (!any) {
        for (int i = 0; i < 2 * F::N; ++i) dst[i] = 0;
        dst[F::N - 1] = INF_FLAG;
        return;
    }
    Fe<F> x, y;
    fe_from_be_bytes(x, wire);
    fe_from_be_bytes(y, wire + F::BYTES);
    fe_to_mont(x, x);
    fe_to_mont(y, y);
    fe_store(dst, x);
    fe_store(dst + F::N, y);
}

}  // namespace kb200
