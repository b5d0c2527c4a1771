// Word-prime NTT on the GPU, behind the reference's ntt_forward /
// ntt_inverse (ntt/c-abi/c_ntt.cpp:81-179).
//
// The reference has three bodies, and each is reproduced operation for
// operation, so results agree for every input (reduced or not, any root):
//
//   CYC   n <= 2^16, modulus 998244353, pinned root: data in standard form,
//         twiddles in Montgomery form with R = 2^32, 64-bit wrapping products
//         (ntt/cpp/ntt.cpp:52-66, 100-172).
//   SMALL n <= 2^16, any other (modulus, root): both butterfly inputs reduced
//         mod q, 128-bit products, an addition without overflow check
//         (ntt/cpp/ntt.cpp:33-45, 176-219).
//   LARGE 2^16 < n <= 2^20: six-step: column sub-NTTs, diagonal twiddles,
//         row sub-NTTs; output left in the transposed layout; the upper
//         butterfly input reduced by the product only, an overflow-checked
//         addition (ntt/cpp/ntt_large.cpp:28-44, 95-122, 145-248).
//
// Every body is a radix-2 decimation-in-time transform after a bit-reversal
// permutation.  On the device each pass loads whole lines (sub-transforms, or
// the blocks and columns of a longer one) into shared memory,
// applies the bit reversal on the load, runs its radix-2 stages with the
// same butterfly pairs and twiddles as the reference, applies the fused
// post-multiply (diagonal twiddles or 1/n) and stores.  Twiddles w^e come
// from two small tables (w^e = lo[e mod 2^h] * hi[e >> h]).
//
// Products use Montgomery multiplication with R = 2^64 for odd q (the result
// equals the reference's (a*b) % q for every a < 2^64, b < q), the
// reference's own R = 2^32 formulas on the CYC path, a reduction of its own for
// 2^64 - 2^32 + 1, and shift-and-add products for even q.
#include <algorithm>
#include <cstring>
#include <map>
#include <stdexcept>
#include <tuple>
#include <vector>

#include "runtime.cuh"
#include "wntt.cuh"

namespace kb200 {
namespace {

// Cyclone-FFT prime, its pinned 2^16-th root and the Montgomery (R = 2^32)
// constant -q^-1 mod 2^32 (ntt/cpp/ntt.hpp:43-64).
constexpr uint64_t CYC_Q = 998244353ull;
constexpr uint64_t CYC_ROOT = 629671588ull;
constexpr uint64_t CYC_QINV32 = 998244351ull;
constexpr uint32_t CYC_MAX_LOG = 16;
constexpr uint32_t LARGE_MAX_LOG = 20;

enum WMode : int { W_CYC = 0, W_SMALL = 1, W_LARGE = 2 };

// Arithmetic of a pass: the mode, and for the two general bodies whether q is
// even (shift-and-add products) or the Goldilocks prime (its own reduction).
enum WKind : int {
    K_CYC = 0,
    K_SMALL = 1,
    K_LARGE = 2,
    K_SMALL_EVEN = 3,
    K_LARGE_EVEN = 4,
    K_SMALL_GOLD = 5,
    K_LARGE_GOLD = 6
};

// Up to 4096 words and 512 threads per CTA: two rounds of four-word butterflies
// a thread and stage pair.  2^20 words took 51.5 us so, 51.6 with 2048 words and 256
// threads, 54 to 60 with 1024 threads or 2048 words and 512.
constexpr int WNTT_THREADS = 512;
constexpr uint32_t WNTT_TILE = 4096;  // words per CTA (32 KiB)
// Fewer words where the lines would give fewer CTAs than SMs, down to 1024 words
// (8 KiB) or, with lines across memory, four of them (one 32-byte sector): 2^17
// words 29 -> 17 us, 2^18 31 -> 23 us.  Eight lines gave 21 us at 2^17; rows of 512
// words no more than 1024.
constexpr uint32_t WNTT_MIN_TILE = 1024;
constexpr uint32_t WNTT_MIN_LINES = 4;
constexpr uint32_t WNTT_MAX_LINE_LOG = 11;

struct WArith {
    uint64_t q;
    uint64_t qinv;  // q^-1 mod 2^64 (odd q)
    int mode;
    int even;       // q even: standard-form twiddles, shift-and-add products
    int gold;       // q = 2^64 - 2^32 + 1: standard-form twiddles
};

struct WPass {
    const uint64_t* in;
    uint64_t* out;
    uint32_t lines, log_L;
    uint64_t in_ls, in_ts, out_ls, out_ts;  // word address = line * ls + t * ts
    uint32_t line_rev_bits;                 // source line index bit-reversed over this many bits
    int bitrev;                             // slot t <- source element bitrev(t)
    int reduce_in;                          // x mod q on load
    uint32_t s_lo, s_hi;                    // radix-2 stages (1-based, inclusive)
    uint32_t gl, log_gt;                    // stage position of (line, t): line * gl + (t << log_gt)
    uint32_t log_n;                         // twiddle of stage s, index j: w^(j << (log_n - s))
    const uint64_t* tw_lo;
    const uint64_t* tw_hi;
    const uint64_t* tw_st;                  // stage twiddles of the longest line, or null
    uint32_t h;
    int post;                               // 0 none, 1: * w^(line * t), 2: * scale
    uint64_t scale;
};

__device__ __forceinline__ uint32_t brev_bits(uint32_t x, uint32_t bits) {
    return bits ? (__brev(x) >> (32 - bits)) : 0u;
}

__device__ __forceinline__ uint64_t cyc_redc(uint64_t t) {
    const uint64_t m = ((t & 0xffffffffull) * CYC_QINV32) & 0xffffffffull;
    const uint64_t u = (t + m * CYC_Q) >> 32;
    return u >= CYC_Q ? u - CYC_Q : u;
}

// a * b, four 32 x 32 products with their sums in the multiply-add's addend.
__device__ __forceinline__ void mul128(uint64_t a, uint64_t b, uint64_t& lo, uint64_t& hi) {
    const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
    const uint64_t p = (uint64_t)a0 * b0;
    const uint64_t m1 = (uint64_t)a0 * b1 + (p >> 32);
    const uint64_t m2 = (uint64_t)a1 * b0 + (uint32_t)m1;
    lo = m2 << 32 | (uint32_t)p;
    hi = (uint64_t)a1 * b1 + (m1 >> 32) + (m2 >> 32);
}

// a - b, plus q where that borrows.  The borrow becomes a mask and the addend is
// masked: seven instructions, no compare and no select.
__device__ __forceinline__ uint64_t sub_wrap(uint64_t a, uint64_t b, uint64_t q) {
    uint64_t r;
    asm("{\n\t.reg .b64 d, q1;\n\t.reg .b32 m, q0h, q0l;\n\t"
        "sub.cc.u64 d, %1, %2;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "mov.b64 {q0l, q0h}, %3;\n\t"
        "and.b32 q0l, q0l, m;\n\t"
        "and.b32 q0h, q0h, m;\n\t"
        "mov.b64 q1, {q0l, q0h};\n\t"
        "add.u64 %0, d, q1;\n\t}"
        : "=l"(r)
        : "l"(a), "l"(b), "l"(q));
    return r;
}

// q = 2^64 - 2^32 + 1.  2^64 = EPS (mod q), and adding q is subtracting EPS.
constexpr uint64_t GOLD_Q = 0xffffffff00000001ull;
constexpr uint32_t GOLD_EPS = 0xffffffffu;

// a - b, minus EPS (plus q) where that borrows.
__device__ __forceinline__ uint64_t gold_sub_wrap(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("{\n\t.reg .b64 d, q1;\n\t.reg .b32 m;\n\t"
        "sub.cc.u64 d, %1, %2;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "mov.b64 q1, {m, 0};\n\t"
        "sub.u64 %0, d, q1;\n\t}"
        : "=l"(r)
        : "l"(a), "l"(b));
    return r;
}

// a * b * 2^-64 mod q, canonical, for any a < 2^64 and b < q (q odd): the high
// words of a b and of the multiple of q with the same low word, subtracted.
__device__ __forceinline__ uint64_t mont64(uint64_t a, uint64_t b, uint64_t q, uint64_t qinv) {
    uint64_t lo, hi, l2, h2;
    mul128(a, b, lo, hi);
    mul128(lo * qinv, q, l2, h2);
    return sub_wrap(hi, h2, q);
}

// (a * b) mod q for the q above, canonical, any a, b < 2^64: with a b = lo +
// 2^64 h0 + 2^96 h1 and 2^96 = -1 (mod q), one product of mont64's three and
// three sums.  None wraps twice: lo - h1 borrows only to 2^64 - 2^32 or more,
// and h0 EPS <= 2^64 - 2^33 + 1.  2^20 words take 51.5 us, 59.7 with mont64.
__device__ __forceinline__ uint64_t gold_mul(uint64_t a, uint64_t b) {
    uint64_t lo, hi;
    mul128(a, b, lo, hi);
    const uint64_t t = gold_sub_wrap(lo, hi >> 32);
    const uint64_t u = (uint64_t)(uint32_t)hi * GOLD_EPS;
    uint64_t r;
    asm("{\n\t.reg .b64 s, e, z;\n\t.reg .b32 m;\n\t.reg .pred p;\n\t"
        "add.cc.u64 s, %1, %2;\n\t"
        "addc.u32 m, 0, 0;\n\t"
        "sub.u32 m, 0, m;\n\t"
        "mov.b64 e, {m, 0};\n\t"
        "add.u64 s, s, e;\n\t"          // s = lo + h0 EPS - h1 (mod q), below 2^64
        "add.cc.u64 z, s, %3;\n\t"      // s + EPS carries exactly from q on
        "addc.u32 m, 0, 0;\n\t"
        "setp.ne.u32 p, m, 0;\n\t"
        "selp.b64 %0, z, s, p;\n\t}"
        : "=l"(r)
        : "l"(t), "l"(u), "l"((uint64_t)GOLD_EPS));
    return r;
}

__device__ __forceinline__ uint64_t add_ovf(uint64_t a, uint64_t b, uint64_t q) {
    uint64_t s = a + b;
    if (s >= q || s < a) s -= q;
    return s;
}

// (a * b) mod q for a, b < q, any q >= 1 (used for even q only).
__device__ __noinline__ uint64_t mulmod_slow(uint64_t a, uint64_t b, uint64_t q) {
    uint64_t r = 0;
    for (int i = 63; i >= 0; --i) {
        r = add_ovf(r, r, q);
        if ((b >> i) & 1ull) r = add_ovf(r, a, q);
    }
    return r;
}

// Data word times a twiddle in the path's representation, canonical result
// (on the CYC path: the reference's mont_mul, wrapping product included).
template <int KIND>
__device__ __forceinline__ uint64_t tw_mul(const WArith& A, uint64_t a, uint64_t w) {
    if constexpr (KIND == K_CYC) return cyc_redc(a * w);
    if constexpr (KIND == K_SMALL_GOLD || KIND == K_LARGE_GOLD) return gold_mul(a, w);
    if constexpr (KIND == K_SMALL_EVEN || KIND == K_LARGE_EVEN) return mulmod_slow(a % A.q, w, A.q);
    return mont64(a, w, A.q, A.qinv);
}

template <int KIND>
__device__ __forceinline__ uint64_t tw_pow(const WArith& A, const WPass& p, uint64_t e) {
    return tw_mul<KIND>(A, p.tw_lo[e & ((1ull << p.h) - 1ull)], p.tw_hi[e >> p.h]);
}

template <int KIND>
__device__ __forceinline__ void butterfly(const WArith& A, uint64_t& x0, uint64_t& x1, uint64_t w) {
    const uint64_t u = x0;
    const uint64_t t = tw_mul<KIND>(A, x1, w);  // below q
    if constexpr (KIND == K_LARGE_GOLD) {
        x0 = gold_sub_wrap(u, GOLD_Q - t);  // u + t, less q from q on or past 2^64
        x1 = gold_sub_wrap(u, t);
    } else if constexpr (KIND == K_LARGE || KIND == K_LARGE_EVEN) {
        x0 = sub_wrap(u, A.q - t, A.q);
        x1 = sub_wrap(u, t, A.q);
    } else {
        const uint64_t s = u + t;  // unchecked: a sum past 2^64 stays wrapped
        x0 = s >= A.q ? s - A.q : s;
        x1 = sub_wrap(u, t, A.q);
    }
}

// One pass over lines of 2^log_L words, 2^log_c lines per CTA (all sizes are
// powers of two, so every index is shifts and masks).  Two stages at a time: a
// thread takes the four words of two pairs of pairs through both, so shared
// memory is read and written once for two stages; an odd stage comes first by
// itself.  Stage s's twiddles lie together in shared memory (entry half - 1 + j
// for pair distance half), so consecutive lanes read consecutive words; in one
// table of the last stage, stage 5 of a 1024-word line had its 16 entries in one
// bank.  A warp takes a contiguous run of words, so while the next stages' words
// stay inside it, only the warp synchronises.  Bound by instructions and their
// latency at two CTAs an SM (issue slots 55 % busy, ALU 50 %, DRAM 5 %).  2^20
// Goldilocks words, both passes: 88 us with runtime modes, divisions, 256 threads
// and one stage at a time; 70 with shifts, templates and these tables; 62 with the
// prime's own reduction; 60 with stage pairs; 54 with borrows as masks; 51.5 with
// the diagonal by steps and the stage table from the cache.  Other moduli gained
// from the same steps but the third: 998244353 and a 61-bit prime both 87.7 -> 59.4.
template <int KIND>
__global__ void __launch_bounds__(WNTT_THREADS) k_wntt_pass(WArith A, WPass p, uint32_t log_c) {
    __shared__ uint64_t sm[WNTT_TILE];
    __shared__ uint64_t stw[1u << WNTT_MAX_LINE_LOG];
    const uint32_t L = 1u << p.log_L;
    const uint32_t line0 = blockIdx.x << log_c;
    const uint32_t cnt = L << log_c;
    for (uint32_t idx = threadIdx.x; idx < cnt; idx += blockDim.x) {
        uint32_t c, t;
        if (p.in_ls == 1) {
            c = idx & ((1u << log_c) - 1);
            t = idx >> log_c;
        } else {
            c = idx >> p.log_L;
            t = idx & (L - 1);
        }
        const uint32_t line = line0 + c;
        const uint64_t sl = p.line_rev_bits ? brev_bits(line, p.line_rev_bits) : line;
        const uint32_t st = p.bitrev ? brev_bits(t, p.log_L) : t;
        uint64_t v = p.in[sl * p.in_ls + (uint64_t)st * p.in_ts];
        if (p.reduce_in) v %= A.q;
        sm[(c << p.log_L) + t] = v;
    }
    const bool local_tw = p.gl == 0 && p.log_gt == 0;
    if (local_tw)
        for (uint32_t k = threadIdx.x + 1; k < L; k += blockDim.x) {
            const uint32_t ls = 31 - __clz(k);  // stage ls + 1, index k - 2^ls
            stw[k - 1] = p.tw_st ? p.tw_st[k - 1]
                                 : tw_pow<KIND>(A, p, (uint64_t)(k - (1u << ls)) << (p.log_n - ls - 1));
        }
    __syncthreads();
    // twiddle of stage s for the pair whose upper word is t0 of line c
    auto twiddle = [&](uint32_t s, uint32_t c, uint32_t t0) -> uint64_t {
        if (local_tw) {
            const uint32_t half = 1u << (s - 1);
            return stw[half - 1 + (t0 & (half - 1))];
        }
        const uint64_t g = (uint64_t)(line0 + c) * p.gl + ((uint64_t)t0 << p.log_gt);
        return tw_pow<KIND>(A, p, (g & ((1ull << (s - 1)) - 1ull)) << (p.log_n - s));
    };
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t run = max(32u, cnt / (blockDim.x >> 5));  // words of a warp
    const uint32_t w0 = (threadIdx.x >> 5) * run;
    const bool any = w0 < cnt;
    uint32_t s = p.s_lo;
    // An odd stage by itself; with bit-serial products (even q) every stage of a tile
    // of fewer than four words a thread: in pairs, a thread ran two of those long
    // products one after the other, four a pair, where one at a time uses twice the
    // threads (2^7 words 65.6 -> 26.7 us, 30.8 before there were pairs; 2^8 71.7 -> 30.8,
    // 34.9; 2^10 98.3 -> 63.6, 90.2; 2^14 127 -> 90).
    auto one_stage = [&] {
        const uint32_t lh = s - 1 - p.log_gt, half = 1u << lh;  // pair distance in t
        for (uint32_t k = lane; any && k < run >> 1; k += 32) {
            const uint32_t b = (w0 >> 1) + k;
            if (b >= cnt >> 1) break;
            const uint32_t i0 = ((b >> lh) << (lh + 1)) + (b & (half - 1));
            uint64_t x0 = sm[i0], x1 = sm[i0 + half];
            butterfly<KIND>(A, x0, x1, twiddle(s, i0 >> p.log_L, i0 & (L - 1)));
            sm[i0] = x0;
            sm[i0 + half] = x1;
        }
        if (s < p.s_hi && half * 8 <= run)
            __syncwarp();
        else
            __syncthreads();
        ++s;
    };
    if (((p.s_hi + 1 - p.s_lo) & 1) && p.s_lo <= p.s_hi) one_stage();
    if constexpr (KIND == K_SMALL_EVEN || KIND == K_LARGE_EVEN)
        while (cnt < 4 * blockDim.x && s <= p.s_hi) one_stage();
    for (; s < p.s_hi; s += 2) {
        const uint32_t lh = s - 1 - p.log_gt, half = 1u << lh;
        for (uint32_t k = lane; any && k < run >> 2; k += 32) {
            const uint32_t b = (w0 >> 2) + k;
            if (b >= cnt >> 2) break;
            const uint32_t i0 = ((b >> lh) << (lh + 2)) + (b & (half - 1));
            const uint32_t c = i0 >> p.log_L, t0 = i0 & (L - 1);
            uint64_t x0 = sm[i0], x1 = sm[i0 + half], x2 = sm[i0 + 2 * half], x3 = sm[i0 + 3 * half];
            const uint64_t w = twiddle(s, c, t0);
            butterfly<KIND>(A, x0, x1, w);
            butterfly<KIND>(A, x2, x3, w);
            butterfly<KIND>(A, x0, x2, twiddle(s + 1, c, t0));
            butterfly<KIND>(A, x1, x3, twiddle(s + 1, c, t0 + half));
            sm[i0] = x0;
            sm[i0 + half] = x1;
            sm[i0 + 2 * half] = x2;
            sm[i0 + 3 * half] = x3;
        }
        if (s + 2 < p.s_hi && half * 16 <= run)
            __syncwarp();
        else
            __syncthreads();
    }
    if (p.post == 1) {
        // w^(line t): a thread's words lie a fixed step apart in t (columns) or in
        // the line (rows), so one power and one step give all of them
        uint32_t c = threadIdx.x & ((1u << log_c) - 1), t = threadIdx.x >> log_c;
        if (p.out_ls == 1) {
            const uint64_t line = line0 + c, dt = blockDim.x >> log_c;
            uint64_t f = tw_pow<KIND>(A, p, line * t);
            const uint64_t g = tw_pow<KIND>(A, p, line * dt);
            for (; t < L; t += dt, f = tw_mul<KIND>(A, f, g))
                p.out[line + t * p.out_ts] = tw_mul<KIND>(A, sm[(c << p.log_L) + t], f);
        } else {
            const uint32_t dc = max(1u, blockDim.x >> p.log_L);
            for (t = threadIdx.x & (L - 1); t < L; t += blockDim.x) {
                c = threadIdx.x >> p.log_L;
                uint64_t f = tw_pow<KIND>(A, p, (uint64_t)(line0 + c) * t);
                const uint64_t g = tw_pow<KIND>(A, p, (uint64_t)dc * t);
                for (; c < 1u << log_c; c += dc, f = tw_mul<KIND>(A, f, g))
                    p.out[(line0 + c) * p.out_ls + t] = tw_mul<KIND>(A, sm[(c << p.log_L) + t], f);
            }
        }
        return;
    }
    for (uint32_t idx = threadIdx.x; idx < cnt; idx += blockDim.x) {
        uint32_t c, t;
        if (p.out_ls == 1) {
            c = idx & ((1u << log_c) - 1);
            t = idx >> log_c;
        } else {
            c = idx >> p.log_L;
            t = idx & (L - 1);
        }
        const uint32_t line = line0 + c;
        uint64_t v = sm[(c << p.log_L) + t];
        if (p.post == 2) v = tw_mul<KIND>(A, v, p.scale);
        p.out[(uint64_t)line * p.out_ls + (uint64_t)t * p.out_ts] = v;
    }
}

// ---- host arithmetic (the reference's pow_mod / inverse semantics) ----------

uint64_t h_mulmod(uint64_t a, uint64_t b, uint64_t q) {
    return (uint64_t)(((unsigned __int128)a * b) % q);
}
// ntt/cpp/ntt.cpp:78-87: r starts at 1, the base is reduced first.
uint64_t h_powmod(uint64_t b, uint64_t e, uint64_t q) {
    uint64_t r = 1;
    b %= q;
    while (e) {
        if (e & 1) r = h_mulmod(r, b, q);
        b = h_mulmod(b, b, q);
        e >>= 1;
    }
    return r;
}

// Standard-form value -> twiddle representation of the path.
uint64_t h_rep(const WArith& A, uint64_t x) {
    if (A.mode == W_CYC) return (uint64_t)(((unsigned __int128)x << 32) % CYC_Q);
    if (A.even || A.gold) return x % A.q;
    return (uint64_t)(((unsigned __int128)(x % A.q) << 64) % A.q);
}

WArith make_arith(int mode, uint64_t q) {
    WArith A{};
    A.mode = mode;
    A.q = q;
    A.even = (mode != W_CYC) && !(q & 1);
    A.gold = mode != W_CYC && q == GOLD_Q;
    if (!A.even && mode != W_CYC) {
        uint64_t x = q;  // Newton: q*x = 1 mod 2^(3*2^k)
        for (int i = 0; i < 5; ++i) x *= 2 - q * x;
        A.qinv = x;
    }
    return A;
}

uint32_t log2_u(size_t n) {
    uint32_t l = 0;
    while (((size_t)1 << l) < n) ++l;
    return l;
}

}  // namespace

struct WordNttCache {
    struct Tables {
        DevBuf buf;
        uint32_t h = 0;
    };
    std::map<std::tuple<uint32_t, uint64_t, uint64_t, int>, Tables> tables;
    ~WordNttCache() {
        for (auto& kv : tables) kv.second.buf.release();
    }
};

WordNttCache* word_ntt_cache_create() { return new WordNttCache(); }
void word_ntt_cache_destroy(WordNttCache* c) { delete c; }

// Tables lo[k] = w^k (k < 2^h) and hi[k] = w^(k 2^h) (k < 2^(log_n - h)), in
// the path's representation, cached per (n, q, w, representation).
static const WordNttCache::Tables& get_tables(WordNttCache* cache, const WArith& A, uint32_t log_n,
                                              uint64_t w, cudaStream_t st) {
    const int rep = A.mode == W_CYC ? 0 : (A.even || A.gold ? 2 : 1);
    const auto key = std::make_tuple(log_n, A.q, w, rep);
    auto it = cache->tables.find(key);
    if (it != cache->tables.end()) return it->second;
    if (cache->tables.size() >= 64) {
        KB_CUDA(cudaStreamSynchronize(st));
        for (auto& kv : cache->tables) kv.second.buf.release();
        cache->tables.clear();
    }
    const uint32_t h = log_n / 2;
    const size_t nlo = (size_t)1 << h, nhi = (size_t)1 << (log_n - h);
    // Stage table of the longest line.  Transforms of one line fill theirs on the
    // device, but for even q, where its bit-serial products were a fifth of the
    // transform (2^8 words 39.0 us with it, 30.8 with the table from here).
    const bool one_line = log_n <= WNTT_MAX_LINE_LOG;
    const size_t nst = one_line ? (A.even ? nlo * nhi : 0) : nhi;
    std::vector<uint64_t> host(nlo + nhi + nst);
    uint64_t cur = 1 % A.q;
    for (size_t k = 0; k < nlo; ++k) {
        host[k] = h_rep(A, cur);
        cur = h_mulmod(cur, w, A.q);
    }
    const uint64_t step = h_powmod(w, nlo, A.q);
    cur = 1 % A.q;
    for (size_t k = 0; k < nhi; ++k) {
        host[nlo + k] = h_rep(A, cur);
        cur = h_mulmod(cur, step, A.q);
    }
    // stage s of a line: w^(j 2^(log_n - s)) at 2^(s-1) - 1 + j
    uint64_t* stage = host.data() + nlo + nhi;
    if (one_line && nst > 1) {
        cur = 1 % A.q;
        for (size_t j = 0; j < nst / 2; ++j) {  // the last stage, then every other of it
            stage[nst / 2 - 1 + j] = h_rep(A, cur);
            cur = h_mulmod(cur, w, A.q);
        }
        for (size_t half = nst / 4; half > 0; half /= 2)
            for (size_t j = 0; j < half; ++j) stage[half - 1 + j] = stage[2 * half - 1 + 2 * j];
    } else {
        for (size_t half = 1; half < nst; half *= 2)
            for (size_t j = 0; j < half; ++j) stage[half - 1 + j] = host[nlo + j * (nhi / (2 * half))];
    }
    WordNttCache::Tables& T = cache->tables[key];
    T.h = h;
    T.buf.reserve(host.size() * 8, st);
    KB_CUDA(cudaMemcpyAsync(T.buf.ptr, host.data(), host.size() * 8, cudaMemcpyHostToDevice, st));
    KB_CUDA(cudaStreamSynchronize(st));  // the host vector dies here
    return T;
}

static void launch_pass(const WArith& A, const WPass& p, cudaStream_t st) {
    const uint32_t sms = (uint32_t)device_sms();
    uint32_t log_c = 0;  // lines per CTA
    const bool cols = p.in_ls == 1 || p.out_ls == 1;
    while ((2u << log_c) << p.log_L <= WNTT_TILE && (2u << log_c) <= p.lines &&
           (p.lines >> (log_c + 1) >= sms ||
            (cols ? 1u << log_c < WNTT_MIN_LINES : (1u << log_c) << p.log_L < WNTT_MIN_TILE)))
        ++log_c;
    const unsigned grid = p.lines >> log_c;
    // Four words a thread, two with the bit-serial products of even q and in blocks
    // of up to 128 threads, whose loads, tables and scaling the further warps shorten
    // (a 61-bit prime, 2^8 words forward 7.2 -> 6.2 us, inverse 7.7 -> 6.2; 2^12 16.4 -> 12.4).
    // With two words a thread 2^10 words take 10.3 us, with four 8.3 to 9.3.
    const unsigned words = 1u << (p.log_L + log_c);
    const unsigned two = words >> 1, some = std::max(words >> 2, std::min(two, 128u));
    const unsigned threads = std::min<unsigned>(WNTT_THREADS, std::max(32u, A.even ? two : some));
    if (A.mode == W_CYC)
        k_wntt_pass<K_CYC><<<grid, threads, 0, st>>>(A, p, log_c);
    else if (A.gold && A.mode == W_SMALL)
        k_wntt_pass<K_SMALL_GOLD><<<grid, threads, 0, st>>>(A, p, log_c);
    else if (A.gold)
        k_wntt_pass<K_LARGE_GOLD><<<grid, threads, 0, st>>>(A, p, log_c);
    else if (A.mode == W_SMALL && !A.even)
        k_wntt_pass<K_SMALL><<<grid, threads, 0, st>>>(A, p, log_c);
    else if (A.mode == W_SMALL)
        k_wntt_pass<K_SMALL_EVEN><<<grid, threads, 0, st>>>(A, p, log_c);
    else if (!A.even)
        k_wntt_pass<K_LARGE><<<grid, threads, 0, st>>>(A, p, log_c);
    else
        k_wntt_pass<K_LARGE_EVEN><<<grid, threads, 0, st>>>(A, p, log_c);
    KB_LAUNCH_CHECK();
}

int word_ntt_device(WordNttCache* cache, uint64_t* d_data, uint64_t* d_scratch, size_t n,
                    uint64_t q, uint64_t root, bool inverse, cudaStream_t st) {
    if (!d_data || n == 0 || (n & (n - 1))) return -1;
    const uint32_t log_n = log2_u(n);
    if (n <= ((size_t)1 << CYC_MAX_LOG)) {
        if (q == 0) return -1;
        if (n <= 1) return 0;
        const uint64_t cyc_root_inv = h_powmod(CYC_ROOT, CYC_Q - 2, CYC_Q);
        const bool cyc = q == CYC_Q &&
                         (inverse ? (root == CYC_ROOT || root == cyc_root_inv) : root == CYC_ROOT);
        const WArith A = make_arith(cyc ? W_CYC : W_SMALL, q);
        uint64_t w, scale = 0;
        if (cyc) {
            w = h_powmod(CYC_ROOT, (1ull << CYC_MAX_LOG) >> log_n, CYC_Q);
            if (inverse) w = h_powmod(w, CYC_Q - 2, CYC_Q);
            if (inverse) scale = h_rep(A, h_powmod(n, CYC_Q - 2, CYC_Q));
        } else {
            w = root;  // the n-th root as given (root_inv for the inverse)
            if (inverse) scale = h_rep(A, h_powmod(n, q - 2, q));
        }
        const auto& T = get_tables(cache, A, log_n, w % q, st);
        WPass p{};
        p.log_n = log_n;
        p.tw_lo = T.buf.as<uint64_t>();
        p.tw_hi = p.tw_lo + ((size_t)1 << T.h);
        p.tw_st = log_n > WNTT_MAX_LINE_LOG || A.even ? p.tw_hi + (n >> T.h) : nullptr;
        p.h = T.h;
        p.reduce_in = A.mode == W_SMALL;
        p.bitrev = 1;
        if (log_n <= WNTT_MAX_LINE_LOG) {
            p.in = d_data;
            p.out = d_data;
            p.lines = 1;
            p.log_L = log_n;
            p.in_ls = p.out_ls = n;
            p.in_ts = p.out_ts = 1;
            p.s_lo = 1;
            p.s_hi = log_n;
            p.post = inverse ? 2 : 0;
            p.scale = scale;
            launch_pass(A, p, st);
            return 0;
        }
        if (!d_scratch) return -1;
        // two halves of the stages: with 2^11-word blocks in pass 1, 2^16 words were
        // 16 CTAs and took 39 us, 18.7 in halves (20.8 and 25.8 one and two stages up)
        const uint32_t la = (log_n + 1) / 2, lb = log_n - la;
        // pass 1: the bit-reversed blocks of 2^la elements, stages 1..la
        p.in = d_data;
        p.out = d_scratch;
        p.lines = 1u << lb;
        p.log_L = la;
        p.in_ls = 1;
        p.in_ts = 1ull << lb;
        p.line_rev_bits = lb;
        p.out_ls = 1ull << la;
        p.out_ts = 1;
        p.s_lo = 1;
        p.s_hi = la;
        launch_pass(A, p, st);
        // pass 2: columns (stride 2^la), stages la + 1..log_n
        WPass p2 = p;
        p2.in = d_scratch;
        p2.out = d_data;
        p2.lines = 1u << la;
        p2.log_L = lb;
        p2.in_ls = p2.out_ls = 1;
        p2.in_ts = p2.out_ts = 1ull << la;
        p2.line_rev_bits = 0;
        p2.bitrev = 0;
        p2.reduce_in = 0;
        p2.s_lo = la + 1;
        p2.s_hi = log_n;
        p2.gl = 1;
        p2.log_gt = la;
        p2.post = inverse ? 2 : 0;
        p2.scale = scale;
        launch_pass(A, p2, st);
        return 0;
    }
    if (n > ((size_t)1 << LARGE_MAX_LOG)) return -1;
    if (q == 0) return -1;  // 2^64: the even n has no inverse (ntt_large.cpp:66-76)
    const WArith A = make_arith(W_LARGE, q);
    // ntt_large.cpp:174-182: the transform root is omega^2; the inverse
    // recovers the forward 2n-th root by Fermat (c_ntt.cpp:147-160).
    const uint64_t omega = inverse ? h_powmod(root, q - 2, q) : root;
    const uint64_t wn = h_mulmod(omega, omega, q);
    const uint64_t w = inverse ? h_powmod(wn, q - 2, q) : wn;
    const auto& T = get_tables(cache, A, log_n, w, st);
    const uint32_t l1 = log_n / 2, l2 = log_n - l1;
    WPass col{};
    col.in = col.out = d_data;
    col.lines = 1u << l2;
    col.log_L = l1;
    col.in_ls = col.out_ls = 1;
    col.in_ts = col.out_ts = 1ull << l2;
    col.bitrev = 1;
    col.s_lo = 1;
    col.s_hi = l1;
    col.log_n = log_n;
    col.tw_lo = T.buf.as<uint64_t>();
    col.tw_hi = col.tw_lo + ((size_t)1 << T.h);
    col.tw_st = col.tw_hi + (n >> T.h);
    col.h = T.h;
    WPass row = col;
    row.lines = 1u << l1;
    row.log_L = l2;
    row.in_ls = row.out_ls = 1ull << l2;
    row.in_ts = row.out_ts = 1;
    row.s_hi = l2;
    if (!inverse) {
        col.post = 1;  // diagonal w^(i*j)
        launch_pass(A, col, st);
        launch_pass(A, row, st);
    } else {
        row.post = 1;
        launch_pass(A, row, st);
        col.post = 2;
        col.scale = h_rep(A, h_powmod(n, q - 2, q));
        launch_pass(A, col, st);
    }
    return 0;
}

}  // namespace kb200
