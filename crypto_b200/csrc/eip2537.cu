// EIP-2537 BLS12_G1MSM on the GPU, behind the reference's bls12_381_g1_msm
// (bls/c-abi/c_bls_pairing.cpp:106-110; body bls/cpp/bls.cpp:194-254, which
// hands the work to blst).  One thread per entry checks, as the reference
// does before its Pippenger call:
//   * each coordinate, a 64-byte big-endian integer, is below p
//     (bls.cpp:33-41; so its top 16 bytes are zero);
//   * the point is on y^2 = x^3 + 4, or is (0,0), the EIP-2537 infinity
//     (bls.cpp:44-58);
//   * the point is in G1 (bls.cpp:217-218), by the endomorphism test:
//     P in G1 iff sigma(P) = -[u^2]P, with sigma(x, y) = (beta x, y), beta a
//     cube root of unity in Fp and u = -0xd201000000010000 the curve
//     parameter (M. Scott, "A note on group membership tests for G1, G2 and
//     GT on BLS pairing-friendly curves", 2021);
// then drops infinity entries (bls.cpp:220-222), reduces the big-endian
// scalar mod r (the sum over points of order r is unchanged), and runs the
// G1 MSM of msm.cu on the resulting table.
#include "curve.cuh"
#include "eip2537.cuh"
#include "g1check.cuh"
#include "msm_reduce.cuh"
#include "runtime.cuh"

namespace kb200 {
namespace {

using F = FpBLS;
using FR = FrBLS;

// A 64-byte big-endian coordinate below p (its top 16 bytes zero).
__device__ bool coord_ok(const uint8_t* c, Fe<F>& v) {
    uint32_t hi = 0;
    for (int i = 0; i < 16; ++i) hi |= c[i];
    fe_from_be_bytes(v, c + 16);
    return hi == 0 && below_modulus(v);
}

// MEMBER: whether the membership test runs here, on the entry's one thread,
// or after this kernel in k_g1msm_member.
template <bool MEMBER>
__global__ void __launch_bounds__(128) k_g1msm_unpack(const uint8_t* __restrict__ xycs, uint32_t n,
                                                      uint32_t* __restrict__ table,
                                                      uint8_t* __restrict__ scalars,
                                                      uint32_t* __restrict__ flag) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint8_t* e = xycs + (size_t)160 * i;
    uint32_t* row = table + (size_t)i * 2 * F::N;
    uint32_t* sc = reinterpret_cast<uint32_t*>(scalars + (size_t)32 * i);
    Fe<F> x, y;
    bool ok = coord_ok(e, x);
    ok = coord_ok(e + 64, y) && ok;
    bool inf = false;
    if (ok) {
        inf = fe_is_zero(x) && fe_is_zero(y);
        if (!inf) {
            Affine<F> a;
            fe_to_mont(a.x, x);
            fe_to_mont(a.y, y);
            ok = g1_on_curve(a);
            if constexpr (MEMBER) ok = ok && g1_in_subgroup(a);
            fe_store(row, a.x);
            fe_store(row + F::N, a.y);
        }
    }
    // GLV row n + i: phi(P) = (beta2 x, y) = [lambda]P, valid because every
    // accepted point is in G1 (the subgroup check above)
    uint32_t* grow = row + (size_t)n * 2 * F::N;
    if (!ok) atomicOr(flag, 1u);
    if (!ok || inf) {
        for (int k = 0; k < 2 * F::N; ++k) row[k] = grow[k] = 0;
        row[F::N - 1] = grow[F::N - 1] = INF_FLAG;
        for (int k = 0; k < 8; ++k) sc[k] = 0;
        return;
    }
    {
        Fe<F> bx, b, yy;
        fe_load(bx, row);
        fe_load(yy, row + F::N);
        for (int k = 0; k < F::N; ++k) b.v[k] = kGlvBeta2Mont[k];
        fe_mul(bx, bx, b);
        fe_store(grow, bx);
        fe_store(grow + F::N, yy);
    }
    Fe<FR> s;
    fe_from_be_bytes(s, e + 128);
    while (!below_modulus(s)) {  // at most twice: 2^256 < 3r
        uint32_t b = 0;
        for (int k = 0; k < FR::N; ++k) {
            const uint64_t d = (uint64_t)s.v[k] - FR::P(k) - b;
            s.v[k] = (uint32_t)d;
            b = (uint32_t)(d >> 63);
        }
    }
    for (int k = 0; k < 8; ++k) sc[k] = s.v[k];
}

// The membership test of g1_in_subgroup by eight lanes per point: the [|u|]
// chains' doublings spread over six lanes, two product latencies each
// (xyzz_dbl_chain_oct), their additions over four.  For few points, where one
// thread per point leaves the chip idle for two chains of about 500 dependent
// products: a call of 1000 entries 1.56 -> 1.01 ms.  A point outside G1 sets the
// flag and becomes an infinity row with a zero scalar, as in k_g1msm_unpack.
constexpr int MEMBER_THREADS = 128, MEMBER_POINTS = MEMBER_THREADS / 8;

__global__ void __launch_bounds__(MEMBER_THREADS) k_g1msm_member(uint32_t n, uint32_t* __restrict__ table,
                                                                 uint8_t* __restrict__ scalars,
                                                                 uint32_t* __restrict__ flag) {
    constexpr int N = F::N, PS = RED_PS<F>;
    // per point: the accumulator, the chain's addend, the chain's scratch
    __shared__ __align__(16) uint32_t s_acc[MEMBER_POINTS * PS], s_add[MEMBER_POINTS * PS],
        s_tmp[MEMBER_POINTS * 8 * N];
    const int oct = threadIdx.x >> 3, ol = threadIdx.x & 7;
    const uint32_t i = blockIdx.x * MEMBER_POINTS + (uint32_t)oct;
    uint32_t* row = table + (size_t)min(i, n - 1) * 2 * N;
    uint32_t* acc = s_acc + oct * PS;
    uint32_t* add = s_add + oct * PS;
    const bool live = i < n && !aff_is_inf_words<F>(row);
    {
        // lane c < 4 sets coordinate c of P = (x, y, 1, 1); infinity rows
        // run the chains on infinity
        Fe<F> v;
        fe_zero(v);
        if (live) {
            if (ol < 2)
                fe_load16(v, row + ol * N);
            else
                fe_one(v);
        }
        if (ol < 4) {
            fe_store16(acc + ol * N, v);
            fe_store16(add + ol * N, v);
        }
    }
    __syncwarp();
    bool ok = true;
#pragma unroll 1
    for (int chain = 0; chain < 2; ++chain) {
        // [|u|] from the top bit: doublings down to each next set bit
        int bit = 63;
#pragma unroll 1
        while (bit > 0) {
            const uint64_t below = BLS_U_ABS & ((1ull << bit) - 1);
            const int next = below ? 63 - __clzll((long long)below) : 0;
            xyzz_dbl_chain_oct<F>(acc, (uint32_t)(bit - next), s_tmp + oct * 8 * N);
            if (below && ol < 4) xyzz_add_quad_pt<F>(acc, add);
            __syncwarp();
            bit = next;
        }
        if (chain == 0) {
            ok = !point_is_inf<F>(acc);  // [|u|]P = O: P is torsion outside G1
            if (ol < 4) quad_copy<F>(add, acc);
            __syncwarp();
        }
    }
    // sigma(P) = -[u^2]P: beta x ZZ == X (lane 0), -y ZZZ == Y (lane 1)
    Fe<F> a, b;
    fe_load16(a, row + (ol & 1) * N);
    if (ol & 1) {
        fe_neg(a, a);
    } else {
        fe_load(b, kG1Beta);
        fe_to_mont(b, b);
        fe_mul(a, a, b);
    }
    fe_load16(b, acc + (2 + (ol & 1)) * N);
    fe_mul(a, a, b);
    fe_load16(b, acc + (ol & 1) * N);
    ok = ok && fe_eq(a, b) && !point_is_inf<F>(acc);
    const unsigned m = __ballot_sync(0xffffffffu, ok) >> (threadIdx.x & 24);
    if (!live || (m & 3u) == 3u) return;
    if (ol == 0) atomicOr(flag, 1u);
    if (ol < 2) {
        uint32_t* r = row + (ol ? (size_t)n * 2 * N : 0);  // the point's row, its GLV row
        for (int k = 0; k < 2 * N; ++k) r[k] = k == N - 1 ? INF_FLAG : 0u;
    } else if (ol == 2) {
        for (int k = 0; k < 8; ++k) reinterpret_cast<uint32_t*>(scalars + (size_t)32 * i)[k] = 0;
    }
}

// Entries up to which eight lanes check a point's membership.  Eight lanes do
// about twice the work of one in a quarter of its depth, so they lose once
// they fill the chip: whole calls with one lane / eight, 1000 entries 1.56 /
// 1.01 ms, 4000 1.66 / 1.25, 8192 1.73 / 1.77, 10000 1.77 / 2.13.
constexpr size_t MEMBER_OCT_MAX = 7168;

}  // namespace

void g1_msm_eip2537_device(MsmEngine* eng, const uint8_t* d_xycs, size_t n, uint32_t* d_table,
                           uint8_t* d_scalars, uint32_t* d_flag, uint8_t* d_out_wire,
                           cudaStream_t st) {
    KB_CUDA(cudaMemsetAsync(d_flag, 0, sizeof(uint32_t), st));
    if (n) {
        const unsigned g = ceil_div_u(n, 128);
        if (n <= MEMBER_OCT_MAX) {
            k_g1msm_unpack<false><<<g, 128, 0, st>>>(d_xycs, (uint32_t)n, d_table, d_scalars, d_flag);
            KB_LAUNCH_CHECK();
            k_g1msm_member<<<ceil_div_u(n, MEMBER_POINTS), MEMBER_THREADS, 0, st>>>((uint32_t)n, d_table,
                                                                                  d_scalars, d_flag);
        } else {
            k_g1msm_unpack<true><<<g, 128, 0, st>>>(d_xycs, (uint32_t)n, d_table, d_scalars, d_flag);
        }
        KB_LAUNCH_CHECK();
    }
    MsmOptions opt;
    opt.glv = true;  // d_table holds the phi rows from row n on
    opt.glv_rows = n;
    msm_run_table(eng, d_scalars, d_table, n, d_out_wire, nullptr, st, opt);
}

}  // namespace kb200
