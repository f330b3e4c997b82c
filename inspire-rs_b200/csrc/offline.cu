// offline.cu — the offline precomputation of the InspiRING packing on the GPU: from the
// encoded DB to a_hat, bold_t, bold_t_bar, bold_t_hat (the arrays respond() streams).
//
// Restates PirServer::perform_offline_precomputation_simplepir (rkdud007/inspire-rs
// src/pir/server/engine.rs:677-1042) for gamma = N: per packing instance I (DB columns
// I*N .. I*N + N)
//   a_j   = NTT(negacyclic_perm(hint column I*N + j))              prep_pack_lwes, packing.rs:1032-1062
//           hint column = INTT(sum_row NTT(DB chunk) * query_row)  multiply_with_db_ring, engine.rs:434-498
//   r_i   = sum_j NTT(+-x^(j g'_i mod 2N)) * a_j,  g'_i = 5^((N-i) mod N)   packing.rs:2627-2679
//   r_all[i] = automorph(N^-1 r_i, 5^i),  r_bar_all[i] likewise with -j g'_i and 2N - 5^i
//   collapse over i = 1022 .. 0 (gadget digits, NTT, MAC with the rotated W mask)  packing.rs:2683-2734
//
// B200 design.  The reference forms r_i by brute force (2048 x 2048 products per slot and
// instance).  With E[s][z] = sum_j a_j[s] psi_z^j, the negacyclic NTT over j of the slot-s
// sequence, the sum collapses to a gather:
//   r_all[i][z] = N^-1 E[tau_{5^i}(z)][z],   r_bar_all[i][z] = N^-1 E[tau_{-5^i}(z)][z]
// (tau_t = the NTT-domain automorphism slot map; 5^i g'_i = 1 mod 2N).  So the whole packing
// sum is one NTT per (instance, limb, slot).  And since negacyclic_perm is x -> x^-1, a_j
// itself is the slot permutation tau_{-1} of NTT(DB column) * query: the hint's INTT/NTT
// pair cancels.  Kernels, per limb:
//   k_off_hint     column NTTs of the DB, * query, tau_{-1}          -> act[l][I][j][s]
//   k_off_jntt     NTT over j of 8 slots per CTA, * N^-1, the gather -> F[I][chain][i][l][z]
//   k_off_collapse one CTA pair per (instance, chain): 1023 sequential steps of register NTTs
//   k_off_finish   bold_t_hat and a_hat per instance
// All values leave canonical, so the outputs equal the reference's bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "host_math.hpp"
#include "ipr_b200.h"
#include "ipr_device.cuh"
#include "kernels.cuh"
#include "ntt_lazy.cuh"
#include "ntt_regs.cuh"
#include "umma.cuh"

namespace ipr {
void set_last_error(const char* msg);

namespace {

using nttr::eA;
using nttr::eD;
using nttr::EPT;
constexpr int HALF = N / 2;   // packing outputs per instance (num_to_pack_half)
constexpr int HCOLS = 4;      // LWE columns per CTA in k_lwe_prep
constexpr int HP = 2;         // DB columns per CTA in k_off_hint
constexpr int JS = 8;         // slots per CTA in k_off_jntt
constexpr uint64_t MASK19 = (1ull << GADGET_BITS) - 1;

__device__ __forceinline__ uint32_t limb_q(int g) { return g ? Q1 : Q0; }
__device__ __forceinline__ uint64_t limb_br(int g) { return g ? BR1 : BR0; }

// 5^i mod 2N (gen_pows, packing.rs:1645-1652)
__device__ __forceinline__ uint32_t gen_pow(uint32_t i) {
    uint32_t r = 1, b = 5;
    for (; i; i >>= 1, b = (b * b) & (2 * N - 1))
        if (i & 1) r = (r * b) & (2 * N - 1);
    return r;
}

// store of eight words: one L2 sector at a time (WIDE: 32-byte aligned), else 8 bytes at a time
template <bool WIDE>
__device__ __forceinline__ void st_sector(uint32_t* p, const uint32_t (&w)[8]) {
    if (!WIDE) {
#pragma unroll
        for (int i = 0; i < 8; i += 2) reinterpret_cast<uint64_t*>(p)[i / 2] = (uint64_t)w[i] | ((uint64_t)w[i + 1] << 32);
        return;
    }
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

// act[l][c][s] = tau_{-1}-permuted NTT_l(DB column c) * query, for chunk-local columns c.
// Bound by instruction issue: one limb and HP columns per CTA of 256 threads (four CTAs per SM),
// the lazily reduced digit transform (DB entries are below 2^16).  129,024 columns 1.36 ms,
// against 2.76 ms for both limbs of four columns in one CTA on canonical butterflies.
// grid (ncols / HP, 2 limbs)
__global__ void __launch_bounds__(256, 4)
    k_off_hint(const uint16_t* __restrict__ db, int64_t db_rows, int64_t col0, int64_t ncols,
               const uint32_t* __restrict__ query, const uint2* __restrict__ fwi, uint32_t* __restrict__ act) {
    __shared__ __align__(16) uint32_t xbuf[HP * N];
    const int g = blockIdx.y, t = threadIdx.x;
    const uint32_t q = limb_q(g);
    const uint64_t br = limb_br(g);
    const int64_t c0 = (int64_t)blockIdx.x * HP;
    const int polys = (int)(db_rows / N);
    uint32_t acc[HP][EPT];  // canonical running sum over the column's row polynomials
#pragma unroll
    for (int p = 0; p < HP; p++)
#pragma unroll
        for (int m = 0; m < EPT; m++) acc[p][m] = 0;
    for (int row = 0; row < polys; row++) {
        uint32_t v[HP][EPT];
#pragma unroll
        for (int p = 0; p < HP; p++) {
            const uint16_t* col = db + (col0 + c0 + p) * db_rows + (int64_t)row * N;
#pragma unroll
            for (int m = 0; m < EPT; m++) v[p][m] = (uint32_t)__ldg(col + eA(t, m));
        }
        nttl::forward_digits<HP, true, true>(v, t, xbuf, 1, fwi + g * N, q);  // layout D, below 10 q
        uint32_t qr[EPT];
        nttl::load_d8(qr, query + ((int64_t)row * 2 + g) * N + eD(t, 0));
#pragma unroll
        for (int p = 0; p < HP; p++)
#pragma unroll
            for (int m = 0; m < EPT; m++) acc[p][m] = mod64((uint64_t)v[p][m] * qr[m] + acc[p][m], q, br);
    }
    // slot w = eD(t, m) holds V[w]; the permuted polynomial has V[w] at tau_{-1}(w) (an involution)
    nttr::group_bar(1);
#pragma unroll
    for (int p = 0; p < HP; p++)
#pragma unroll
        for (int m = 0; m < EPT; m++) xbuf[p * N + auto_src(2 * N - 1, eD(t, m))] = acc[p][m];
    nttr::group_bar(1);
#pragma unroll
    for (int p = 0; p < HP; p++) {
        uint32_t* dst = act + ((int64_t)g * ncols + c0 + p) * N;
#pragma unroll
        for (int m = 0; m < EPT; m++) dst[eA(t, m)] = xbuf[p * N + eA(t, m)];
    }
}

// rows of F: v[u >> 1] = chain * HALF + i with u = 5^i (chain 0) or -5^i (chain 1) mod 2N; every
// odd u is one of them
struct RowOfPower {
    uint16_t v[N];
};
constexpr RowOfPower rows_of_powers() {
    RowOfPower r{};
    uint32_t u = 1;
    for (int i = 0; i < HALF; i++, u = u * 5 % (2 * N)) {
        r.v[u >> 1] = (uint16_t)i;
        r.v[(2 * N - u) >> 1] = (uint16_t)(HALF + i);
    }
    return r;
}
__device__ const RowOfPower d_row_of_power = rows_of_powers();

__host__ __device__ constexpr int rev3(int x) { return ((x & 1) << 2) | (x & 2) | ((x >> 2) & 1); }

// E[s][z] = v[s - s0][z - z8], s = s0 .. s0 + 7, z = z8 .. z8 + 7 -> the F sectors made of them.
// A group of eight slots has exponents e + 512 r (r = the reversed low bits of the slot), and
// u (e + 512 r) = u e + 512 u r: tau_u takes groups to groups.  The eight u that take this z group
// to this s group are (e_s + 512 h) / e_z, h = 0 .. 7, all with the same u mod 8 = A, and tau_u
// takes r to h + A r.
template <int A>
__device__ __forceinline__ void store_sectors(const uint32_t (&v)[JS][EPT], uint32_t es, uint32_t ez_inv,
                                              uint32_t* __restrict__ F) {
#pragma unroll
    for (int h = 0; h < 8; h++) {
        const uint32_t u = ((es + 512 * h) * ez_inv) & (2 * N - 1);
        uint32_t* dst = F + (int64_t)__ldg(&d_row_of_power.v[u >> 1]) * 2 * N;
        uint32_t w[8];
#pragma unroll
        for (int m = 0; m < 8; m++) w[m] = v[rev3((h + A * rev3(m)) & 7)][m];
        st_sector<true>(dst, w);
    }
}

// E[l][I][s][z] = N^-1 * NTT over j of act[l][I][j][s], JS consecutive slots per CTA (the 32 bytes
// of a row that they take are one sector).  GATHER: written as
//   F[I][chain][i][l][z] = E[l][I][tau(z)][z], tau = tau_{5^i} (chain 0) or tau_{-5^i} (chain 1),
// which a thread can do from its registers, a whole sector at a time (store_sectors); else as E
// (`out`, 32-byte aligned, is not act).
// 96 instances (act and F 3.2 GB each): 2.73 ms (2.4 TB/s; bound by the transforms' issue), against
// 2.50 ms for writing E and 1.76 ms for a gather over tiles of eight columns of it.
// grid (N / JS, instances, 2 limbs), 256 threads, 64 KB of dynamic shared memory
template <bool GATHER>
__global__ void __launch_bounds__(256, 2)
    k_off_jntt(const uint32_t* __restrict__ act, int64_t inst, const uint2* __restrict__ fwi, uint32_t* __restrict__ out) {
    extern __shared__ __align__(16) uint32_t jbuf[];  // [JS][N]
    const int t = threadIdx.x;
    const int s0 = blockIdx.x * JS, l = blockIdx.z;
    const int64_t base = ((int64_t)l * inst + blockIdx.y) * N * N;
    const uint32_t q = limb_q(l);
    uint32_t v[JS][EPT];
#pragma unroll
    for (int m = 0; m < EPT; m++) {
        const uint4* src = reinterpret_cast<const uint4*>(act + base + (int64_t)eA(t, m) * N + s0);
        const uint4 a = __ldg(src), b = __ldg(src + 1);
        v[0][m] = a.x; v[1][m] = a.y; v[2][m] = a.z; v[3][m] = a.w;
        v[4][m] = b.x; v[5][m] = b.y; v[6][m] = b.z; v[7][m] = b.w;
    }
    nttl::forward_digits<JS, false, true>(v, t, jbuf, 1, fwi + l * N, q);  // canonical in: below 15 q through stage 6
    const uint32_t ninv = q - (q - 1) / N, ninvp = (uint32_t)(((uint64_t)ninv << 32) / q);  // N^-1 mod q_l
#pragma unroll
    for (int p = 0; p < JS; p++)
#pragma unroll
        for (int k = 0; k < EPT; k++) v[p][k] = nttl::mul_canon(v[p][k], ninv, ninvp, q);
    const int z8 = eD(t, 0);
    if (!GATHER) {
#pragma unroll
        for (int p = 0; p < JS; p++) st_sector<true>(out + base + (int64_t)(s0 + p) * N + z8, v[p]);
        return;
    }
    const uint32_t es = exponent_of_slot((uint32_t)s0), ez = exponent_of_slot((uint32_t)z8);
    uint32_t inv = ez;  // 1 / ez mod 8, then mod 64, 2^12
    inv *= 2 - ez * inv;
    inv *= 2 - ez * inv;
    uint32_t* F = out + ((int64_t)blockIdx.y * 2 * HALF * 2 + l) * N + z8;
    switch ((es * inv) & 7) {  // the same for a warp: ez mod 8 comes from the two high bits of t
        case 1: store_sectors<1>(v, es, inv, F); break;
        case 3: store_sectors<3>(v, es, inv, F); break;
        case 5: store_sectors<5>(v, es, inv, F); break;
        default: store_sectors<7>(v, es, inv, F); break;
    }
}
constexpr int JNTT_SMEM = JS * N * 4;

// smem of the finish kernel
struct CollapseSmem {
    uint64_t x[N];               // raw value of the chain (canonical mod q)
    uint32_t wm[3][2][N];        // V mask, NTT domain
    uint32_t xb[2][3][N];        // per limb group: NTT exchange buffers / limb staging
};

// digits of x in layout A for group-local thread t: v[k][m] = bits [19k, 19k + 19) of x[eA(t, m)]
// (gadget_invert_transposed_into, packing.rs:2740-2768)
__device__ __forceinline__ void digits(const uint64_t* x, int t, uint32_t (&v)[3][EPT]) {
#pragma unroll
    for (int m = 0; m < EPT; m++) {
        const uint64_t e = x[eA(t, m)];
#pragma unroll
        for (int k = 0; k < 3; k++) v[k][m] = (uint32_t)((e >> (GADGET_BITS * k)) & MASK19);
    }
}

// y (layout D, canonical limb g) -> raw x = CRT of both limbs, through the staging buffers;
// all 512 threads take part
__device__ __forceinline__ void to_raw(CollapseSmem& sm, uint32_t (&y)[1][EPT], int g, int t,
                                       const uint32_t* __restrict__ iw, const uint32_t* __restrict__ iwp) {
    const uint32_t q = limb_q(g);
    nttr::inverse<1, 1>(y, t, &sm.xb[g][0][0], 1 + g, iw + g * N, iwp + g * N, q);  // layout A, canonical
    __syncthreads();  // both groups are done with their exchange buffers
#pragma unroll
    for (int m = 0; m < EPT; m++) sm.xb[g][1][eA(t, m)] = y[0][m];
    __syncthreads();
    for (int e = threadIdx.x; e < N; e += 512) sm.x[e] = crt2(sm.xb[0][1][e], sm.xb[1][1][e], Q0INV, BR1);
    __syncthreads();
}

// N^-1 mod q_l and N^-1 R mod q_l (R = 2^32), each with its Shoup companion
struct CollapseScale {
    uint32_t ninv[4], ninvr[4];  // {w0, wp0, w1, wp1}
};

struct ChainSmem {
    uint32_t xb[3][N];            // exchange buffer of the transforms
    uint32_t wm[3][N];            // this limb's W mask times N^-1 R
    uint4 ex[2][5][256];          // from the other limb, halves used in turn: x's residues (2), digits (3)
    uint64_t bars[2];
};

constexpr uint32_t INV5 = 3277;  // 5^-1 mod 2N

// One cluster of two CTAs (one per limb) of 256 threads per (instance, chain); chain 0 folds
// r_all with W rotated by 5^i into bold_t, chain 1 folds r_bar_all with W rotated by -5^i
// into bold_t_bar.  Leaves the final NTT-domain r_all[0] (chain 0) or raw(r_bar_all[0])
// (chain 1) for k_off_finish.  With WROWS the W row of step i is read from
// wrows[chain][i][k][l][z] instead of being rotated out of the mask (the reference's collapse
// takes w_all / w_bar_all as arrays).
//
// Bound by the latency of a step where chains are few and by instruction issue where they
// fill the chip: 1023 dependent steps of three forward transforms, a product and one inverse
// transform per limb.  A limb needs the other only for the CRT, so each has an SM's
// schedulers to itself, and one exchange per step through distributed shared memory
// (asynchronous stores counted on an mbarrier of the receiver) carries the residues; both CTAs
// then compose x, which thread t keeps as its 8 coefficients of layout A.  The same exchange
// carries half of the transformed digits, so that each CTA stores whole 32-byte sectors of the
// interleaved bold_t rows.  A CTA sends into a half of the exchange buffer again only after it
// has received what its partner sent after reading that half.  A wait that runs out is
// remembered, later waits are skipped, the chain runs on to the common last barrier and the
// error is reported.  The transforms are the fold's lazily
// reduced ones; their N^-1 sits in the W mask (with the Montgomery R) and in F.
// One instance (2 chains) 4.6 us a step, 74 instances (two chains' CTAs per SM) 7.5 us, against
// 14 us a step for one 512-thread CTA per chain, which also stored bold_t in 4-byte pieces.
// A cluster barrier per exchange in place of the counted stores: 5.0 us (its memory barrier); a
// team of 256 threads per digit: 5.4 us (two more CTA barriers).  FEW, for at most one CTA per
// SM, has the registers to load twiddles above the barriers: 4.4 us.
template <bool WROWS, bool FEW, bool WIDE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(256, FEW ? 1 : 2)
    k_off_collapse(const uint32_t* __restrict__ F, int64_t inst0, const uint32_t* __restrict__ wmask,
                   const uint2* __restrict__ fwi, const uint2* __restrict__ iwi, CollapseScale sc,
                   uint64_t* __restrict__ bt, uint64_t* __restrict__ btb, uint32_t* __restrict__ r0,
                   uint64_t* __restrict__ xbar0, const uint32_t* __restrict__ wrows, int* __restrict__ err_flag) {
    extern __shared__ __align__(16) uint8_t csm_raw[];
    ChainSmem& sm = *reinterpret_cast<ChainSmem*>(csm_raw);
    const int t = threadIdx.x;
    const int g = (int)umma::cluster_rank(), peer = g ^ 1;
    const int64_t I = blockIdx.x >> 1;
    const int chain = blockIdx.y;
    const uint32_t q = limb_q(g);
    const uint32_t* Fc = F + (I * 2 + chain) * (int64_t)HALF * 2 * N + g * N;  // [i][l][z], this limb
    uint32_t* out = reinterpret_cast<uint32_t*>((chain ? btb : bt) + (inst0 + I) * (int64_t)NINNER * N);
    const uint2 *fw = fwi + g * N, *iw = iwi + g * N;
    const uint32_t nv = sc.ninv[2 * g], nvp = sc.ninv[2 * g + 1];
    if (!WROWS)
        for (int e = t; e < 3 * N; e += 256)
            sm.wm[e / N][e % N] = nttl::mul_canon(__ldg(wmask + (e / N * 2 + g) * N + e % N), sc.ninvr[2 * g],
                                                  sc.ninvr[2 * g + 1], q);
    const uint32_t* wr = WROWS ? wrows + (int64_t)chain * NROT * 3 * 2 * N + g * N : nullptr;
    const int z8 = 8 * t;  // layout D: this thread's slots z8 .. z8 + 7
    const uint32_t ez = exponent_of_slot((uint32_t)z8);
    uint64_t x[EPT];
    uint32_t y[EPT];
    bool ok = true;
    // 16 bytes of step use n to slot k of the same thread of the other CTA
    auto send = [&](uint32_t n, int k, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
        umma::st_async16(umma::map_to_rank(&sm.ex[n & 1][k][t], (uint32_t)peer), w0, w1, w2, w3,
                         umma::map_to_rank(&sm.bars[n & 1], (uint32_t)peer));
    };
    auto receive = [&](uint32_t n, uint32_t bytes) {  // thread 0 says how many bytes this use counts
        if (t == 0) umma::mbar_expect_tx(&sm.bars[n & 1], bytes);
        if (ok) ok = umma::mbar_wait_cluster(&sm.bars[n & 1], (n >> 1) & 1);
    };
    // y (N^-1 times the limb's values, layout D) -> x: inverse transform, exchange, CRT
    auto to_raw2 = [&](uint32_t n, uint32_t bytes) {
        nttl::inverse_one<FEW>(y, t, &sm.xb[0][0], 1, iw, q);
        send(n, 0, y[0], y[1], y[2], y[3]);
        send(n, 1, y[4], y[5], y[6], y[7]);
        receive(n, bytes);
        const uint4 a = sm.ex[n & 1][0][t], b = sm.ex[n & 1][1][t];
        const uint32_t o[EPT] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int m = 0; m < EPT; m++) x[m] = crt2m(g ? o[m] : y[m], g ? y[m] : o[m]);
    };
    if (t == 0) {
        umma::mbar_init(&sm.bars[0], 1);
        umma::mbar_init(&sm.bars[1], 1);
        umma::fence_mbar_init();
    }
    // x = raw(r_all[1023]): r_all[1023] is never updated (packing.rs:2691)
    nttl::load_d8(y, Fc + (int64_t)(HALF - 1) * 2 * N + z8);
#pragma unroll
    for (int m = 0; m < EPT; m++) y[m] = nttl::mul_canon(y[m], nv, nvp, q);
    umma::cluster_sync();  // both CTAs run, their mbarriers may be signalled, and wm is loaded
    to_raw2(0, 2 * 256 * 16);
    uint32_t n = 0;  // exchanges done since
    uint32_t gi = gen_pow(HALF - 2);
    for (int i = HALF - 2; i >= 0; i--) {
        n++;
        uint32_t f[EPT];
        nttl::load_d8(f, Fc + (int64_t)i * 2 * N + z8);
        uint32_t v[3][EPT];
#pragma unroll
        for (int m = 0; m < EPT; m++)
#pragma unroll
            for (int k = 0; k < 3; k++) v[k][m] = (uint32_t)((x[m] >> (GADGET_BITS * k)) & MASK19);
        nttl::forward_digits<3, FEW>(v, t, &sm.xb[0][0], 1, fw, q);
        uint32_t own[3][4];
#pragma unroll
        for (int k = 0; k < 3; k++) {
#pragma unroll
            for (int m = 0; m < EPT; m++) v[k][m] = nttr::csub(v[k][m], q);
#pragma unroll
            for (int m = 0; m < 4; m++) own[k][m] = g ? v[k][4 + m] : v[k][m];
            send(n, 2 + k, g ? v[k][0] : v[k][4], g ? v[k][1] : v[k][5], g ? v[k][2] : v[k][6], g ? v[k][3] : v[k][7]);
        }
        const uint32_t ti = chain ? 2 * N - gi : gi;
        if (WROWS) {
            uint64_t acc[EPT];
#pragma unroll
            for (int m = 0; m < EPT; m++) acc[m] = f[m];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                uint32_t w[EPT];
                nttl::load_d8(w, wr + ((int64_t)i * 3 + k) * 2 * N + z8);
#pragma unroll
                for (int m = 0; m < EPT; m++) acc[m] += (uint64_t)w[m] * v[k][m];  // < 2^31 + 3 q^2
            }
#pragma unroll
            for (int m = 0; m < EPT; m++) y[m] = nttl::mul_canon(mod64(acc[m], q, limb_br(g)), nv, nvp, q);
        } else {
#pragma unroll
            for (int m = 0; m < EPT; m++) {
                // exponent of slot z8 + m: the three low bits of a slot are the high bits of its exponent
                const uint32_t em = ez + (uint32_t)((((m & 1) << 2) | (m & 2) | (m >> 2)) << 9);
                const uint32_t src = slot_of_exponent((ti * em) & (2 * N - 1));  // W rotated by t_i (apply_automorph_ntt)
                uint64_t acc = 0;
#pragma unroll
                for (int k = 0; k < 3; k++) acc += (uint64_t)sm.wm[k][src] * v[k][m];  // < 3 q^2 < q R
                const uint32_t s = redc(acc, q) + shoup_lazy(f[m], nv, nvp, q);        // < 4 q
                y[m] = nttr::csub(nttr::csub(s, 2 * q), q);
            }
        }
        gi = (gi * INV5) & (2 * N - 1);
        const bool last = i == 0 && chain == 0;
        if (last) {  // r_all[0] stays in the NTT domain for k_off_finish, without the N^-1
            uint4* d = reinterpret_cast<uint4*>(r0 + (I * 2 + g) * N + z8);
            uint32_t o[EPT];
#pragma unroll
            for (int m = 0; m < EPT; m++) o[m] = mod64((uint64_t)y[m] * N, q, limb_br(g));
            d[0] = make_uint4(o[0], o[1], o[2], o[3]);
            d[1] = make_uint4(o[4], o[5], o[6], o[7]);
            receive(n, 3 * 256 * 16);
        } else {
            to_raw2(n, 5 * 256 * 16);
        }
        // bold_t[i][k] condensed: limb 0 in the low word, limb 1 in the high word
        // (condense_matrix); this CTA stores slots z8 + 4 g .. + 4
#pragma unroll
        for (int k = 0; k < 3; k++) {
            uint32_t w[8];
            const uint4 e = sm.ex[n & 1][2 + k][t];
            const uint32_t o[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
            for (int m = 0; m < 4; m++) {
                w[2 * m] = g ? o[m] : own[k][m];
                w[2 * m + 1] = g ? own[k][m] : o[m];
            }
            st_sector<WIDE>(out + (((int64_t)i * 3 + k) * N + z8 + 4 * g) * 2, w);
        }
    }
    if (chain == 1 && g == 0)
#pragma unroll
        for (int m = 0; m < EPT; m++) xbar0[I * N + eA(t, m)] = x[m];
    umma::cluster_sync();  // every store into this CTA has landed
    if (!ok) {  // device memory or mapped host memory
        *static_cast<volatile int*>(err_flag) = 33;
        __threadfence_system();
    }
}

// per instance: bold_t_hat = NTT(digits(raw(r_bar_all[0]))), a_hat = raw(r_all[0] + V * bold_t_hat)
// (packing.rs:2721-2734)
__global__ void __launch_bounds__(512, 1)
    k_off_finish(const uint32_t* __restrict__ r0, const uint64_t* __restrict__ xbar0, int64_t inst0,
                 const uint32_t* __restrict__ vmask, const uint32_t* __restrict__ fw, const uint32_t* __restrict__ fwp,
                 const uint32_t* __restrict__ iw, const uint32_t* __restrict__ iwp, uint64_t* __restrict__ bth,
                 uint64_t* __restrict__ a_hat) {
    extern __shared__ __align__(16) uint8_t fsm_raw[];
    CollapseSmem& sm = *reinterpret_cast<CollapseSmem*>(fsm_raw);
    const int g = threadIdx.x >> 8, t = threadIdx.x & 255;
    const int64_t I = blockIdx.x;
    const uint32_t q = limb_q(g);
    const uint64_t br = limb_br(g);
    for (int e = threadIdx.x; e < 3 * 2 * N; e += 512) (&sm.wm[0][0][0])[e] = __ldg(vmask + e);
    for (int e = threadIdx.x; e < N; e += 512) sm.x[e] = xbar0[I * N + e];
    __syncthreads();
    uint32_t v[3][EPT];
    digits(sm.x, t, v);
    nttr::forward<3, 3>(v, t, &sm.xb[g][0][0], 1 + g, fw + g * N, fwp + g * N, q);
    uint32_t* out = reinterpret_cast<uint32_t*>(bth + (inst0 + I) * 3 * (int64_t)N);
    uint32_t y[1][EPT];
#pragma unroll
    for (int m = 0; m < EPT; m++) {
        const int z = eD(t, m);
        uint64_t acc = r0[(I * 2 + g) * N + z];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            out[((int64_t)k * N + z) * 2 + g] = v[k][m];
            acc += (uint64_t)sm.wm[k][g][z] * v[k][m];
        }
        y[0][m] = mod64(acc, q, br);
    }
    __syncthreads();
    to_raw(sm, y, g, t, iw, iwp);
    for (int e = threadIdx.x; e < N; e += 512) a_hat[(inst0 + I) * N + e] = sm.x[e];
}

// act[l][c][i][s] = NTT_l(negacyclic_perm(a-vector of LWE i of set c)) (prep_pack_lwes,
// packing.rs:1032-1062) for LWE matrices lwe[c][N + 1][N] (row j = coefficient j of the 2048
// a-vectors, row N = the b values).  negacyclic_perm keeps coefficient 0 and puts
// q - a[N - k] at k >= 1; modulo q_l (q = 0 mod q_l) that is -a[N - k].
// grid (N / HCOLS, sets, 2 limbs): a CTA takes one limb of HCOLS LWEs, whose entries of a row are
// one sector (WIDE: 32-byte aligned matrices, one load; 8-byte loads otherwise).
// 37 / 74 sets packed in 7.75 / 13.8 ms, against 8.67 / 15.7 ms with both limbs of four LWEs in one
// 512-thread CTA, 8-byte loads and canonical butterflies.
template <bool WIDE>
__global__ void __launch_bounds__(256, 3)
    k_lwe_prep(const uint64_t* __restrict__ lwe, int64_t sets, const uint2* __restrict__ fwi,
               uint32_t* __restrict__ act) {
    __shared__ __align__(16) uint32_t xbuf[HCOLS * N];
    const int g = blockIdx.z, t = threadIdx.x;
    const uint32_t q = limb_q(g);
    const uint64_t br = limb_br(g);
    const int i0 = blockIdx.x * HCOLS;
    const int64_t c = blockIdx.y;
    const uint64_t* L = lwe + c * (int64_t)(N + 1) * N + i0;
    static_assert(HCOLS == 4, "one sector of a row");
    uint32_t v[HCOLS][EPT];
#pragma unroll
    for (int m = 0; m < EPT; m++) {
        const int k = eA(t, m);
        const uint64_t* row = L + (int64_t)(k ? N - k : 0) * N;
        uint64_t w[HCOLS];
        if (WIDE)
            asm volatile("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
                         : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                         : "l"(row));
        else
#pragma unroll
            for (int p = 0; p < HCOLS; p++) w[p] = __ldg(row + p);
#pragma unroll
        for (int p = 0; p < HCOLS; p++) {
            const uint32_t x = mod64(w[p], q, br);
            v[p][m] = (k == 0 || x == 0) ? x : q - x;
        }
    }
    nttl::forward_digits<HCOLS>(v, t, xbuf, 1, fwi + g * N, q);  // canonical in: below 15 q through stage 6
#pragma unroll
    for (int p = 0; p < HCOLS; p++) {
        uint4* dst = reinterpret_cast<uint4*>(act + (((int64_t)g * sets + c) * N + i0 + p) * N + eD(t, 0));
#pragma unroll
        for (int m = 0; m < EPT; m++) v[p][m] = nttr::csub(v[p][m], q);
        dst[0] = make_uint4(v[p][0], v[p][1], v[p][2], v[p][3]);
        dst[1] = make_uint4(v[p][4], v[p][5], v[p][6], v[p][7]);
    }
}

// packed RLWE of set c: row 0 = a_hat, row 1 = b + raw(sum), the sum not reduced (add_raw,
// packing.rs:3011-3016)
__global__ void k_inspiring_out(const uint64_t* __restrict__ a_hat, const uint64_t* __restrict__ R,
                                const uint64_t* __restrict__ lwe, int64_t sets, uint64_t* __restrict__ out) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < sets * N; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = e / N, k = e % N;
        out[c * 2 * N + k] = a_hat[e];
        out[c * 2 * N + N + k] = lwe[(c * (N + 1) + N) * N + k] + R[e];
    }
}

// F[c][chain][i][l][z] (u32) from the reference's r_all / r_bar_all ([c][i][l*N + z] u64, canonical)
__global__ void k_off_to_f(const uint64_t* __restrict__ r_all, const uint64_t* __restrict__ r_bar_all, int64_t cols,
                           uint32_t* __restrict__ F) {
    const int64_t n = cols * HALF * 2 * N;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = e / ((int64_t)HALF * 2 * N), rest = e % ((int64_t)HALF * 2 * N);
        F[(c * 2 + 0) * (int64_t)HALF * 2 * N + rest] = (uint32_t)r_all[e];
        F[(c * 2 + 1) * (int64_t)HALF * 2 * N + rest] = (uint32_t)r_bar_all[e];
    }
}

// u64 [n] -> u32 [n] (canonical residues)
__global__ void k_narrow(const uint64_t* __restrict__ in, int64_t n, uint32_t* __restrict__ out) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        out[e] = (uint32_t)in[e];
}

// [limb][N] twiddles and companions -> interleaved pairs; the pre-halved inverse twiddles doubled
__global__ void k_interleave(const uint32_t* __restrict__ fw, const uint32_t* __restrict__ fwp,
                             const uint32_t* __restrict__ iw, uint2* __restrict__ fwi, uint2* __restrict__ iwi) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 2 * N) return;
    const uint32_t q = limb_q(e / N);
    fwi[e] = make_uint2(fw[e], fwp[e]);
    const uint32_t w = nttr::csub(2 * iw[e], q);
    iwi[e] = make_uint2(w, (uint32_t)(((uint64_t)w << 32) / q));
}

constexpr uint64_t pow_mod(uint64_t b, uint64_t e, uint64_t q) {
    uint64_t r = 1;
    for (; e; e >>= 1, b = b * b % q)
        if (e & 1) r = r * b % q;
    return r;
}

CollapseScale collapse_scale() {
    CollapseScale sc;
    for (int l = 0; l < 2; l++) {
        const uint64_t q = l ? Q1 : Q0, n = pow_mod(N, q - 2, q), nr = n * ((1ull << 32) % q) % q;
        sc.ninv[2 * l] = (uint32_t)n;
        sc.ninv[2 * l + 1] = (uint32_t)((n << 32) / q);
        sc.ninvr[2 * l] = (uint32_t)nr;
        sc.ninvr[2 * l + 1] = (uint32_t)((nr << 32) / q);
    }
    return sc;
}

// shared-memory sizes of the collapse kernels, on the current device
cudaError_t collapse_attributes() {
    cudaError_t e;
    const int smem = (int)sizeof(ChainSmem);
    if ((e = cudaFuncSetAttribute(k_off_collapse<false, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) ||
        (e = cudaFuncSetAttribute(k_off_collapse<false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) ||
        (e = cudaFuncSetAttribute(k_off_collapse<false, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) ||
        (e = cudaFuncSetAttribute(k_off_collapse<true, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) ||
        (e = cudaFuncSetAttribute(k_off_collapse<true, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)))
        return e;
    return cudaFuncSetAttribute(k_off_finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CollapseSmem));
}

// whether the collapse can write whole 32-byte sectors (the branch inside the kernel's serial loop
// made one instance 4.58 ms instead of 4.49, so it is a form of its own)
bool whole_sectors(const uint64_t* bt, const uint64_t* btb) {
    return ((reinterpret_cast<uintptr_t>(bt) | reinterpret_cast<uintptr_t>(btb)) & 31) == 0;
}

// the collapse of c instances from F; wrows as k_off_collapse
void launch_collapse(const uint32_t* F, int64_t inst0, int64_t c, const uint32_t* wmask, const uint2* fw, const uint2* iw,
                     uint64_t* bt, uint64_t* btb, uint32_t* r0, uint64_t* xb, int* err_flag, int sm_count,
                     cudaStream_t st) {
    const dim3 grid((unsigned)(2 * c), 2);
    const int smem = (int)sizeof(ChainSmem);
    const auto kernel = !whole_sectors(bt, btb)  ? k_off_collapse<false, false, false>
                        : 4 * c <= sm_count ? k_off_collapse<false, true, true>
                                            : k_off_collapse<false, false, true>;
    kernel<<<grid, 256, smem, st>>>(F, inst0, wmask, fw, iw, collapse_scale(), bt, btb, r0, xb, nullptr, err_flag);
}

int cuda_fail(cudaError_t e, const char* what) {
    static thread_local char buf[256];
    snprintf(buf, sizeof(buf), "offline precomputation: %s: %s", what, cudaGetErrorString(e));
    set_last_error(buf);
    return e == cudaErrorMemoryAllocation ? IPR_E_OOM : IPR_E_CUDA;
}

}  // namespace

// The collapse of `cols` columns from the reference's r_all / r_bar_all arrays with explicit W
// rows (wrows = [2][1023][3][2][N] u32: w_all then w_bar_all) and the V mask ([3][2][N] u32):
// bold_t / bold_t_bar [cols][3069][N], bold_t_hat [cols][3][N] condensed, a_hat [cols][N].
// Scratch: F (cols * 32 MB), r0 (cols * 16 KB), xb (cols * 16 KB), itab (8 N words: the given
// tables with their companions interleaved, the inverse twiddles without the halving).
cudaError_t offline_collapse_arrays(const uint64_t* r_all, const uint64_t* r_bar_all, int64_t cols,
                                    const uint32_t* wrows, const uint32_t* vmask, const uint32_t* tab /*fw fwp iw iwp*/,
                                    uint32_t* F, uint32_t* r0, uint64_t* xb, uint32_t* itab, int* err_flag, uint64_t* bt, uint64_t* btb,
                                    uint64_t* bth, uint64_t* a_hat, cudaStream_t st) {
    const int coll_smem = (int)sizeof(CollapseSmem);
    cudaError_t e = collapse_attributes();
    if (e) return e;
    const uint32_t *fw = tab, *fwp = tab + 2 * N, *iw = tab + 4 * N, *iwp = tab + 6 * N;
    k_off_to_f<<<148 * 8, 256, 0, st>>>(r_all, r_bar_all, cols, F);
    uint2* it = reinterpret_cast<uint2*>(itab);
    k_interleave<<<2 * N / 256, 256, 0, st>>>(fw, fwp, iw, it, it + 2 * N);
    const auto kernel = whole_sectors(bt, btb) ? k_off_collapse<true, false, true> : k_off_collapse<true, false, false>;
    kernel<<<dim3((unsigned)(2 * cols), 2), 256, (int)sizeof(ChainSmem), st>>>(
        F, 0, nullptr, it, it + 2 * N, collapse_scale(), bt, btb, r0, xb, wrows, err_flag);
    k_off_finish<<<(unsigned)cols, 512, coll_smem, st>>>(r0, xb, 0, vmask, fw, fwp, iw, iwp, bth, a_hat);
    return cudaGetLastError();
}

// E[l][I][s][z] = N^-1 * NTT over j of act[l][I][j][s] for `inst` instances
cudaError_t offline_jntt(const uint32_t* act, int64_t inst, const uint2* fwi, uint32_t* E, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(k_off_jntt<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, JNTT_SMEM);
    if (e != cudaSuccess) return e;
    k_off_jntt<false><<<dim3(N / JS, (unsigned)inst, 2), 256, JNTT_SMEM, st>>>(act, inst, fwi, E);
    return cudaGetLastError();
}

cudaError_t narrow_u64(const uint64_t* in, int64_t n, uint32_t* out, cudaStream_t st) {
    k_narrow<<<148 * 4, 256, 0, st>>>(in, n, out);
    return cudaGetLastError();
}

// scratch bytes per instance: F (32 MB) and the chain ends (32 KB); act (32 MB) is dead before the
// collapse writes bold_t (48 MB per instance) and lives there when that is 16-byte aligned and
// apart from the DB (which is read until act is complete), else in scratch too
constexpr uint64_t kOfflineScratchPerInstance = 2ull * N * N * 4 + 2ull * N * 4 + (uint64_t)N * 8;
static_assert(2ull * N * N * 4 <= (uint64_t)NINNER * N * 8, "act fits in bold_t");

int offline_precompute_device(const uint16_t* d_db, uint64_t db_rows, uint64_t instances, uint64_t* d_a_hat,
                              uint64_t* d_bt, uint64_t* d_btb, uint64_t* d_bth, uint64_t scratch_budget,
                              cudaStream_t st) {
    if (!d_db || !d_a_hat || !d_bt || !d_btb || !d_bth || !instances || !db_rows || db_rows % N ||
        db_rows > (1u << 20) || instances > (1u << 20)) {
        set_last_error("offline precomputation: db_rows must be a positive multiple of 2048, instances > 0");
        return IPR_E_ARGS;
    }
    int device = 0, sm_count = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        sm_count = 0;  // the general form
    HostParams hp;
    host_params_init(hp);
    std::vector<uint32_t> query, wmask, vmask;
    offline_host_inputs(hp, (unsigned)(db_rows / N), query, wmask, vmask);
    // chunk of instances per pass, bounded by the scratch budget (0 = 4 GiB)
    const uint64_t budget = scratch_budget ? scratch_budget : (4ull << 30);
    const uint64_t db0 = reinterpret_cast<uintptr_t>(d_db), bt0 = reinterpret_cast<uintptr_t>(d_bt);
    const bool apart = db0 >= bt0 + instances * NINNER * N * 8 || bt0 >= db0 + instances * N * db_rows * 2;
    const bool in_place = apart && bt0 % 16 == 0;
    const uint64_t per = kOfflineScratchPerInstance + (in_place ? 0 : 2ull * N * N * 4);
    const uint64_t chunk = std::max<uint64_t>(1, std::min<uint64_t>(instances, budget / per));
    // one allocation for everything (each costs about 0.8 ms with its release): the parts, each a
    // multiple of 256 bytes
    const size_t tb = 2 * N * sizeof(uint32_t);
    uint8_t* d_scratch = nullptr;
    size_t used = 0;
    auto part = [&](size_t bytes) {
        const size_t at = used;
        used += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t plane = chunk * 2ull * N * N * 4;
    const size_t o_F = part(plane), o_act = part(in_place ? 0 : plane),
                 o_r0 = part(chunk * 2ull * N * 4), o_xb = part(chunk * (uint64_t)N * 8), o_tab = part(8 * tb),
                 o_query = part(query.size() * 4), o_wv = part(2 * wmask.size() * 4), o_err = part(sizeof(int));
    cudaError_t e = cudaMalloc(&d_scratch, used);
    if (e != cudaSuccess) return cuda_fail(e, "scratch allocation");
    auto u32 = [&](size_t at) { return reinterpret_cast<uint32_t*>(d_scratch + at); };
    uint32_t *d_tab = u32(o_tab), *d_query = u32(o_query), *d_wv = u32(o_wv), *d_F = u32(o_F), *d_r0 = u32(o_r0);
    uint64_t* d_xb = reinterpret_cast<uint64_t*>(d_scratch + o_xb);
    int* d_err = reinterpret_cast<int*>(d_scratch + o_err);
    uint32_t *d_fw = d_tab, *d_fwp = d_tab + 2 * N, *d_iw = d_tab + 4 * N, *d_iwp = d_tab + 6 * N;
    uint32_t *d_fwi = d_tab + 8 * N, *d_iwi = d_tab + 12 * N;  // interleaved with their companions
    uint32_t *d_wm = d_wv, *d_vm = d_wv + wmask.size();
    int status = IPR_OK;
    do {
        if ((e = cudaMemsetAsync(d_err, 0, sizeof(int), st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(d_fw, hp.fw.data(), tb, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(d_fwp, hp.fwp.data(), tb, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(d_iw, hp.iw.data(), tb, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(d_iwp, hp.iwp.data(), tb, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(d_fwi, hp.fwi.data(), 2 * tb, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(d_iwi, hp.iwi.data(), 2 * tb, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(d_query, query.data(), query.size() * 4, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(d_wm, wmask.data(), wmask.size() * 4, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(d_vm, vmask.data(), vmask.size() * 4, cudaMemcpyHostToDevice, st)) != cudaSuccess) {
            status = cuda_fail(e, "table upload");
            break;
        }
        const int coll_smem = (int)sizeof(CollapseSmem);
        if ((e = cudaFuncSetAttribute(k_off_jntt<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, JNTT_SMEM)) ||
            (e = collapse_attributes())) {
            status = cuda_fail(e, "kernel attributes");
            break;
        }
        for (uint64_t i0 = 0; i0 < instances && status == IPR_OK; i0 += chunk) {
            const int64_t c = (int64_t)std::min<uint64_t>(chunk, instances - i0);
            const int64_t ncols = c * N;
            const uint2* fwi = reinterpret_cast<uint2*>(d_fwi);
            uint32_t* d_act = in_place ? reinterpret_cast<uint32_t*>(d_bt + i0 * NINNER * N) : u32(o_act);
            k_off_hint<<<dim3((unsigned)(ncols / HP), 2), 256, 0, st>>>(d_db, (int64_t)db_rows, (int64_t)i0 * N, ncols,
                                                                        d_query, fwi, d_act);
            k_off_jntt<true><<<dim3(N / JS, (unsigned)c, 2), 256, JNTT_SMEM, st>>>(d_act, c, fwi, d_F);
            launch_collapse(d_F, (int64_t)i0, c, d_wm, fwi, reinterpret_cast<uint2*>(d_iwi), d_bt, d_btb, d_r0, d_xb,
                            d_err, sm_count, st);
            k_off_finish<<<(unsigned)c, 512, coll_smem, st>>>(d_r0, d_xb, (int64_t)i0, d_vm, d_fw, d_fwp, d_iw, d_iwp,
                                                              d_bth, d_a_hat);
            if ((e = cudaGetLastError()) != cudaSuccess) status = cuda_fail(e, "launch");
        }
        int flag = 0;
        if (status == IPR_OK &&
            ((e = cudaMemcpyAsync(&flag, d_err, sizeof(int), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
             (e = cudaStreamSynchronize(st)) != cudaSuccess))
            status = cuda_fail(e, "run");
        if (status == IPR_OK && flag) {
            set_last_error("offline precomputation: a device-side wait ran out");
            status = IPR_E_TIMEOUT;
        }
    } while (false);
    cudaStreamSynchronize(st);
    cudaFree(d_scratch);
    return status;
}

}  // namespace ipr

extern "C" int ipr_offline_precompute(int device, const uint16_t* d_db, uint64_t db_rows, uint64_t instances,
                                      uint64_t* d_a_hat, uint64_t* d_bold_t, uint64_t* d_bold_t_bar,
                                      uint64_t* d_bold_t_hat, uint64_t scratch_bytes, void* stream) {
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        ipr::set_last_error(cudaGetErrorString(e));
        return IPR_E_CUDA;
    }
    return ipr::offline_precompute_device(d_db, db_rows, instances, d_a_hat, d_bold_t, d_bold_t_bar, d_bold_t_hat,
                                          scratch_bytes, static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------
// InspiRING packing of LWE sets (packing_fully_online, packing.rs:3122-3162): the offline
// kernels above on the sets' own a-vectors, then the online packing sum and INTT of the
// respond() path (k_pack, k_intt_crt) with the caller's packing keys.
// ---------------------------------------------------------------------------
struct ipr_inspiring {
    int device = 0;
    int max_sets = 0;
    int sm_count = 148;
    CUtensorMap tm_bt, tm_btb;
    std::vector<void*> allocs;
    uint32_t *fw = nullptr, *fwp = nullptr, *iw = nullptr, *iwp = nullptr, *wm = nullptr, *vm = nullptr;
    uint32_t *fwi = nullptr, *iwi = nullptr;  // the twiddles interleaved with their companions
    uint32_t *act = nullptr, *F = nullptr, *r0 = nullptr, *S = nullptr;
    int *h_err = nullptr, *d_err = nullptr;  // mapped host memory: a device-side wait ran out
    uint64_t *xb = nullptr, *a_hat = nullptr, *bt = nullptr, *btb = nullptr, *bth = nullptr, *R = nullptr;
    template <typename T>
    cudaError_t alloc(T** p, size_t bytes) {
        void* v = nullptr;
        cudaError_t e = cudaMalloc(&v, bytes);
        if (e == cudaSuccess) allocs.push_back(v), *p = static_cast<T*>(v);
        return e;
    }
};

namespace {
// the status of the calls whose kernels have run since the last report: the error word is taken
// and cleared in one, so each failure is reported once
int inspiring_error(ipr_inspiring* c) {
    const int code = __atomic_exchange_n(c->h_err, 0, __ATOMIC_ACQ_REL);
    if (!code) return IPR_OK;
    char buf[128];
    snprintf(buf, sizeof(buf), "ipr_inspiring: a device-side wait of an earlier pack ran out (code %d)", code);
    ipr::set_last_error(buf);
    return IPR_E_TIMEOUT;
}
}  // namespace

extern "C" {

void ipr_inspiring_destroy(ipr_inspiring* ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    for (void* p : ctx->allocs) cudaFree(p);
    if (ctx->h_err) cudaFreeHost(ctx->h_err);
    delete ctx;
}

int ipr_inspiring_create(int device, int max_sets, ipr_inspiring** out) {
    if (!out || max_sets < 1 || max_sets > 1024) {
        ipr::set_last_error("ipr_inspiring_create: max_sets must be in [1, 1024]");
        return IPR_E_ARGS;
    }
    *out = nullptr;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return ipr::cuda_fail(e, "set device");
    auto* c = new ipr_inspiring();
    c->device = device;
    c->max_sets = max_sets;
    cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, device);
    ipr::HostParams hp;
    ipr::host_params_init(hp);
    std::vector<uint32_t> query, wmask, vmask;
    ipr::offline_host_inputs(hp, 1, query, wmask, vmask);
    const size_t tb = 2 * ipr::N * 4, ms = (size_t)max_sets, NN = (size_t)ipr::N * ipr::N;
    if ((e = c->alloc(&c->fw, tb)) || (e = c->alloc(&c->fwp, tb)) || (e = c->alloc(&c->iw, tb)) ||
        (e = c->alloc(&c->iwp, tb)) || (e = c->alloc(&c->fwi, 2 * tb)) || (e = c->alloc(&c->iwi, 2 * tb)) || (e = c->alloc(&c->wm, wmask.size() * 4)) ||
        (e = c->alloc(&c->vm, vmask.size() * 4)) || (e = c->alloc(&c->act, ms * 2 * NN * 4)) ||
        (e = c->alloc(&c->F, ms * 2 * NN * 4)) || (e = c->alloc(&c->r0, ms * 2 * ipr::N * 4)) ||
        (e = c->alloc(&c->xb, ms * ipr::N * 8)) || (e = c->alloc(&c->a_hat, ms * ipr::N * 8)) ||
        (e = c->alloc(&c->bt, ms * ipr::NINNER * ipr::N * 8)) || (e = c->alloc(&c->btb, ms * ipr::NINNER * ipr::N * 8)) ||
        (e = c->alloc(&c->bth, ms * 3 * ipr::N * 8)) || (e = c->alloc(&c->S, ms * 2 * ipr::N * 4)) ||
        (e = c->alloc(&c->R, ms * ipr::N * 8)) ||
        (e = cudaHostAlloc(&c->h_err, sizeof(int), cudaHostAllocMapped)) ||
        (e = cudaHostGetDevicePointer(&c->d_err, c->h_err, 0)) ||
        (e = cudaMemcpy(c->fw, hp.fw.data(), tb, cudaMemcpyHostToDevice)) ||
        (e = cudaMemcpy(c->fwp, hp.fwp.data(), tb, cudaMemcpyHostToDevice)) ||
        (e = cudaMemcpy(c->iw, hp.iw.data(), tb, cudaMemcpyHostToDevice)) ||
        (e = cudaMemcpy(c->iwp, hp.iwp.data(), tb, cudaMemcpyHostToDevice)) ||
        (e = cudaMemcpy(c->fwi, hp.fwi.data(), 2 * tb, cudaMemcpyHostToDevice)) ||
        (e = cudaMemcpy(c->iwi, hp.iwi.data(), 2 * tb, cudaMemcpyHostToDevice)) ||
        (e = cudaMemcpy(c->wm, wmask.data(), wmask.size() * 4, cudaMemcpyHostToDevice)) ||
        (e = cudaMemcpy(c->vm, vmask.data(), vmask.size() * 4, cudaMemcpyHostToDevice)) ||
        (e = ipr::make_pack_map(&c->tm_bt, c->bt, max_sets)) || (e = ipr::make_pack_map(&c->tm_btb, c->btb, max_sets)) ||
        (e = ipr::init_device_kernels()) || (e = ipr::set_constants(hp.barrett, hp.q0_inv_mod_q1)) ||
        (e = cudaFuncSetAttribute(ipr::k_off_jntt<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, ipr::JNTT_SMEM)) ||
        (e = ipr::collapse_attributes())) {
        ipr_inspiring_destroy(c);
        return ipr::cuda_fail(e, "ipr_inspiring_create");
    }
    *c->h_err = 0;
    *out = c;
    return IPR_OK;
}

int ipr_inspiring_pack(ipr_inspiring* c, int sets, const uint64_t* d_lwe, const uint64_t* d_y_body,
                       const uint64_t* d_z_body, uint64_t* d_out, void* stream) {
    if (!c || !d_lwe || !d_y_body || !d_z_body || !d_out || sets < 1 || sets > c->max_sets) {
        ipr::set_last_error("ipr_inspiring_pack: null argument or sets outside [1, max_sets]");
        return IPR_E_ARGS;
    }
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return ipr::cuda_fail(e, "set device");
    int st0 = inspiring_error(c);
    if (st0) return st0;
    using namespace ipr;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int coll_smem = (int)sizeof(CollapseSmem);
    const uint2* fwi = reinterpret_cast<uint2*>(c->fwi);
    const dim3 lwe_grid(N / HCOLS, (unsigned)sets, 2);
    if (reinterpret_cast<uintptr_t>(d_lwe) % 32 == 0) k_lwe_prep<true><<<lwe_grid, 256, 0, st>>>(d_lwe, sets, fwi, c->act);
    else k_lwe_prep<false><<<lwe_grid, 256, 0, st>>>(d_lwe, sets, fwi, c->act);
    k_off_jntt<true><<<dim3(N / JS, (unsigned)sets, 2), 256, JNTT_SMEM, st>>>(c->act, sets, fwi, c->F);
    launch_collapse(c->F, 0, sets, c->wm, reinterpret_cast<uint2*>(c->fwi), reinterpret_cast<uint2*>(c->iwi), c->bt,
                    c->btb, c->r0, c->xb, c->d_err, c->sm_count, st);
    k_off_finish<<<(unsigned)sets, 512, coll_smem, st>>>(c->r0, c->xb, 0, c->vm, c->fw, c->fwp, c->iw, c->iwp, c->bth,
                                                         c->a_hat);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "offline kernels");
    if ((e = launch_pack(&c->tm_bt, &c->tm_btb, c->bth, d_y_body, d_z_body, c->S, sets, c->sm_count, c->d_err, st)) != cudaSuccess ||
        (e = launch_intt_crt(c->S, c->iw, c->iwp, c->R, sets, st)) != cudaSuccess)
        return cuda_fail(e, "online kernels");
    k_inspiring_out<<<148, 256, 0, st>>>(c->a_hat, c->R, d_lwe, sets, d_out);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "output");
    return IPR_OK;
}

int ipr_inspiring_sync(ipr_inspiring* c, void* stream) {
    if (!c) {
        ipr::set_last_error("ipr_inspiring_sync: null context");
        return IPR_E_ARGS;
    }
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return ipr::cuda_fail(e, "set device");
    if ((e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream))) != cudaSuccess) return ipr::cuda_fail(e, "run");
    return inspiring_error(c);
}

int ipr_debug_inspiring_error(ipr_inspiring* c, int code) {
    if (!c || !code) return IPR_E_ARGS;
    __atomic_store_n(c->h_err, code, __ATOMIC_RELEASE);
    return IPR_OK;
}

}  // extern "C"
