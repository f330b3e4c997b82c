// ntt_lazy.cuh — the lazily reduced register NTTs of the dependent chains (the RGSW fold and
// the offline collapse): forward transforms of gadget digits (< 2^19) and inverse transforms
// of canonical values without the factor N^-1, on the register layouts of ntt_regs.cuh.
//
// The inverse transforms are Gentleman-Sande butterflies with the plain inverse twiddles;
// N^-1 is folded into their callers' operands.  Every reduction is a few conditional
// subtractions with the stated bounds, all below 16 q < 2^32.
#pragma once
#include <cstdint>

#include "ipr_device.cuh"
#include "ntt_regs.cuh"

namespace ipr {
namespace nttl {

constexpr int EPT = nttr::EPT;
using nttr::csub;
using nttr::eA;
using nttr::eB;

// x < 16q (< 2^32) to [0, 2q) by three conditional subtractions on the ALU pipe: the fold is
// bound by its integer multiplies, so these cost less than a Barrett reduction's two
__device__ __forceinline__ uint32_t red16(uint32_t x, uint32_t q) {
    return csub(csub(csub(x, 8 * q), 4 * q), 2 * q);
}

// forward butterfly by stage: MODE 0 leaves x unreduced (the bound grows by 2q), MODE 1
// first brings x (< 16q) to [0, 2q).  Outputs: x + w*y, x - w*y + 2q, w*y in [0, 2q).
template <int MODE>
__device__ __forceinline__ void fwd_b(uint32_t& x, uint32_t& y, uint32_t w, uint32_t wp, uint32_t q) {
    const uint32_t xx = MODE == 1 ? red16(x, q) : x;
    const uint32_t qn = shoup_lazy(y, w, wp, q);
    x = xx + qn;
    y = xx + 2 * q - qn;
}

// twiddle tables interleaved with their Shoup companions ([limb][N] of (w, wp)): one 8-byte
// load per twiddle, half the L1 requests of two separate tables.  The twiddle of element k of
// a thread is (1 << mm) + (e >> (11 - mm)) with e = hi + k * RS + lo in every layout: hi, the
// thread's part, is a multiple of 2^(11 - mm) at the stages run in that layout, and lo (the
// thread bits below the register stride RS) never carries into the shifted value.  So the
// index is the thread's base plus a compile-time constant, and the elements of one stage that
// share a twiddle share its load.  Layout A: hi = 0, RS = 256; B: hi = 256 w, RS = 32;
// C: hi = 256 w + 32 (l / 4), RS = 4; D: hi = 256 w + 8 l, RS = 1 (w = t / 32, l = t % 32).
template <int RS>
__device__ __forceinline__ int tw_idx(int mm, int hi, int k) {
    return (1 << mm) + (hi >> (11 - mm)) + ((k * RS) >> (11 - mm));
}

// the consecutive twiddles of a stage with register distance dd: 4 / dd of them (elements k that
// share k / (2 dd) share one), in one 8-, 16- or 32-byte load.  The first index is a multiple
// of their number, so the load is aligned.  HOIST lets the compiler move the loads above the
// exchanges' barriers: faster where registers are free (the four-CTA fold 181 -> 167 us, the
// batched NTT), slower where they are not (the collapse 5.21 -> 5.41 ms, two chains per SM 472 ->
// 507 us).
struct Tw4 {
    uint2 w[4];
};
template <int DD, int RS, bool HOIST>
__device__ __forceinline__ Tw4 load_tw(const uint2* __restrict__ tw, int mm, int hi) {
    const uint2* p = tw + tw_idx<RS>(mm, hi, 0);
    Tw4 r;
    if constexpr (DD == 4) {
        r.w[0] = __ldg(p);
    } else if constexpr (DD == 2) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(p));
        r.w[0] = make_uint2(a.x, a.y);
        r.w[1] = make_uint2(a.z, a.w);
    } else {
        if constexpr (HOIST)
            asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                : "=r"(r.w[0].x), "=r"(r.w[0].y), "=r"(r.w[1].x), "=r"(r.w[1].y), "=r"(r.w[2].x), "=r"(r.w[2].y),
                  "=r"(r.w[3].x), "=r"(r.w[3].y)
                : "l"(p));
        else
            asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=r"(r.w[0].x), "=r"(r.w[0].y), "=r"(r.w[1].x), "=r"(r.w[1].y), "=r"(r.w[2].x),
                           "=r"(r.w[2].y), "=r"(r.w[3].x), "=r"(r.w[3].y)
                         : "l"(p));
    }
    return r;
}

template <int P, int MODE, int DD, int RS, bool HOIST>
__device__ __forceinline__ void fstage(uint32_t (&v)[P][EPT], int mm, int hi, const uint2* __restrict__ tw, uint32_t q) {
    const Tw4 w = load_tw<DD, RS, HOIST>(tw, mm, hi);
#pragma unroll
    for (int k = 0; k < EPT; k++) {
        if (k & DD) continue;
#pragma unroll
        for (int p = 0; p < P; p++) fwd_b<MODE>(v[p][k], v[p][k + DD], w.w[k / (2 * DD)].x, w.w[k / (2 * DD)].y, q);
    }
}

// Team exchanges through xbuf.  The intra-warp transposes (B <-> C <-> D) use only the warp's
// own 256-word region of each polynomial and synchronise only the warp, so the cross-warp
// exchanges are fenced by where they write: A -> B stores into every warp's region, so a
// team barrier first lets every warp finish with its region; its loads read the warp's own
// region, which nothing else writes before the next such barrier.  B -> A stores into the
// warp's own region (no other warp reads it until the barrier) and loads from all regions,
// which nothing writes before the next A -> B barrier.
template <int P>
__device__ __forceinline__ void xchg_a2b(uint32_t (&v)[P][EPT], int t, uint32_t* xbuf, int bar) {
    nttr::group_bar(bar);
#pragma unroll
    for (int p = 0; p < P; p++)
#pragma unroll
        for (int m = 0; m < EPT; m++) xbuf[p * N + eA(t, m)] = v[p][m];
    nttr::group_bar(bar);
#pragma unroll
    for (int p = 0; p < P; p++)
#pragma unroll
        for (int m = 0; m < EPT; m++) v[p][m] = xbuf[p * N + eB(t, m)];
}

// XB < P: the buffer holds XB polynomials, moved XB at a time; a later chunk's stores wait at
// a team barrier for every warp to finish loading the previous chunk from this warp's region
template <int P, int XB = P>
__device__ __forceinline__ void xchg_b2a(uint32_t (&v)[P][EPT], int t, uint32_t* xbuf, int bar) {
#pragma unroll
    for (int c0 = 0; c0 < P; c0 += XB) {
        if (c0) nttr::group_bar(bar);
#pragma unroll
        for (int p = c0; p < c0 + XB && p < P; p++)
#pragma unroll
            for (int m = 0; m < EPT; m++) xbuf[(p - c0) * N + eB(t, m)] = v[p][m];
        nttr::group_bar(bar);
#pragma unroll
        for (int p = c0; p < c0 + XB && p < P; p++)
#pragma unroll
            for (int m = 0; m < EPT; m++) v[p][m] = xbuf[(p - c0) * N + eA(t, m)];
    }
}

// forward NTT of P gadget-digit polynomials (< 2^19) of one limb: layout A in, layout D out
// in [0, 2q), or below 10q with RAW; xbuf holds XP >= P polynomials of this team.  Bounds: after stage s <= 6 every
// value is below 2^19 + 2q (s + 1) <= 2^19 + 14q; stage 7 reduces x first (outputs < 4q);
// stages 8..10 add 2q each (< 10q < 2^32); one reduction at the end.
template <int P, bool HOIST = false, bool RAW = false>
__device__ __forceinline__ void forward_digits(uint32_t (&v)[P][EPT], int t, uint32_t* xbuf, int bar,
                                               const uint2* __restrict__ tw, uint32_t q) {
    const int l = t & 31, w = t >> 5;
    uint32_t* wb = xbuf + w * 256;
    const int hb = 256 * w, hc = 256 * w + 32 * (l >> 2), hd = 256 * w + 8 * l;
    fstage<P, 0, 4, 256, HOIST>(v, 0, 0, tw, q);
    fstage<P, 0, 2, 256, HOIST>(v, 1, 0, tw, q);
    fstage<P, 0, 1, 256, HOIST>(v, 2, 0, tw, q);
    xchg_a2b<P>(v, t, xbuf, bar);
    fstage<P, 0, 4, 32, HOIST>(v, 3, hb, tw, q);
    fstage<P, 0, 2, 32, HOIST>(v, 4, hb, tw, q);
    fstage<P, 0, 1, 32, HOIST>(v, 5, hb, tw, q);
    nttr::b_to_c<P>(v, l, wb);
    fstage<P, 0, 4, 4, HOIST>(v, 6, hc, tw, q);
    fstage<P, 1, 2, 4, HOIST>(v, 7, hc, tw, q);
    fstage<P, 0, 1, 4, HOIST>(v, 8, hc, tw, q);
    nttr::c_to_d<P>(v, l, wb);
    fstage<P, 0, 2, 1, HOIST>(v, 9, hd, tw, q);
    fstage<P, 0, 1, 1, HOIST>(v, 10, hd, tw, q);
    if constexpr (!RAW) {
#pragma unroll
        for (int p = 0; p < P; p++)
#pragma unroll
            for (int k = 0; k < EPT; k++) v[p][k] = red16(v[p][k], q);
    }
}

// Gentleman-Sande butterfly with a plain inverse twiddle: x + y, (x - y) * w.  Inputs below
// OFF * q; the difference is taken as x + OFF q - y (< 2 OFF q <= 16q < 2^32); the product
// lands in [0, 2q); the sum (< 2 OFF q <= 16q) is reduced to [0, 2q) when RED.
template <int OFF, bool RED>
__device__ __forceinline__ void inv_b(uint32_t& x, uint32_t& y, uint32_t w, uint32_t wp, uint32_t q) {
    const uint32_t s = x + y;
    const uint32_t d = x + OFF * q - y;
    x = RED ? red16(s, q) : s;
    y = shoup_lazy(d, w, wp, q);
}

// one inverse stage over 2 * PL polynomials: [0, PL) of limb 0, [PL, 2 PL) of limb 1
template <int PL, int OFF, bool RED, int DD, int RS>
__device__ __forceinline__ void istage(uint32_t (&v)[2 * PL][EPT], int mm, int hi, const uint2* __restrict__ iw) {
#pragma unroll
    for (int l = 0; l < 2; l++) {
        const Tw4 w = load_tw<DD, RS, false>(iw + l * N, mm, hi);
#pragma unroll
        for (int k = 0; k < EPT; k++) {
            if (k & DD) continue;
            const uint2 x = w.w[k / (2 * DD)];
#pragma unroll
            for (int p = l * PL; p < (l + 1) * PL; p++) inv_b<OFF, RED>(v[p][k], v[p][k + DD], x.x, x.y, l ? Q1 : Q0);
        }
    }
}

// N * INTT of 2 * PL canonical polynomials (PL per limb): layout D in, layout A canonical out;
// xbuf holds XB polynomials.  Value bounds entering each stage: q, 2q, 4q, 8q (then the sums
// are reduced), 2q, 4q, 8q (reduced), 2q, 4q, 8q (reduced), 2q; below 4q at the end.
template <int PL, int XB = 2 * PL>
__device__ __forceinline__ void inverse_limbs(uint32_t (&v)[2 * PL][EPT], int t, uint32_t* xbuf, int bar,
                                              const uint2* __restrict__ iw) {
    const int l = t & 31, w = t >> 5;
    uint32_t* wb = xbuf + w * 256;
    const int hb = 256 * w, hc = 256 * w + 32 * (l >> 2), hd = 256 * w + 8 * l;
    istage<PL, 1, false, 1, 1>(v, 10, hd, iw);
    istage<PL, 2, false, 2, 1>(v, 9, hd, iw);
    nttr::d_to_c<2 * PL, XB>(v, l, wb);
    istage<PL, 4, false, 1, 4>(v, 8, hc, iw);
    istage<PL, 8, true, 2, 4>(v, 7, hc, iw);
    istage<PL, 2, false, 4, 4>(v, 6, hc, iw);
    nttr::c_to_b<2 * PL, XB>(v, l, wb);
    istage<PL, 4, false, 1, 32>(v, 5, hb, iw);
    istage<PL, 8, true, 2, 32>(v, 4, hb, iw);
    istage<PL, 2, false, 4, 32>(v, 3, hb, iw);
    xchg_b2a<2 * PL, XB>(v, t, xbuf, bar);
    istage<PL, 4, false, 1, 256>(v, 2, 0, iw);
    istage<PL, 8, true, 2, 256>(v, 1, 0, iw);
    istage<PL, 2, false, 4, 256>(v, 0, 0, iw);
#pragma unroll
    for (int p = 0; p < 2 * PL; p++)
#pragma unroll
        for (int k = 0; k < EPT; k++) {
            const uint32_t q = p < PL ? Q0 : Q1;
            v[p][k] = csub(csub(v[p][k], 2 * q), q);
        }
}

// one inverse stage of P polynomials of one limb
template <int P, int OFF, bool RED, int DD, int RS, bool HOIST>
__device__ __forceinline__ void istage_limb(uint32_t (&v)[P][EPT], int mm, int hi, const uint2* __restrict__ iw,
                                            uint32_t q) {
    const Tw4 w = load_tw<DD, RS, HOIST>(iw, mm, hi);
#pragma unroll
    for (int k = 0; k < EPT; k++) {
        if (k & DD) continue;
#pragma unroll
        for (int p = 0; p < P; p++) inv_b<OFF, RED>(v[p][k], v[p][k + DD], w.w[k / (2 * DD)].x, w.w[k / (2 * DD)].y, q);
    }
}

// N * INTT of P canonical polynomials of one limb (iw: that limb's table): layout D in, layout
// A canonical out; the bounds of inverse_limbs
template <int P, bool HOIST = false>
__device__ __forceinline__ void inverse_polys(uint32_t (&v)[P][EPT], int t, uint32_t* xbuf, int bar,
                                              const uint2* __restrict__ iw, uint32_t q) {
    const int l = t & 31, w = t >> 5;
    uint32_t* wb = xbuf + w * 256;
    const int hb = 256 * w, hc = 256 * w + 32 * (l >> 2), hd = 256 * w + 8 * l;
    istage_limb<P, 1, false, 1, 1, HOIST>(v, 10, hd, iw, q);
    istage_limb<P, 2, false, 2, 1, HOIST>(v, 9, hd, iw, q);
    nttr::d_to_c<P>(v, l, wb);
    istage_limb<P, 4, false, 1, 4, HOIST>(v, 8, hc, iw, q);
    istage_limb<P, 8, true, 2, 4, HOIST>(v, 7, hc, iw, q);
    istage_limb<P, 2, false, 4, 4, HOIST>(v, 6, hc, iw, q);
    nttr::c_to_b<P>(v, l, wb);
    istage_limb<P, 4, false, 1, 32, HOIST>(v, 5, hb, iw, q);
    istage_limb<P, 8, true, 2, 32, HOIST>(v, 4, hb, iw, q);
    istage_limb<P, 2, false, 4, 32, HOIST>(v, 3, hb, iw, q);
    xchg_b2a<P>(v, t, xbuf, bar);
    istage_limb<P, 4, false, 1, 256, HOIST>(v, 2, 0, iw, q);
    istage_limb<P, 8, true, 2, 256, HOIST>(v, 1, 0, iw, q);
    istage_limb<P, 2, false, 4, 256, HOIST>(v, 0, 0, iw, q);
#pragma unroll
    for (int p = 0; p < P; p++)
#pragma unroll
        for (int k = 0; k < EPT; k++) v[p][k] = csub(csub(v[p][k], 2 * q), q);
}
template <bool HOIST = false>
__device__ __forceinline__ void inverse_one(uint32_t (&v)[EPT], int t, uint32_t* xbuf, int bar,
                                            const uint2* __restrict__ iw, uint32_t q) {
    inverse_polys<1, HOIST>(reinterpret_cast<uint32_t (&)[1][EPT]>(v), t, xbuf, bar, iw, q);
}

// the 8 consecutive words of layout D held by thread t (two 16-byte loads)
__device__ __forceinline__ void load_d8(uint32_t (&r)[EPT], const uint32_t* __restrict__ p) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(p)), b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
    r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
    r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
}

__device__ __forceinline__ uint32_t mul_canon(uint32_t x, uint32_t w, uint32_t wp, uint32_t q) {
    return csub(shoup_lazy(x, w, wp, q), q);
}

}  // namespace nttl
}  // namespace ipr
