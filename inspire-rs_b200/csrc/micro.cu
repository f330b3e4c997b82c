// micro.cu — kernel-level entry points over device buffers: batched negacyclic
// NTT / INTT of one CRT limb and batched NTT-domain Galois automorphisms.
//
// These are the building blocks respond() uses internally (ntt_forward /
// ntt_inverse, src/core/ntt.rs:111-160, 731-780 of rkdud007/inspire-rs; the
// rotation gather of native/cuda/rotation_kernel.cu:21-59 in the closed form
// of generate_automorph_tables_brute_force, src/pir/packing.rs:1423-1468),
// exposed on their own so they can be checked and timed in isolation.
// Polynomials are 2048 u64 coefficients (one limb, canonical residues), the
// reference's per-limb storage.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <vector>

#include "host_math.hpp"
#include "ipr_b200.h"
#include "ipr_device.cuh"
#include "ntt_lazy.cuh"
#include "ntt_regs.cuh"
#include "umma.cuh"

namespace ipr {
void set_last_error(const char* msg);

namespace {

// N^-1 mod q and its Shoup companion
struct LimbScale {
    uint32_t w, wp;
};

// 32 bytes of four 64-bit words whose high halves are zero
__device__ __forceinline__ void ld_words4(const uint64_t* p, uint32_t (&v)[4]) {
    asm volatile("{\n\t.reg .b32 h0, h1, h2, h3;\n\tld.global.v8.b32 {%0,h0,%1,h1,%2,h2,%3,h3}, [%4];\n\t}\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "l"(p));
}
__device__ __forceinline__ void st_words4(uint64_t* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.global.v8.b32 [%0], {%1,%5,%2,%5,%3,%5,%4,%5};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d), "r"(0)
                 : "memory");
}

// One CTA of 256 threads per polynomial, lazily reduced transforms (ntt_lazy.cuh).  The
// coefficient side is read or written in layout A (coalesced 8-byte accesses), the NTT side in
// layout D, where a thread's 8 consecutive words are two whole 32-byte sectors (WIDE: 32-byte
// aligned buffers; 8-byte accesses otherwise), so neither side passes through shared memory.
// Bound by HBM and, nearly as much, by the shared-memory exchanges; two or four polynomials per
// CTA share their twiddles but fill the last wave worse.  4096 / 1501 polynomials, out of
// L2: 28.2 / 13.8 us forward, 28.8 / 14.4 us inverse (4.7 TB/s), against 34 / 21 us for the
// canonical butterflies on four polynomials with both sides staged.
template <bool INVERSE, bool WIDE>
__global__ void __launch_bounds__(256, 6)
    k_ntt_limb(uint64_t* __restrict__ polys, uint32_t q, const uint2* __restrict__ tw, LimbScale ni) {
    __shared__ __align__(16) uint32_t xbuf[N];
    const int t = threadIdx.x;
    uint64_t* poly = polys + (int64_t)blockIdx.x * N;
    uint32_t v[1][nttr::EPT];
    if (INVERSE && WIDE) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t w[4];
            ld_words4(poly + 8 * t + 4 * h, w);
#pragma unroll
            for (int i = 0; i < 4; i++) v[0][4 * h + i] = w[i];
        }
    } else {
#pragma unroll
        for (int m = 0; m < nttr::EPT; m++) v[0][m] = (uint32_t)poly[INVERSE ? nttr::eD(t, m) : nttr::eA(t, m)];
    }
#pragma unroll
    for (int m = 0; m < nttr::EPT; m++) v[0][m] = nttr::canon(v[0][m], q);  // any input below 4q
    if (INVERSE) {
        nttl::inverse_polys<1, true>(v, t, xbuf, 1, tw, q);
#pragma unroll
        for (int m = 0; m < nttr::EPT; m++) poly[nttr::eA(t, m)] = nttl::mul_canon(v[0][m], ni.w, ni.wp, q);
    } else {
        nttl::forward_digits<1, true>(v, t, xbuf, 1, tw, q);  // inputs below q: below 15 q through stage 6
#pragma unroll
        for (int m = 0; m < nttr::EPT; m++) v[0][m] = nttr::csub(v[0][m], q);
        uint64_t* dst = poly + 8 * t;
        if (WIDE) {
            st_words4(dst, v[0][0], v[0][1], v[0][2], v[0][3]);
            st_words4(dst + 4, v[0][4], v[0][5], v[0][6], v[0][7]);
        } else {
#pragma unroll
            for (int m = 0; m < nttr::EPT; m++) dst[m] = v[0][m];
        }
    }
}

// count <= 2^36: launches of at most 2^30 polynomials
template <bool INVERSE>
void launch_ntt_limb(uint64_t* polys, int64_t count, uint32_t q, const uint2* tw, LimbScale ni, cudaStream_t st) {
    constexpr int64_t MOST = 1ll << 30;
    for (int64_t p0 = 0; p0 < count; p0 += MOST) {
        const unsigned blocks = (unsigned)std::min(MOST, count - p0);
        uint64_t* d = polys + p0 * N;
        if (reinterpret_cast<uintptr_t>(d) % 32 == 0) k_ntt_limb<INVERSE, true><<<blocks, 256, 0, st>>>(d, q, tw, ni);
        else k_ntt_limb<INVERSE, false><<<blocks, 256, 0, st>>>(d, q, tw, ni);
    }
}

// out[j][p][s] = in[p][auto_src(ks[j], s)]: a CTA stages one input polynomial in shared memory and
// writes its image under its share of the requested automorphisms (blockIdx.y with SPLIT, else
// all).  Bound by the writes.  Without SPLIT a polynomial is read by one CTA alone, before that CTA
// writes, so an output block may lie on the input; with SPLIT the two must not overlap.
// 256 polynomials under 64 automorphisms 45 us (6.1 TB/s); 64 under 64 15 us, against 37 us with a CTA
// per polynomial alone.  More CTAs per SM, eight unrolled stores or 32-byte stores of four slots
// measured 47.5 us at 256 x 64.
template <bool SPLIT>
__global__ void __launch_bounds__(256) k_automorph(const uint64_t* __restrict__ in, int64_t count,
                                                   const uint32_t* __restrict__ ks, int nk,
                                                   uint64_t* __restrict__ out) {
    __shared__ uint64_t poly[N];
    const int j0 = SPLIT ? (int)((int64_t)nk * blockIdx.y / gridDim.y) : 0;
    const int j1 = SPLIT ? (int)((int64_t)nk * (blockIdx.y + 1) / gridDim.y) : nk;
    for (int64_t p = blockIdx.x; p < count; p += gridDim.x) {
        __syncthreads();
        for (int s = threadIdx.x; s < N; s += blockDim.x) poly[s] = in[p * N + s];
        __syncthreads();
        for (int j = j0; j < j1; j++) {
            const uint32_t k = __ldg(ks + j);
            uint64_t* o = out + ((int64_t)j * count + p) * N;
            for (int s = threadIdx.x; s < N; s += blockDim.x) o[s] = poly[auto_src(k, (uint32_t)s)];
        }
    }
}

// The bounded waits that the kernels use on their mbarriers (umma::mbar_wait, and
// umma::mbar_wait_cluster for data from another CTA of the cluster), one after the other on a
// barrier nothing arrives on: each gives up after `limit_ns` of global time and the kernel reports
// it instead of hanging, as the kernels do through their error flags.  out: the waits that
// completed, a bit each.
__global__ void k_wait_selftest(uint64_t limit_ns, int* out) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        umma::mbar_init(&bar, 1);
        umma::fence_mbar_init();
    }
    __syncthreads();
    const bool done = umma::mbar_wait(&bar, 0, limit_ns);  // phase 0 never completes
    const bool cluster_done = umma::mbar_wait_cluster(&bar, 0, limit_ns);
    if (threadIdx.x == 0) *out = (done ? 1 : 0) | (cluster_done ? 2 : 0);
}

// per-device NTT tables (forward and plain inverse twiddles interleaved with their Shoup companions:
// [2][2 limbs][N] pairs), built on first use
std::mutex g_mu;
std::vector<uint2*> g_tables;

int tables_for(int device, const uint2** out) {
    std::lock_guard<std::mutex> lk(g_mu);
    if ((int)g_tables.size() <= device) g_tables.resize(device + 1, nullptr);
    uint2*& d = g_tables[device];
    if (!d) {
        HostParams hp;
        host_params_init(hp);
        std::vector<uint32_t> h(8 * N);
        std::copy(hp.fwi.begin(), hp.fwi.end(), h.begin());
        std::copy(hp.iwi.begin(), hp.iwi.end(), h.begin() + 4 * N);
        cudaError_t e = cudaMalloc(&d, h.size() * sizeof(uint32_t));
        if (e == cudaSuccess) e = cudaMemcpy(d, h.data(), h.size() * sizeof(uint32_t), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            if (d) cudaFree(d);
            d = nullptr;
            set_last_error(cudaGetErrorString(e));
            return e == cudaErrorMemoryAllocation ? IPR_E_OOM : IPR_E_CUDA;
        }
    }
    *out = d;
    return IPR_OK;
}

int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return IPR_OK;
    set_last_error(cudaGetErrorString(e));
    return IPR_E_CUDA;
}

}  // namespace

int ntt_tables(int device, const uint2** out) { return tables_for(device, out); }
}  // namespace ipr

extern "C" {

int ipr_ntt_batch(int device, uint64_t* d_polys, uint64_t count, int limb, int inverse, void* stream) {
    if (!d_polys || (limb != 0 && limb != 1) || count > (1ull << 36)) {
        ipr::set_last_error("ipr_ntt_batch: bad argument (null buffer, limb not 0/1, or too many polynomials)");
        return IPR_E_ARGS;
    }
    if (count == 0) return IPR_OK;
    int st = ipr::cuda_status(cudaSetDevice(device));
    if (st) return st;
    const uint2* tb;
    if ((st = ipr::tables_for(device, &tb))) return st;
    const int n = ipr::N;
    const uint32_t q = limb ? ipr::Q1 : ipr::Q0;
    const uint2* tw = tb + (inverse ? 2 * n : 0) + limb * n;
    const uint32_t w = q - (q - 1) / n;  // N^-1 mod q
    const ipr::LimbScale ni{w, (uint32_t)(((uint64_t)w << 32) / q)};
    auto cs = static_cast<cudaStream_t>(stream);
    const int64_t c = (int64_t)count;
    if (inverse) ipr::launch_ntt_limb<true>(d_polys, c, q, tw, ni, cs);
    else ipr::launch_ntt_limb<false>(d_polys, c, q, tw, ni, cs);
    return ipr::cuda_status(cudaGetLastError());
}

int ipr_automorph_batch(int device, const uint64_t* d_in, uint64_t count, const uint32_t* d_ks, int nk,
                        uint64_t* d_out, void* stream) {
    if (!d_in || !d_out || !d_ks || nk < 0 || count > (1ull << 36)) {
        ipr::set_last_error("ipr_automorph_batch: bad argument");
        return IPR_E_ARGS;
    }
    if (count == 0 || nk == 0) return IPR_OK;
    int st = ipr::cuda_status(cudaSetDevice(device));
    if (st) return st;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // fewer polynomials than two CTAs per SM are shared out by automorphism, unless the output overlaps
    // the input: another CTA could then have written a polynomial before it is read
    const uint64_t bytes = count * ipr::N * 8, in0 = reinterpret_cast<uintptr_t>(d_in),
                   out0 = reinterpret_cast<uintptr_t>(d_out);
    const bool overlap = in0 < out0 + bytes * (uint64_t)nk && out0 < in0 + bytes;
    const int64_t gx = std::min<int64_t>((int64_t)count, (int64_t)sms * 8);
    const int64_t share = overlap ? 1 : std::max<int64_t>((int64_t)sms * 2 / gx, 1);
    const int64_t gy = std::min<int64_t>(share, std::min(nk, 65535));
    const dim3 grid((unsigned)gx, (unsigned)gy);
    auto cs = static_cast<cudaStream_t>(stream);
    if (gy > 1) ipr::k_automorph<true><<<grid, 256, 0, cs>>>(d_in, (int64_t)count, d_ks, nk, d_out);
    else ipr::k_automorph<false><<<grid, 256, 0, cs>>>(d_in, (int64_t)count, d_ks, nk, d_out);
    return ipr::cuda_status(cudaGetLastError());
}

int ipr_device_binary_version(int device, int* binary_version) {
    if (!binary_version) return IPR_E_ARGS;
    int st = ipr::cuda_status(cudaSetDevice(device));
    if (st) return st;
    cudaFuncAttributes a{};
    st = ipr::cuda_status(cudaFuncGetAttributes(&a, ipr::k_wait_selftest));
    if (st) return st;
    *binary_version = a.binaryVersion;
    return IPR_OK;
}

int ipr_selftest_bounded_wait(int device, uint32_t limit_us) {
    if (limit_us == 0 || limit_us > 1000000u) {
        ipr::set_last_error("ipr_selftest_bounded_wait: limit_us must be in [1, 1000000]");
        return IPR_E_ARGS;
    }
    int st = ipr::cuda_status(cudaSetDevice(device));
    if (st) return st;
    int* d = nullptr;
    int h = -1;
    cudaError_t e = cudaMalloc(&d, sizeof(int));
    if (e == cudaSuccess) {
        ipr::k_wait_selftest<<<1, 32>>>((uint64_t)limit_us * 1000u, d);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(int), cudaMemcpyDeviceToHost);
        cudaFree(d);
    }
    if (e != cudaSuccess) return ipr::cuda_status(e);
    if (h == 0) {
        ipr::set_last_error("bounded wait ran out (self-test: nothing arrives on the barrier)");
        return IPR_E_TIMEOUT;
    }
    ipr::set_last_error("bounded wait self-test: the barrier completed unexpectedly");
    return IPR_E_STATE;
}

}  // extern "C"
