// pack_tc.cu — the InspiRING packing inner product for a batch of clients on
// the 5th-generation tensor cores.
//
// For output j, NTT slot z, limb l (packing_online_kernel.cu:18-92 /
// full_packing_with_preprocessing_online, src/pir/packing.rs:2941-3012):
//   S[c][j][l][z] = sum_{i<1023,k<3} y_c[k][rot_i(z)] T[j][i,k][z] + y_c[k][rotbar_i(z)] Tbar[j][i,k][z]
//                 + sum_k z_c[k][z] That[j][k][z]                          (mod q_l)
// The rotated slots rot_i(z) = auto_src(5^i, z) and rotbar_i(z) = auto_src(2N - 5^i, z)
// are distinct for every (i, kind) at a fixed z (5 generates a subgroup of the
// odd residues mod 2N that excludes -1), so re-indexing the precomputation by
// the slot it multiplies turns the client side into a z-independent matrix:
//   S[c][j][l][z] = sum_{k, s} Y_l[c][k*N + s] * Tpp_{z,l}[j][k*N + s]   (+ the z_body term,
//                   which k_intt_crt adds before its inverse NTT)
//   Y_l[c][k*N + s]      = y_c[k][s] (limb l)
//   Tpp_{z,l}[j][k*N+s]  = T[j][i,k][z] if s = rot_i(z), Tbar[j][i,k][z] if s = rotbar_i(z), else 0
// Tpp is built once at setup.  Both operands are split into bytes (28-bit
// residues = 4 bytes) so every term is a u8 x u8 product:
//   S = sum_{a,b} 256^(a+b) P_ab,  P_ab = sum_K Y_l,a[c][K] * Tpp_{z,l},b[j][K]
// with P_ab < 255^2 * 6144 < 2^29 exact in a 32-bit accumulator.
//
// The client matrix is the same for every slot, so the rows of the GEMM are all (j, z) pairs of
// a limb, densely packed: a tile is 32 consecutive slots of one output, 4 bytes b each,
//   row ((l * instances + j) * N + z) * 4 + b,
// M = 128 rows, N = 4 bytes a x clients (<= 256), K = 6144.  No output is padded, and the
// epilogue's writes of a client run along z.  Persistent CTAs of 18 warps: TMA producer, MMA
// issuer, 16 epilogue warps; each unit is two tiles that share the client operand.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "bounds.cuh"
#include "ipr_device.cuh"
#include "kernels.cuh"
#include "umma.cuh"

namespace ipr {

namespace {

constexpr int P_THREADS = 576;
constexpr int P_EPI_WARPS = 16;
constexpr int P_TILE_M = 128;
constexpr int P_TILE_K = 128;
constexpr int P_K = 3 * N;  // 6144
constexpr int P_A_STAGE = P_TILE_M * P_TILE_K;
constexpr int P_MAX_STAGES = 8;
constexpr int P_UNITS = N / 64;  // units (64 slots) per limb and output

struct PSmem {
    uint64_t full[P_MAX_STAGES], empty[P_MAX_STAGES], acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int err;
};

__device__ __forceinline__ uint32_t pow5(uint32_t i) {  // 5^i mod 2N
    uint32_t r = 1, b = 5;
    while (i) {
        if (i & 1) r = (r * b) & (2 * N - 1);
        b = (b * b) & (2 * N - 1);
        i >>= 1;
    }
    return r;
}

}  // namespace

// Tpp rows ((l * instances + j) * N + z) * 4 + b, columns k*N + s: byte b of limb l of T[j][i,k][z] at
// s = rot_i(z) and of Tbar[j][i,k][z] at s = rotbar_i(z); the two columns of i = 1023 (no such
// row) are 0.  One CTA scatters the 2046 precomputation rows of (j, k) at R_Z consecutive slots
// (64-byte pieces) into a byte tile in shared memory and writes it as whole 2 KB row
// segments.  grid (N / R_Z, instances, 3)
constexpr int R_Z = 8, R_THREADS = 512;
constexpr int R_SMEM = 2 * R_Z * 4 * N;

__global__ void __launch_bounds__(R_THREADS)
    k_relayout_tpp(const uint64_t* __restrict__ bt, const uint64_t* __restrict__ btb, uint8_t* __restrict__ tpp,
                   int instances) {
    extern __shared__ __align__(16) uint8_t rtile[];  // [2 limbs][R_Z][4 bytes][N]
    const int z0 = blockIdx.x * R_Z, j = blockIdx.y, k = blockIdx.z;
    for (int i = threadIdx.x; i < R_SMEM / 16; i += R_THREADS) reinterpret_cast<uint4*>(rtile)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const int zz = threadIdx.x % R_Z, z = z0 + zz;
    const uint32_t ez = exponent_of_slot((uint32_t)z);
    const int64_t base = ((int64_t)j * NINNER + k) * N + z;
    constexpr int STEP = R_THREADS / R_Z;
    uint32_t g = pow5(threadIdx.x / R_Z);
    const uint32_t g_step = pow5(STEP);
#pragma unroll 4
    for (int i = threadIdx.x / R_Z; i < NROT; i += STEP) {
        const uint64_t v[2] = {__ldg(bt + base + (int64_t)i * T_EXP * N), __ldg(btb + base + (int64_t)i * T_EXP * N)};
        const uint32_t s[2] = {slot_of_exponent((g * ez) & (2 * N - 1)),
                               slot_of_exponent(((2 * N - g) * ez) & (2 * N - 1))};
        g = (g * g_step) & (2 * N - 1);
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int l = 0; l < 2; l++) {
                const uint32_t limb = (uint32_t)(l ? (v[h] >> 32) : v[h]);
#pragma unroll
                for (int b = 0; b < 4; b++) rtile[((l * R_Z + zz) * 4 + b) * N + s[h]] = (uint8_t)(limb >> (8 * b));
            }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < R_SMEM / 16; c += R_THREADS) {
        const int r = c / (N / 16), seg = c % (N / 16);  // r = (l * R_Z + zz) * 4 + b
        const int l = r / (R_Z * 4), rb = r % (R_Z * 4);
        const int64_t row = (((int64_t)l * instances + j) * N + z0) * 4 + rb;
        *reinterpret_cast<uint4*>(tpp + row * P_K + k * N + seg * 16) = reinterpret_cast<const uint4*>(rtile)[c];
    }
}

// Y8[l][c*4 + a][k*N + s] = byte a of y_c[k][s] (limb l); rows c >= clients stay as zeroed
__global__ void k_build_y8(const uint64_t* __restrict__ y_bodies, uint8_t* __restrict__ y8, int clients, int np) {
    const int64_t total = (int64_t)clients * T_EXP * N;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(idx / (T_EXP * N));
        const int ks = (int)(idx % (T_EXP * N));  // k*N + s
        const uint64_t v = y_bodies[idx];
#pragma unroll
        for (int l = 0; l < 2; l++) {
            const uint32_t limb = (uint32_t)(l ? (v >> 32) : v);
#pragma unroll
            for (int a = 0; a < 4; a++) y8[((int64_t)l * np + c * 4 + a) * P_K + ks] = (uint8_t)(limb >> (8 * a));
        }
    }
}

// The 4x4 transpose of one register per lane within each group of 4 lanes: lane b (of the group)
// holds r[i] of column i and ends with r'[i] = the value lane i held in r[b].
__device__ __forceinline__ void transpose4(uint32_t (&r)[4], int lane) {
#pragma unroll
    for (int s = 1; s <= 2; s <<= 1) {
        const bool up = lane & s;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (i & s) continue;
            const uint32_t send = up ? r[i] : r[i + s];
            const uint32_t got = __shfl_xor_sync(0xffffffffu, send, s);
            if (up) r[i] = got;
            else r[i + s] = got;
        }
    }
}

// Each unit is two consecutive tiles (64 slots of one output and limb): both multiply the same
// Y_l K-slice, so every B stage feeds two MMAs and the client operand crosses L2 once per
// unit.  Accumulators: tile t at TMEM columns [buf * 2 nt + t nt, + nt).
// At full batches the accumulators fill TMEM (one buffer), so the epilogue runs while the ring
// prefetches but no MMA is issued: it has to fit in the ring's slack.  Sixteen warps drain it,
// two per tile and TMEM lane quarter: lane 4 zz + b holds byte b of slot zz, reduces the four
// a-byte columns of four clients, the 4 lanes of a slot transpose their residues with
// shuffles so that each finishes one client, and a client's stores cover whole sectors.
// 192 outputs (19.3 GB): 2.72 ms with 16 clients (7.1 TB/s), 3.61 ms with 64 (5.3 TB/s); 8 outputs
// with 7 clients 139 us, against 472 us when outputs were padded to tiles of 32 and 3.67 ms for a
// form on CTA pairs with four epilogue warps whose stores went to one sector per lane.
__global__ void __launch_bounds__(P_THREADS, 1)
    k_pack_mma(const __grid_constant__ CUtensorMap tm_t, const __grid_constant__ CUtensorMap tm_y, int instances,
               int clients, int np, int nt, int stages, uint32_t* __restrict__ S, int* __restrict__ err_flag) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((1024 - (umma::smem_addr(smem_raw) & 1023)) & 1023);
    PSmem* sh = reinterpret_cast<PSmem*>(base);
    volatile int* err = &sh->err;
    uint8_t* a_tiles = base + 1024;  // [stage][tile][128 x 128]
    const int b_stage = nt * P_TILE_K;
    uint8_t* b_tiles = a_tiles + stages * 2 * P_A_STAGE;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nbuf = (4 * nt <= 512) ? 2 : 1;
    uint32_t ncols = 32;
    while (ncols < (uint32_t)(nbuf * 2 * nt)) ncols <<= 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            umma::mbar_init(&sh->full[s], 1);
            umma::mbar_init(&sh->empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            umma::mbar_init(&sh->acc_full[b], 1);
            umma::mbar_init(&sh->acc_empty[b], P_EPI_WARPS);
        }
        *err = 0;
        umma::fence_mbar_init();
    }
    if (warp == 1) umma::tmem_alloc(&sh->tmem_base, ncols);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = sh->tmem_base;

    const int ks_total = P_K / P_TILE_K;              // 48
    const int64_t total = (int64_t)2 * instances * P_UNITS;  // units in row order: (l, j, 64 slots)

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int last_phase[P_MAX_STAGES];
            for (int s = 0; s < P_MAX_STAGES; s++) last_phase[s] = -1;
            for (int64_t u = blockIdx.x; u < total && !*err; u += gridDim.x) {
                const int arow = (int)(u * 2 * P_TILE_M);
                const int l = u >= total / 2;
                for (int ks = 0; ks < ks_total; ks++) {
                    if (!umma::mbar_wait(&sh->empty[stage], phase ^ 1)) {
                        *err = 11;
                        break;
                    }
                    uint8_t* at = a_tiles + stage * 2 * P_A_STAGE;
                    umma::mbar_expect_tx(&sh->full[stage], 2 * P_A_STAGE + b_stage);
                    umma::tma_load_2d(at, &tm_t, ks * P_TILE_K, arow, &sh->full[stage]);
                    umma::tma_load_2d(at + P_A_STAGE, &tm_t, ks * P_TILE_K, arow + P_TILE_M,
                                      &sh->full[stage]);
                    umma::tma_load_2d(b_tiles + stage * b_stage, &tm_y, ks * P_TILE_K, l * np, &sh->full[stage]);
                    last_phase[stage] = (int)phase;
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            for (int s = 0; s < stages; s++)
                if (last_phase[s] >= 0) umma::mbar_wait(&sh->full[s], (uint32_t)last_phase[s], umma::kDrainLimitNs);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma::idesc_u8(P_TILE_M, nt);
            int stage = 0, buf = 0, last_stage = -1;
            uint32_t phase = 0, acc_phase = 0, last_parity = 0;
            for (int64_t u = blockIdx.x; u < total && !*err; u += gridDim.x) {
                if (!umma::mbar_wait(&sh->acc_empty[buf], acc_phase ^ 1)) {
                    *err = 12;
                    break;
                }
                umma::fence_after();
                bool ok = true;
                const uint32_t d0 = tmem + (uint32_t)(buf * 2 * nt), d1 = d0 + (uint32_t)nt;
                for (int ks = 0; ks < ks_total; ks++) {
                    if (!umma::mbar_wait(&sh->full[stage], phase)) {
                        *err = 13;
                        ok = false;
                        break;
                    }
                    umma::fence_after();
                    const uint32_t sa = umma::smem_addr(a_tiles + stage * 2 * P_A_STAGE);
                    const uint32_t sb = umma::smem_addr(b_tiles + stage * b_stage);
#pragma unroll
                    for (int k4 = 0; k4 < P_TILE_K / 32; k4++) {
                        const uint64_t db = umma::desc_sw128(sb + 32 * k4);
                        const uint32_t acc = (ks == 0 && k4 == 0) ? 0u : 1u;
                        umma::mma_u8(d0, umma::desc_sw128(sa + 32 * k4), db, idesc, acc);
                        umma::mma_u8(d1, umma::desc_sw128(sa + P_A_STAGE + 32 * k4), db, idesc, acc);
                    }
                    umma::commit(&sh->empty[stage]);
                    last_stage = stage;
                    last_parity = phase;
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                umma::commit(&sh->acc_full[buf]);
                if (nbuf == 2) {
                    buf ^= 1;
                    if (buf == 0) acc_phase ^= 1;
                } else {
                    acc_phase ^= 1;
                }
            }
            if (last_stage >= 0) umma::mbar_wait(&sh->empty[last_stage], last_parity, umma::kDrainLimitNs);
        }
    } else {
        // epilogue warps 2..17: TMEM lane quarter = warp % 4 (8 slots x 4 bytes), tile t and half h of
        // the column groups (16 columns = 4 clients) by warp / 4
        const int quarter = warp & 3, t = ((warp - 2) >> 2) & 1, h = (warp - 2) >> 3;
        const int b = lane & 3;
        int buf = 0;
        uint32_t acc_phase = 0;
        const int groups = nt / 16;
        for (int64_t u = blockIdx.x; u < total; u += gridDim.x) {
            const bool got = umma::mbar_wait(&sh->acc_full[buf], acc_phase);
            if (!__all_sync(0xffffffffu, got)) {  // the warp stops together
                if (lane == 0) *err = 14;
                break;
            }
            umma::fence_after();
            const int l = u >= total / 2;
            const int64_t lj = u / P_UNITS;
            const int j = (int)(lj - (int64_t)l * instances);
            const int z = (int)(u % P_UNITS) * 64 + t * 32 + quarter * 8 + (lane >> 2);
            const uint32_t q = l ? Q1 : Q0;
            const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * 2 * nt + t * nt);
            uint32_t d[16];
            for (int g = h; g < groups; g += 2) {
                umma::tmem_ld16(taddr + (uint32_t)(g * 16), d);
                umma::tmem_wait_ld();
                if (g + 2 >= groups) {  // this warp's last TMEM read of the unit
                    umma::fence_before();
                    __syncwarp();
                    if (lane == 0) umma::mbar_arrive(&sh->acc_empty[buf]);
                }
                uint32_t r[4];  // client 4 g + i: sum_a 256^a P_ab mod q of this lane's byte b
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    uint64_t v = 0;
#pragma unroll
                    for (int a = 0; a < 4; a++) v += (uint64_t)d[i * 4 + a] << (8 * a);
                    r[i] = mod64m(v, q);
                }
                transpose4(r, lane);  // r[i] = byte i's residue of client 4 g + b
                const int c = 4 * g + b;
                // sum_b 256^b r_b < 2^28 * (1 + 2^8 + 2^16 + 2^24) < 2^53: one reduction.  The z_body x That
                // term is added by the kernel that consumes S.
                const uint64_t tot = (uint64_t)r[0] + ((uint64_t)r[1] << 8) + ((uint64_t)r[2] << 16) + ((uint64_t)r[3] << 24);
                if (c < clients) S[(((int64_t)c * instances + j) * 2 + l) * N + z] = mod64m(tot, q);
            }
            if (h >= groups) {  // a single column group: the second half's warps have nothing to read
                umma::fence_before();
                __syncwarp();
                if (lane == 0) umma::mbar_arrive(&sh->acc_empty[buf]);
            }
            if (nbuf == 2) {
                buf ^= 1;
                if (buf == 0) acc_phase ^= 1;
            } else {
                acc_phase ^= 1;
            }
        }
    }
    umma::fence_before();
    __syncthreads();
    if (warp == 1) umma::tmem_dealloc(tmem, ncols);
    if (threadIdx.x == 0 && *err) atomicExch(err_flag, *err);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
int pack_mma_nt(int clients) {
    int n = (4 * clients + 15) / 16 * 16;
    return n < 16 ? 16 : n;
}

int pack_mma_stages(int nt) {
    const int per = 2 * P_A_STAGE + nt * P_TILE_K;
    int s = (216 * 1024) / per;
    return s > P_MAX_STAGES ? P_MAX_STAGES : (s < 2 ? 2 : s);
}

size_t pack_mma_smem(int nt) {
    return 2048 + (size_t)pack_mma_stages(nt) * (2 * P_A_STAGE + nt * P_TILE_K);
}

cudaError_t init_pack_mma_kernel() {
    size_t mx = 0;  // the largest footprint over every client count the launcher can pick
    for (int nt = 16; nt <= 256; nt += 16) mx = pack_mma_smem(nt) > mx ? pack_mma_smem(nt) : mx;
    return cudaFuncSetAttribute(k_pack_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mx);
}

uint64_t tpp_bytes(int instances) { return (uint64_t)N * 2 * instances * 4 * P_K; }

cudaError_t launch_relayout_tpp(const uint64_t* bt, const uint64_t* btb, uint8_t* tpp, int instances,
                                cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(k_relayout_tpp, cudaFuncAttributeMaxDynamicSharedMemorySize, R_SMEM);
    if (e != cudaSuccess) return e;
    k_relayout_tpp<<<dim3(N / R_Z, instances, T_EXP), R_THREADS, R_SMEM, st>>>(bt, btb, tpp, instances);
    return cudaGetLastError();
}

cudaError_t launch_build_y8(const uint64_t* y_bodies, uint8_t* y8, int clients, int np, cudaStream_t st) {
    cudaError_t e;
    if ((e = check_extent(y_bodies, (uint64_t)clients * T_EXP * N * 8, "client operand: y bodies")) != cudaSuccess ||
        (e = check_extent(y8, (uint64_t)2 * np * P_K, "client operand: byte rows")) != cudaSuccess)
        return e;
    e = cudaMemsetAsync(y8, 0, (size_t)2 * np * P_K, st);
    if (e != cudaSuccess) return e;
    k_build_y8<<<148 * 4, 256, 0, st>>>(y_bodies, y8, clients, np);
    return cudaGetLastError();
}

cudaError_t launch_pack_mma(const CUtensorMap* tm_t, const CUtensorMap* tm_y, int instances, int clients, int np,
                            uint32_t* S, int* err_flag, int sm_count, cudaStream_t st) {
    const int nt = pack_mma_nt(clients);
    if (clients < 1 || clients > 64 || np < nt) return cudaErrorInvalidValue;
    cudaError_t e = check_extent(S, (uint64_t)clients * instances * 2 * N * 4, "packing: outputs");
    if (e != cudaSuccess) return e;
    const int64_t units = (int64_t)2 * instances * P_UNITS;
    const int grid = units < sm_count ? (int)units : sm_count;
    k_pack_mma<<<grid, P_THREADS, pack_mma_smem(nt), st>>>(*tm_t, *tm_y, instances, clients, np, nt,
                                                           pack_mma_stages(nt), S, err_flag);
    return cudaGetLastError();
}

}  // namespace ipr
