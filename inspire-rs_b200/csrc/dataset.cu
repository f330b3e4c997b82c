// dataset.cu — DatasetGenerator on the GPU: seeded ML-KEM public keys and their IDs.
//
// Restates (rkdud007/inspire-rs) DatasetGenerator::generate_record
// (src/dataset/generator.rs:171-193): record idx of a dataset with seed `seed` is
//   seed64 = ChaCha20Rng::seed_from_u64(seed) keystream at word position 16 * idx: one
//            64-byte ChaCha20 block, counter idx (rand_chacha: 64-bit counter in words
//            12-13, stream id 0 in words 14-15),
//   pk     = the encapsulation key of KemCore::generate_deterministic(d, z) with
//            d = seed64[0..32], z = seed64[32..64] (src/dataset/kem.rs:27-44): FIPS 203
//            ML-KEM.KeyGen_internal, whose ek = K-PKE.KeyGen(d).ek depends on d only,
//   id     = SHA3-256("pq-key:v1:" || kem_name || pk) (src/dataset/dataset.rs:36-46).
// Output rows are id (32 bytes) || pk (384 k + 32 bytes), the reference's flat record
// layout (generator.rs:101-118).  The ChaCha20 key (rand_core's seed_from_u64: PCG32 words)
// is derived on the host.  Keccak-f[1600] round constants and rotation offsets come from
// FIPS 202's definitions (the rc(t) LFSR, the (t+1)(t+2)/2 rho offsets).
//
// Two kernels.  k_dataset_keys gives each SHAKE stream of a record (k^2 matrix entries, 2k noise
// polynomials) a thread of its own with the Keccak state in registers, collects the sampled
// polynomials of a few records in shared memory, and transforms and multiplies them there a
// warp per polynomial; k_dataset_ids hashes one record per thread.  Both are bound by Keccak
// instruction issue (ALU pipe 81% busy): 20,000 ML-KEM-768 records 0.52 ms,
// against 2.85 ms for one thread per record with its sponge in local memory.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "ipr_b200.h"
#include "kernels.cuh"

namespace ipr {

namespace {

constexpr int MQ = 3329;

// FIPS 202 Algorithm 5, bit i of r holds R[i]
constexpr int rc_bit(int t) {
    if (t % 255 == 0) return 1;
    unsigned r = 1;
    for (int i = 1; i <= t % 255; i++) {
        r <<= 1;
        r ^= ((r >> 8) & 1) * 0x71u;
        r &= 0xFF;
    }
    return r & 1;
}
constexpr int brv7(int x) {
    int r = 0;
    for (int i = 0; i < 7; i++) r |= ((x >> i) & 1) << (6 - i);
    return r;
}
constexpr int pow17(int e) {
    int r = 1, b = 17;
    for (; e; e >>= 1, b = b * b % MQ)
        if (e & 1) r = r * b % MQ;
    return r;
}
struct KeccakTable {
    uint64_t rc[24];
};
constexpr KeccakTable keccak_table() {
    KeccakTable t{};
    for (int ir = 0; ir < 24; ir++)
        for (int j = 0; j <= 6; j++)
            if (rc_bit(j + 7 * ir)) t.rc[ir] |= 1ull << ((1 << j) - 1);
    return t;
}
struct MlkemTable {
    uint16_t zeta[128], gamma[128];  // 17^BitRev7(i), 17^(2 BitRev7(i) + 1) mod 3329
};
constexpr MlkemTable mlkem_table() {
    MlkemTable t{};
    for (int i = 0; i < 128; i++) {
        t.zeta[i] = (uint16_t)pow17(brv7(i));
        t.gamma[i] = (uint16_t)pow17(2 * brv7(i) + 1);
    }
    return t;
}
__constant__ KeccakTable c_keccak = keccak_table();
__device__ const MlkemTable d_mlkem = mlkem_table();

__host__ __device__ constexpr int rho_offset(int x, int y) {  // FIPS 202 Algorithm 2
    if (x == 0 && y == 0) return 0;
    int cx = 1, cy = 0;
    for (int t = 0; t < 24; t++) {
        if (cx == x && cy == y) return ((t + 1) * (t + 2) / 2) % 64;
        const int nx = cy, ny = (2 * cx + 3 * cy) % 5;
        cx = nx;
        cy = ny;
    }
    return 0;
}

__device__ __forceinline__ uint64_t rotl64(uint64_t v, int n) { return n ? (v << n) | (v >> (64 - n)) : v; }

__device__ __forceinline__ void keccakf(uint64_t (&a)[25]) {
#pragma unroll 1
    for (int ir = 0; ir < 24; ir++) {
        uint64_t c[5], d[5], b[25];
#pragma unroll
        for (int x = 0; x < 5; x++) c[x] = a[x] ^ a[x + 5] ^ a[x + 10] ^ a[x + 15] ^ a[x + 20];
#pragma unroll
        for (int x = 0; x < 5; x++) d[x] = c[(x + 4) % 5] ^ rotl64(c[(x + 1) % 5], 1);
#pragma unroll
        for (int i = 0; i < 25; i++) a[i] ^= d[i % 5];
#pragma unroll
        for (int x = 0; x < 5; x++)
#pragma unroll
            for (int y = 0; y < 5; y++) b[y + 5 * ((2 * x + 3 * y) % 5)] = rotl64(a[x + 5 * y], rho_offset(x, y));
#pragma unroll
        for (int x = 0; x < 5; x++)
#pragma unroll
            for (int y = 0; y < 5; y++)
                a[x + 5 * y] = b[x + 5 * y] ^ (~b[(x + 1) % 5 + 5 * y] & b[(x + 2) % 5 + 5 * y]);
        a[0] ^= c_keccak.rc[ir];
    }
}

__device__ __forceinline__ uint32_t rotl32(uint32_t v, int n) { return (v << n) | (v >> (32 - n)); }

__device__ __forceinline__ void chacha20_block(const uint32_t key[8], uint64_t counter, uint32_t (&out)[16]) {
    uint32_t s[16], x[16];
    s[0] = 0x61707865u;
    s[1] = 0x3320646eu;
    s[2] = 0x79622d32u;
    s[3] = 0x6b206574u;
#pragma unroll
    for (int i = 0; i < 8; i++) s[4 + i] = key[i];
    s[12] = (uint32_t)counter;
    s[13] = (uint32_t)(counter >> 32);
    s[14] = 0;
    s[15] = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = s[i];
    auto qr = [&](int a, int b, int c, int d) {
        x[a] += x[b]; x[d] ^= x[a]; x[d] = rotl32(x[d], 16);
        x[c] += x[d]; x[b] ^= x[c]; x[b] = rotl32(x[b], 12);
        x[a] += x[b]; x[d] ^= x[a]; x[d] = rotl32(x[d], 8);
        x[c] += x[d]; x[b] ^= x[c]; x[b] = rotl32(x[b], 7);
    };
#pragma unroll 1
    for (int r = 0; r < 10; r++) {
        qr(0, 4, 8, 12); qr(1, 5, 9, 13); qr(2, 6, 10, 14); qr(3, 7, 11, 15);
        qr(0, 5, 10, 15); qr(1, 6, 11, 12); qr(2, 7, 8, 13); qr(3, 4, 9, 14);
    }
#pragma unroll
    for (int i = 0; i < 16; i++) out[i] = x[i] + s[i];
}

// x mod 3329 for x < 2^32: quotient by the high half of a product with floor(2^32 / 3329),
// which is at most one too small, and one correction
__device__ __forceinline__ uint32_t modq12(uint32_t x) {
    constexpr uint32_t INV = (uint32_t)((1ull << 32) / MQ);
    const uint32_t r = x - __umulhi(x, INV) * MQ;
    return min(r, r - MQ);
}

// One CTA: R records.  Its first MW warps run the K*K matrix streams of all records, the next NW
// warps the 2K noise streams, so that a warp's lanes take the same branch and the same number of
// permutations (3 or 4 against 1, or 2 for eta 3).
template <int K>
struct Keys {
    static constexpr int R = K == 2 ? 16 : (K == 3 ? 7 : 4);  // the matrix streams fill two warps
    static constexpr int MW = (R * K * K + 31) / 32, NW = (R * 2 * K + 31) / 32;
    static constexpr int THREADS = 32 * (MW + NW);
    static constexpr int STREAMS = K * K + 2 * K;
    static constexpr int ETA1 = K == 2 ? 3 : 2;
    static constexpr int LD = 258;              // halfwords per polynomial: an odd word count, no bank conflicts
    static constexpr int PK = 384 * K + 32, REC = 32 + PK;
    uint16_t poly[R][STREAMS][LD];              // A[i][j] (i * K + j), then s[0..K), e[0..K)
    uint64_t seed[R][8];                        // rho (4 words), sigma (4 words)
};

// eight coefficients of a polynomial in registers: layout B e = lane + 32 m, layout C
// e = 32 (lane / 4) + 4 m + lane % 4, layout D e = 8 lane + m, so that every butterfly of FIPS 203
// Algorithm 9 (NTT) pairs two registers
__device__ __forceinline__ void mlkem_ntt_warp(uint16_t* f, int lane) {
    uint32_t v[8];
    auto layer = [&](int dd, int shift, int base, auto e) {  // zeta index base + (e >> shift)
#pragma unroll
        for (int m = 0; m < 8; m++) {
            if (m & dd) continue;
            const uint32_t z = d_mlkem.zeta[base + (e(m) >> shift)];
            const uint32_t t = modq12(z * v[m + dd]);
            const uint32_t a = v[m], lo = a + t, hi = a + MQ - t;
            v[m] = min(lo, lo - MQ);
            v[m + dd] = min(hi, hi - MQ);
        }
    };
    auto eb = [&](int m) { return lane + 32 * m; };
    auto ec = [&](int m) { return 32 * (lane >> 2) + 4 * m + (lane & 3); };
    auto ed = [&](int m) { return 8 * lane + m; };
#pragma unroll
    for (int m = 0; m < 8; m++) v[m] = f[eb(m)];
    layer(4, 8, 1, eb);  // length 128
    layer(2, 7, 2, eb);
    layer(1, 6, 4, eb);
#pragma unroll
    for (int m = 0; m < 8; m++) f[eb(m)] = (uint16_t)v[m];
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 8; m++) v[m] = f[ec(m)];
    layer(4, 5, 8, ec);  // length 16
    layer(2, 4, 16, ec);
    layer(1, 3, 32, ec);
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 8; m++) f[ec(m)] = (uint16_t)v[m];
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 8; m++) v[m] = f[ed(m)];
    layer(2, 2, 64, ed);  // length 2
#pragma unroll
    for (int m = 0; m < 8; m++) f[ed(m)] = (uint16_t)v[m];
}

template <int K>
__global__ void __launch_bounds__(Keys<K>::THREADS, 4)
    k_dataset_keys(uint4 key_lo, uint4 key_hi, uint64_t first, uint64_t count, uint8_t* __restrict__ out, bool words) {
    using C = Keys<K>;
    extern __shared__ __align__(16) uint8_t ds_smem[];
    C& sm = *reinterpret_cast<C*>(ds_smem);
    const int t = threadIdx.x, lane = t & 31;
    const uint64_t rec0 = (uint64_t)blockIdx.x * C::R;
    const int live = (int)min((uint64_t)C::R, count - rec0);
    if (t < live) {
        // record seed: ChaCha20 block number first + record; its first half is d
        const uint32_t key[8] = {key_lo.x, key_lo.y, key_lo.z, key_lo.w, key_hi.x, key_hi.y, key_hi.z, key_hi.w};
        uint32_t blk[16];
        chacha20_block(key, first + rec0 + t, blk);
        // K-PKE.KeyGen (FIPS 203 Algorithm 13): (rho, sigma) = SHA3-512(d || k)
        uint64_t a[25];
#pragma unroll
        for (int i = 0; i < 25; i++) a[i] = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = (uint64_t)blk[2 * i] | ((uint64_t)blk[2 * i + 1] << 32);
        a[4] = (uint64_t)K | (0x06ull << 8);
        a[8] = 0x80ull << 56;  // byte 71, the last of the 72-byte rate
        keccakf(a);
#pragma unroll
        for (int i = 0; i < 8; i++) sm.seed[t][i] = a[i];
    }
    __syncthreads();
    {
        const bool matrix = t < 32 * C::MW;
        const int u = matrix ? t : t - 32 * C::MW, per = matrix ? K * K : 2 * K;
        const int rec = u / per, st = matrix ? u % per : K * K + u % per;
        if (rec < live) {
            uint16_t* p = sm.poly[rec][st];
            uint64_t a[25];
#pragma unroll
            for (int i = 0; i < 25; i++) a[i] = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = sm.seed[rec][matrix ? i : 4 + i];
            if (matrix) {  // SampleNTT(SHAKE128(rho || j || i)) (Algorithm 7), rate 168
                a[4] = (uint64_t)(st % K) | ((uint64_t)(st / K) << 8) | (0x1Full << 16);
                a[20] = 0x80ull << 56;
            } else {       // SamplePolyCBD(SHAKE256(sigma || n)) (Algorithm 8), rate 136
                a[4] = (uint64_t)(st - K * K) | (0x1Full << 8);
                a[16] = 0x80ull << 56;
            }
            int have = 0;
            while (have < 256) {
                keccakf(a);
                if (matrix) {  // 21 words = 56 triples of bytes, two 12-bit candidates each
#pragma unroll
                    for (int g = 0; g < 7; g++) {
                        const uint64_t w0 = a[3 * g], w1 = a[3 * g + 1], w2 = a[3 * g + 2];
#pragma unroll
                        for (int c = 0; c < 16; c++) {
                            constexpr int B = 12;
                            const int bit = B * c, w = bit >> 6, sh = bit & 63;
                            const uint64_t lo = w == 0 ? w0 : (w == 1 ? w1 : w2), hi = w == 0 ? w1 : w2;
                            const uint32_t v =
                                (uint32_t)(sh <= 52 ? lo >> sh : (lo >> sh) | (hi << (64 - sh))) & 0xFFFu;
                            if (v < MQ && have < 256) p[have++] = (uint16_t)v;
                        }
                    }
                } else if (C::ETA1 == 2) {  // 16 words, a nibble per coefficient
#pragma unroll
                    for (int w = 0; w < 16; w++) {
                        const uint64_t x = (a[w] & 0x5555555555555555ull) + ((a[w] >> 1) & 0x5555555555555555ull);
#pragma unroll
                        for (int c = 0; c < 16; c++) {
                            const uint32_t n = (uint32_t)(x >> (4 * c)) & 15u;
                            const uint32_t d = (n & 3u) + MQ - (n >> 2);
                            p[16 * w + c] = (uint16_t)min(d, d - MQ);
                        }
                    }
                    have = 256;
                } else {  // eta 3: six bits per coefficient; 136 bytes of the first block, 56 of the second
                    // coefficient c takes bits [6 c, 6 c + 6): 1088 bits of a block hold 181 and 2 bits
                    const int c0 = have;
                    auto put = [&](int c, uint32_t s6) {
                        const uint32_t x = (s6 & 1) + ((s6 >> 1) & 1) + ((s6 >> 2) & 1);
                        const uint32_t y = ((s6 >> 3) & 1) + ((s6 >> 4) & 1) + ((s6 >> 5) & 1);
                        const uint32_t d = x + MQ - y;
                        p[c] = (uint16_t)min(d, d - MQ);
                    };
                    if (c0 == 0) {
#pragma unroll
                        for (int c = 0; c < 181; c++) {
                            const int bit = 6 * c, w = bit >> 6, sh = bit & 63;
                            const uint64_t hi = a[w + 1 < 17 ? w + 1 : 16];
                            put(c, (uint32_t)(sh <= 58 ? a[w] >> sh : (a[w] >> sh) | (hi << (64 - sh))) & 63u);
                        }
                        p[181] = (uint16_t)(a[16] >> 62);  // the two bits that the next block completes
                        have = 181;
                    } else {
                        put(181, ((uint32_t)p[181] | ((uint32_t)a[0] << 2)) & 63u);
#pragma unroll
                        for (int c = 182; c < 256; c++) {
                            const int bit = 6 * c - 1088, w = bit >> 6, sh = bit & 63;
                            put(c, (uint32_t)(sh <= 58 ? a[w] >> sh : (a[w] >> sh) | (a[w + 1] << (64 - sh))) & 63u);
                        }
                        have = 256;
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int i = t >> 5; i < live * 2 * K; i += C::THREADS / 32)  // NTT of every s and e, a warp each
        mlkem_ntt_warp(sm.poly[i / (2 * K)][K * K + i % (2 * K)], lane);
    __syncthreads();
    // t_i = sum_j A_ij s_j + e_i (base-case products, Algorithms 11 and 12), four coefficient
    // pairs per thread, and ByteEncode_12 (Algorithm 5) of them: 12 bytes
    for (int i = t; i < live * K * 32; i += C::THREADS) {
        const int rec = i / (K * 32), row = i / 32 % K, p0 = (i % 32) * 4;
        uint32_t o[3] = {0, 0, 0};
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int p = p0 + u;
            const uint32_t gm = d_mlkem.gamma[p];
            const uint16_t* e = sm.poly[rec][K * K + K + row];
            uint32_t c0 = e[2 * p], c1 = e[2 * p + 1];
#pragma unroll
            for (int j = 0; j < K; j++) {
                const uint16_t *A = sm.poly[rec][row * K + j], *s = sm.poly[rec][K * K + j];
                const uint32_t a0 = A[2 * p], a1 = A[2 * p + 1], b0 = s[2 * p], b1 = s[2 * p + 1];
                c0 += a0 * b0 + modq12(a1 * b1) * gm;  // each below q^2, at most 8 q^2 + q
                c1 += a0 * b1 + a1 * b0;
            }
            const uint32_t w = modq12(c0) | (modq12(c1) << 12);  // 24 bits
            if (u == 0) o[0] = w;
            else if (u == 1) o[0] |= w << 24, o[1] = w >> 8;
            else if (u == 2) o[1] |= w << 16, o[2] = w >> 16;
            else o[2] |= w << 8;
        }
        uint8_t* dst = out + (rec0 + rec) * (uint64_t)C::REC + 32 + 384 * row + 3 * p0;
        if (words) {
#pragma unroll
            for (int w = 0; w < 3; w++) reinterpret_cast<uint32_t*>(dst)[w] = o[w];
        } else {
            for (int b = 0; b < 12; b++) dst[b] = (uint8_t)(o[b >> 2] >> (8 * (b & 3)));
        }
    }
    for (int i = t; i < live * 32; i += C::THREADS) {
        const int rec = i >> 5, b = i & 31;
        out[(rec0 + rec) * (uint64_t)C::REC + 32 + 384 * K + b] = (uint8_t)(sm.seed[rec][b >> 3] >> (8 * (b & 7)));
    }
}

// id = SHA3-256("pq-key:v1:" || kem_name || pk), one record per thread.  The prefix is 16 bytes
// and PART more (4 for "-512" and "-768", 5 for "-1024"), so message word 2 + n is made of pk words
// n - 1 and n; `words`: the records are 8-byte aligned.
template <int K>
__global__ void __launch_bounds__(128) k_dataset_ids(uint64_t count, uint8_t* __restrict__ out, bool words) {
    constexpr int PK = 384 * K + 32, REC = 32 + PK, PART = K == 4 ? 5 : 4;
    constexpr int PW = PK / 8;                       // pk words
    constexpr int MSG = 16 + PART + PK;              // message bytes
    constexpr int BLOCKS = MSG / 136 + 1;            // padding takes at least one byte
    const uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (r >= count) return;
    uint8_t* rec = out + r * (uint64_t)REC;
    const uint8_t* pk = rec + 32;
    auto word = [&](int n) -> uint64_t {
        if (words) return reinterpret_cast<const uint64_t*>(pk)[n];
        uint64_t v = 0;
        for (int b = 0; b < 8; b++) v |= (uint64_t)pk[8 * n + b] << (8 * b);
        return v;
    };
    auto chars = [](const char* s, int n) {
        uint64_t v = 0;
        for (int b = 0; b < n; b++) v |= (uint64_t)(uint8_t)s[b] << (8 * b);
        return v;
    };
    const char* tail = K == 2 ? "-512" : (K == 3 ? "-768" : "-1024");
    uint64_t carry = chars(tail, PART), a[25], m[17];
    int n = 0;  // next pk word
    // the next block's 17 message words, loaded while the previous block is permuted
    auto load = [&](int blk) {
#pragma unroll
        for (int i = 0; i < 17; i++) {
            if (i < 2 && blk == 0) m[i] = i ? chars(":ml-kem", 7) << 8 | '1' : chars("pq-key:v", 8);
            else m[i] = n < PW ? word(n++) : 0;
        }
    };
#pragma unroll
    for (int i = 0; i < 25; i++) a[i] = 0;
    load(0);
    int absorbed = 0;  // pk words absorbed
#pragma unroll 1
    for (int blk = 0; blk < BLOCKS; blk++) {
#pragma unroll
        for (int i = 0; i < 17; i++) {
            uint64_t x = m[i];
            if (i >= 2 || blk) {
                if (absorbed < PW) {
                    x = carry | (m[i] << (8 * PART));
                    carry = m[i] >> (64 - 8 * PART);
                } else {
                    x = absorbed == PW ? carry | (0x06ull << (8 * PART)) : 0;  // the last bytes and the domain byte
                }
                absorbed++;
            }
            if (i == 16 && blk == BLOCKS - 1) x ^= 0x80ull << 56;
            a[i] ^= x;
        }
        if (blk + 1 < BLOCKS) load(blk + 1);
        keccakf(a);
    }
    if (words) {
#pragma unroll
        for (int i = 0; i < 4; i++) reinterpret_cast<uint64_t*>(rec)[i] = a[i];
    } else {
        for (int b = 0; b < 32; b++) {
            uint64_t v = a[0];
            if (b >= 8) v = b >= 24 ? a[3] : (b >= 16 ? a[2] : a[1]);
            rec[b] = (uint8_t)(v >> (8 * (b & 7)));
        }
    }
}

template <int K>
cudaError_t launch_dataset(const uint32_t (&key)[8], uint64_t first, uint64_t count, uint8_t* d_records,
                           cudaStream_t st) {
    const uint4 lo = make_uint4(key[0], key[1], key[2], key[3]), hi = make_uint4(key[4], key[5], key[6], key[7]);
    const int smem = (int)sizeof(Keys<K>);
    cudaError_t e = cudaFuncSetAttribute(k_dataset_keys<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const bool words = reinterpret_cast<uintptr_t>(d_records) % 8 == 0;
    k_dataset_keys<K><<<(unsigned)((count + Keys<K>::R - 1) / Keys<K>::R), Keys<K>::THREADS, smem, st>>>(lo, hi, first, count,
                                                                                                    d_records, words);
    k_dataset_ids<K><<<(unsigned)((count + 127) / 128), 128, 0, st>>>(count, d_records, words);
    return cudaGetLastError();
}

// rand_core SeedableRng::seed_from_u64: PCG32 output words, little endian
void seed_from_u64(uint64_t state, uint32_t key[8]) {
    const uint64_t mul = 6364136223846793005ull, inc = 11634580027462260723ull;
    for (int w = 0; w < 8; w++) {
        state = state * mul + inc;
        const uint32_t xs = (uint32_t)(((state >> 18) ^ state) >> 27);
        const int rot = (int)(state >> 59);
        key[w] = rot ? (xs >> rot) | (xs << (32 - rot)) : xs;
    }
}

}  // namespace

void set_last_error(const char* msg);  // server.cu: the text ipr_last_error() returns

namespace {
int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return IPR_OK;
    set_last_error(cudaGetErrorString(e));
    return IPR_E_CUDA;
}
}  // namespace

}  // namespace ipr

extern "C" int ipr_dataset_generate(int device, int kem, uint64_t seed, uint64_t first, uint64_t count,
                                    uint8_t* d_records, void* stream) {
    const int k = kem == 512 ? 2 : (kem == 768 ? 3 : (kem == 1024 ? 4 : 0));
    if (!k) {
        ipr::set_last_error("ipr_dataset_generate: kem must be 512, 768 or 1024");
        return IPR_E_ARGS;
    }
    if (count == 0) return IPR_OK;
    if (!d_records) {
        ipr::set_last_error("ipr_dataset_generate: null output");
        return IPR_E_ARGS;
    }
    int st = ipr::cuda_status(cudaSetDevice(device));
    if (st) return st;
    const uint64_t blocks = (count + 3) / 4;
    if (blocks > 0x7fffffffull) {
        ipr::set_last_error("ipr_dataset_generate: count too large for one call");
        return IPR_E_ARGS;
    }
    uint32_t key[8];
    ipr::seed_from_u64(seed, key);
    auto cs = static_cast<cudaStream_t>(stream);
    const cudaError_t e = k == 2   ? ipr::launch_dataset<2>(key, first, count, d_records, cs)
                          : k == 3 ? ipr::launch_dataset<3>(key, first, count, d_records, cs)
                                   : ipr::launch_dataset<4>(key, first, count, d_records, cs);
    return ipr::cuda_status(e);
}

// the same records into host memory: a device buffer of one batch (at most 65,536 records)
// is filled and copied back batch by batch
extern "C" int ipr_dataset_generate_host(int device, int kem, uint64_t seed, uint64_t first, uint64_t count,
                                         uint8_t* h_records) {
    const uint64_t pk_len = kem == 512 ? 800 : (kem == 768 ? 1184 : (kem == 1024 ? 1568 : 0));
    if (!pk_len) {
        ipr::set_last_error("ipr_dataset_generate_host: kem must be 512, 768 or 1024");
        return IPR_E_ARGS;
    }
    if (count == 0) return IPR_OK;
    if (!h_records) {
        ipr::set_last_error("ipr_dataset_generate_host: null output");
        return IPR_E_ARGS;
    }
    int st = ipr::cuda_status(cudaSetDevice(device));
    if (st) return st;
    const uint64_t rs = 32 + pk_len, batch = count < 65536 ? count : 65536;
    uint8_t* d = nullptr;
    if (cudaMalloc(&d, batch * rs) != cudaSuccess) {
        cudaGetLastError();
        ipr::set_last_error("ipr_dataset_generate_host: cudaMalloc failed");
        return IPR_E_OOM;
    }
    for (uint64_t c0 = 0; c0 < count && !st; c0 += batch) {
        const uint64_t n = count - c0 < batch ? count - c0 : batch;
        st = ipr_dataset_generate(device, kem, seed, first + c0, n, d, nullptr);
        if (!st) st = ipr::cuda_status(cudaMemcpy(h_records + c0 * rs, d, n * rs, cudaMemcpyDeviceToHost));
    }
    cudaFree(d);
    return st;
}
