// encode.cu — setup-time database layout and encode on the GPU.
//
// k_raw_db:    KeywordCuckooTable::to_raw_db (rkdud007/inspire-rs
//              src/pir/keyword/cuckoo.rs:314-353): bucket entries (row-major bytes) ->
//              the column-major u16 raw DB, big-endian u16 per byte pair, zero for empty
//              buckets.
// k_encode<I>: gpu_encode_db (native/cuda/encode_kernel.cu:18-228, 264-386): per DB row
//              and fold group, the I = interp polynomials of columns wp*I*N + j*N + k are
//              interpolated by a radix-2 Cooley-Tukey pass over Z_65535[X]/(X^N + 1) with
//              monomial twiddles, then scaled by I^-1 mod 65535.
//
// B200 design.  Every twiddle X^e of the pass has e a multiple of S = 2N/I, so a shift
// moves whole chunks of S coefficients and keeps the offset o = k mod S: the pass
// splits into S independent sub-problems of I polynomials x I/2 chunks.  The first three
// levels stay inside sets of 8 polynomials x 4 chunks and the last two, after a fixed rotation
// of each polynomial, inside sets of 4 x 2, so a warp takes 64 DB rows of such a set in
// registers (32 words of two rows each per lane) and the values cross shared memory once
// between the two rounds: one HBM round trip for the whole encode where the reference makes
// one per level plus a gather and a scatter.
#include <cuda_runtime.h>

#include <cstdint>

#include "ipr_b200.h"
#include "ipr_device.cuh"

namespace ipr {
void set_last_error(const char* msg);

namespace {

constexpr int E_ROWS = 32;  // the row count is a multiple of this
constexpr uint32_t PMOD = 65535;

__device__ __forceinline__ uint32_t fold65535(uint32_t x) {
    uint32_t r = (x & 0xFFFFu) + (x >> 16);
    r = (r & 0xFFFFu) + (r >> 16);
    return r >= PMOD ? r - PMOD : r;
}

// raw[(item * ise + j) * db_rows + row] for bucket row * per + item, any entry size, row count
// and alignment; one CTA per (32 rows, item): the 32 entries are staged in shared memory
// byte by byte and written column-wise
__global__ void __launch_bounds__(256) k_raw_db(const uint8_t* __restrict__ entries,
                                                const uint8_t* __restrict__ occupied, int64_t num_buckets,
                                                int entry_size, int64_t db_rows, int64_t per,
                                                uint16_t* __restrict__ raw) {
    extern __shared__ uint8_t ent[];  // [32][stride]: an odd word count per row spreads the column reads
    const int stride = (entry_size + 3) / 4 * 4 + 4;
    const int64_t item = blockIdx.y;
    const int64_t row0 = (int64_t)blockIdx.x * 32;
    for (int i = threadIdx.x; i < 32 * entry_size; i += blockDim.x) {
        const int r = i / entry_size, byte = i % entry_size;
        const int64_t row = row0 + r, b = row * per + item;
        ent[r * stride + byte] = (row < db_rows && b < num_buckets && occupied[b]) ? entries[b * entry_size + byte] : 0;
    }
    __syncthreads();
    const int ise = entry_size / 2;
    for (int i = threadIdx.x; i < 32 * ise; i += blockDim.x) {
        const int r = i & 31, j = i >> 5;
        const int64_t row = row0 + r;
        if (row >= db_rows) continue;
        const uint16_t v = (uint16_t)(((uint16_t)ent[r * stride + 2 * j] << 8) | ent[r * stride + 2 * j + 1]);
        raw[(item * ise + j) * db_rows + row] = v;
    }
}

// The same for entries of 16-byte multiples (every entry of the ML-KEM tables) and rows of 8-row
// multiples, both buffers 16-byte aligned.  A transpose of 2-byte values, bound by HBM: one CTA
// moves RT_ROWS = 64 rows x RT_BYTES = 256 bytes of one item, reading each entry piece with
// 16-byte loads and writing full 128-byte lines of a column; the 16-byte pieces of a row group
// are XOR-swizzled so that neither side has bank conflicts.
// 250,000 ML-KEM-768 keys (305 MB of occupied entries in, 805 MB out): 244 us (4.6 TB/s), against
// about 1,760 us for the byte-wise form after clearing the whole output.
constexpr int RT_ROWS = 64, RT_BYTES = 256, RT_THREADS = 256;

__global__ void __launch_bounds__(RT_THREADS) k_raw_db_vec(const uint8_t* __restrict__ entries,
                                                           const uint8_t* __restrict__ occupied, int64_t num_buckets,
                                                           int entry_size, int64_t db_rows, int64_t per,
                                                           uint16_t* __restrict__ raw) {
    __shared__ __align__(16) uint32_t tile[RT_ROWS][RT_BYTES / 4];
    const int64_t row0 = (int64_t)blockIdx.x * RT_ROWS, item = blockIdx.y;
    const int byte0 = blockIdx.z * RT_BYTES;
    const int pieces = min(RT_BYTES, entry_size - byte0) / 16;  // 16-byte pieces of this chunk
    constexpr int PPR = RT_BYTES / 16;
    constexpr int LPT = RT_ROWS * PPR / RT_THREADS;
    uint4 v[LPT];
#pragma unroll
    for (int u = 0; u < LPT; u++) {
        const int i = threadIdx.x + u * RT_THREADS, r = i / PPR, c = i % PPR;
        const int64_t row = row0 + r, b = row * per + item;
        v[u] = make_uint4(0, 0, 0, 0);
        if (c < pieces && row < db_rows && b < num_buckets && __ldg(occupied + b))
            v[u] = __ldg(reinterpret_cast<const uint4*>(entries + b * entry_size + byte0) + c);
    }
#pragma unroll
    for (int u = 0; u < LPT; u++) {
        const int i = threadIdx.x + u * RT_THREADS, r = i / PPR, c = i % PPR;
        // big-endian 16-bit values
        const uint4 w = make_uint4(__byte_perm(v[u].x, 0, 0x2301), __byte_perm(v[u].y, 0, 0x2301),
                                   __byte_perm(v[u].z, 0, 0x2301), __byte_perm(v[u].w, 0, 0x2301));
        *reinterpret_cast<uint4*>(&tile[r][(c ^ (r >> 3)) * 4]) = w;
    }
    __syncthreads();
    // a thread takes 8 rows of one word (two columns)
    const int64_t col0 = item * (entry_size / 2) + byte0 / 2;
    for (int i = threadIdx.x; i < (RT_ROWS / 8) * pieces * 4; i += RT_THREADS) {
        const int rg = i & 7, w = i >> 3;
        const int64_t row = row0 + rg * 8;
        if (row >= db_rows) continue;
        uint32_t x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = tile[rg * 8 + k][w ^ (rg * 4)];
        uint16_t* dst = raw + (col0 + 2 * w) * db_rows + row;
        *reinterpret_cast<uint4*>(dst) = make_uint4(__byte_perm(x[0], x[1], 0x5410), __byte_perm(x[2], x[3], 0x5410),
                                                    __byte_perm(x[4], x[5], 0x5410), __byte_perm(x[6], x[7], 0x5410));
        *reinterpret_cast<uint4*>(dst + db_rows) =
            make_uint4(__byte_perm(x[0], x[1], 0x7632), __byte_perm(x[2], x[3], 0x7632),
                       __byte_perm(x[4], x[5], 0x7632), __byte_perm(x[6], x[7], 0x7632));
    }
}

// interp = 1: the pass is empty, the scale is 1: values reduced mod 65535
__global__ void k_encode_scale1(const uint16_t* __restrict__ in, uint16_t* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (uint16_t)fold65535(in[i]);
}

constexpr int E_THREADS = 256, E_TILE = 64;  // 8 warps, 64 DB rows (2 per lane)

// a + b * s on the multiply pipe: `s` is a kernel argument (1 or -1), so that the sums do not
// compete with the shifts, permutes and minima for the ALU pipe
__device__ __forceinline__ uint32_t e_add(uint32_t a, uint32_t b, uint32_t s) { return a + b * s; }

// one radix-G pass (G a power of two) over G positions x G/2 ring elements, two unpacked rows:
// level lv pairs positions ev, ev + 2^lv, the second one turned by G t / 2^(lv+1) elements of a ring in
// which element G/2 is minus element 0.  Signed sums: below 65536 G in magnitude.
template <int G>
__device__ __forceinline__ void e_radix(uint32_t (&lo)[G][G > 1 ? G / 2 : 1], uint32_t (&hi)[G][G > 1 ? G / 2 : 1],
                                        uint32_t one, uint32_t minus) {
    constexpr int M = G > 1 ? G / 2 : 1;
#pragma unroll
    for (int half = 1; half < G; half *= 2) {
#pragma unroll
        for (int ev = 0; ev < G; ev++) {
            if (ev & half) continue;
            const int od = ev + half, t = ev % half;
            uint32_t a[M], b[M];
#pragma unroll
            for (int m = 0; m < M; m++) a[m] = lo[od][m], b[m] = hi[od][m];
#pragma unroll
            for (int m = 0; m < M; m++) {
                const int src = (m + G * t / (2 * half)) % G;
                const uint32_t x = lo[ev][m], y = hi[ev][m], u = a[src % M], v = b[src % M];
                const uint32_t s = src >= M ? minus : one, d = src >= M ? one : minus;
                lo[ev][m] = e_add(x, u, s);
                lo[od][m] = e_add(x, u, d);
                hi[ev][m] = e_add(y, v, s);
                hi[od][m] = e_add(y, v, d);
            }
        }
    }
}

// x mod 65535, canonical, for a signed x of magnitude below 65536 G, G <= 8
template <int G>
__device__ __forceinline__ uint32_t e_mod(uint32_t x, uint32_t one) {
    const uint32_t y = x + one * (G * PMOD);         // below 2^20; on the multiply pipe
    const uint32_t f = y - (y >> 16) * PMOD;         // (y mod 2^16) + (y >> 16) <= 65535 + 15
    return __viaddmin_u32(f, 0u - PMOD, f);          // f - 65535 wraps above f when f < 65535
}
template <int G>
__device__ __forceinline__ uint32_t e_pack(uint32_t lo, uint32_t hi, uint32_t one) {
    return __byte_perm(e_mod<G>(lo, one), e_mod<G>(hi, one), 0x5410);
}

// both canonical halves times 2^K mod 65535: a rotation of the 16 bits (never all ones)
template <int K>
__device__ __forceinline__ uint32_t e_scale(uint32_t w) {
    constexpr uint32_t HI = ((0xFFFFu << K) & 0xFFFFu) * 0x10001u;
    return ((w << K) & HI) | ((w >> (16 - K)) & ~HI);
}

// I = 32: a CTA takes one offset o, each warp two sets of the first round and eight of the second;
// I = 16: two offsets; I <= 8: an offset per warp, no second round.
// Bound by integer issue (ALU pipe 66-80% busy), hence the sums on the multiply pipe and the second
// round's chunk table.  250,000 ML-KEM-768 keys (interp 32, 1.6 GB): 414 us (3.9 TB/s) against
// 508 us for packed sums with a pass over shared memory per level; interp 8: 33 against 61 us
// at 16,384 columns.
template <int I>
__global__ void __launch_bounds__(E_THREADS, I > 8 ? 3 : 2) k_encode(const uint16_t* __restrict__ in, uint16_t* __restrict__ out,
                                                         int64_t db_rows, uint32_t one, uint32_t minus) {
    constexpr int H = I / 2;      // chunks of S coefficients in [0, N)
    constexpr int S = 2 * N / I;  // coefficient stride between chunks
    constexpr int LOGI = I == 2 ? 1 : I == 4 ? 2 : I == 8 ? 3 : I == 16 ? 4 : 5;
    constexpr int G = I < 8 ? I : 8, M = G / 2, G2 = I / G, M2 = G2 > 1 ? G2 / 2 : 1;
    constexpr int C1 = I / G;               // chunk step of the first round's sets
    constexpr int SETS1 = G2 * C1;          // per offset
    constexpr int SETS2 = G * (H / M2);
    constexpr int OFFS = 8 / SETS1 > 0 ? 8 / SETS1 : 1;  // offsets per CTA
    extern __shared__ uint32_t ebuf[];      // [offset][position][chunk][32 lanes]
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp-uniform
    const int64_t row0 = (int64_t)blockIdx.x * E_TILE + 2 * lane;
    const bool live = row0 < db_rows;
    const int64_t row = live ? row0 : db_rows - 2;  // lanes past the end read the last rows and store nothing
    const int64_t base = (int64_t)blockIdx.z * I * N + (int64_t)blockIdx.y * OFFS;  // first column
    auto at = [&](int off, int poly, int chunk) {  // byte offset of this lane's two rows
        return 2 * ((base + off + (int64_t)poly * N + (int64_t)chunk * S) * db_rows + row);
    };
    // within a set, every column is a compile-time number of quarter polynomials away: one 32 x 32 ->
    // 64-bit product (a quarter polynomial has 2^32 bytes at 2^22 rows; no memory holds 2^32 rows)
    const uint32_t rows = (uint32_t)db_rows;
    auto quarters = [&](int n) { return (uint64_t)rows * (uint32_t)(2 * (N / 4) * n); };
    const char* inb = reinterpret_cast<const char*>(in);
    char* outb = reinterpret_cast<char*>(out);
    for (int set = warp; set < OFFS * SETS1; set += E_THREADS / 32) {
        const int off = set / SETS1, grp = set % SETS1 / C1, c0 = set % C1;
        uint32_t w[G][M], lo[G][M], hi[G][M];
        // bit-reversed order: position grp * G + p holds polynomial brev(p) * G2 + brev(grp)
        const char* src = inb + at(off, G2 > 1 ? (int)(__brev((unsigned)grp) >> (32 - (LOGI - 3))) : 0, c0);
#pragma unroll
        for (int p = 0; p < G; p++) {
            int bp = 0;
            for (int bit = 1, r = G / 2; bit < G; bit *= 2, r /= 2) bp += p & bit ? r : 0;
#pragma unroll
            for (int m = 0; m < M; m++)  // chunks C1 apart: N / M coefficients
                w[p][m] = __ldg(reinterpret_cast<const uint32_t*>(src + quarters(bp * G2 * 4 + m * (4 / M))));
        }
#pragma unroll
        for (int p = 0; p < G; p++)
#pragma unroll
            for (int m = 0; m < M; m++) hi[p][m] = w[p][m] >> 16, lo[p][m] = w[p][m] - hi[p][m] * 65536u;
        e_radix<G>(lo, hi, one, minus);
        uint32_t* dst = ebuf + ((off * I + grp * G) * H + c0) * 32 + lane;
        char* od = outb + at(off, 0, c0);
#pragma unroll
        for (int p = 0; p < G; p++)
#pragma unroll
            for (int m = 0; m < M; m++) {
                const uint32_t r = e_pack<G>(lo[p][m], hi[p][m], one);
                if constexpr (G2 > 1) dst[(p * H + m * C1) * 32] = r;
                else if (live)
                    *reinterpret_cast<uint32_t*>(od + quarters(p * 4 + m * (4 / M))) = e_scale<16 - LOGI>(r);
            }
    }
    if constexpr (G2 > 1) {
        // chunk and sign of every value of the second round: {byte offset in the buffer, complement mask}
        uint2* tab = reinterpret_cast<uint2*>(ebuf + OFFS * I * H * 32);  // [t][chunk of the set][g][m]
        for (int i = threadIdx.x; i < SETS2 * G2 * M2; i += E_THREADS) {
            const int m = i % M2, g = i / M2 % G2, c0 = i / (M2 * G2) % (H / M2), t = i / (M2 * G2 * (H / M2));
            // the twiddles common to the set: X^-(S * shift) on position g * G + t
            const int shift = (g & 1) * (I * t / (2 * G)) + (g >> 1) * (I * t / (4 * G));
            const int c = (c0 + m * (H / 2) + shift) % I;
            tab[i] = make_uint2((uint32_t)(((g * G + t) * H + c % H) * 32 * 4), c >= H ? 0xFFFFFFFFu : 0u);  // X^N = -1
        }
        __syncthreads();
        for (int set = warp; set < OFFS * SETS2; set += E_THREADS / 32) {
            const int off = set / SETS2, t = set % SETS2 / (H / M2), c0 = set % (H / M2);
            uint32_t lo[G2][M2], hi[G2][M2];
            const char* buf = reinterpret_cast<const char*>(ebuf + off * I * H * 32 + lane);
            const uint2* tb = tab + set % SETS2 * (G2 * M2);
#pragma unroll
            for (int g = 0; g < G2; g++)
#pragma unroll
                for (int m = 0; m < M2; m++) {
                    const uint2 e = tb[g * M2 + m];
                    const uint32_t x = *reinterpret_cast<const uint32_t*>(buf + e.x) ^ e.y;
                    hi[g][m] = x >> 16;
                    lo[g][m] = x - hi[g][m] * 65536u;
                }
            e_radix<G2>(lo, hi, one, minus);
            char* od = outb + at(off, t, c0);
#pragma unroll
            for (int g = 0; g < G2; g++)
#pragma unroll
                for (int m = 0; m < M2; m++)
                    if (live)
                        *reinterpret_cast<uint32_t*>(od + quarters(g * G * 4 + m * 2)) =
                            e_scale<16 - LOGI>(e_pack<G2>(lo[g][m], hi[g][m], one));
        }
    }
}

template <int I>
cudaError_t launch_encode(const uint16_t* in, uint16_t* out, uint64_t db_rows, unsigned groups, cudaStream_t st) {
    constexpr int G = I < 8 ? I : 8, SETS1 = (I / G) * (I / G), OFFS = 8 / SETS1 > 0 ? 8 / SETS1 : 1;
    constexpr int smem = I > 8 ? OFFS * I * (I / 2) * 32 * 4 + G * (I / 2) * (I / G) * 8 : 0;  // values, then the table
    cudaError_t e = cudaFuncSetAttribute(k_encode<I>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)((db_rows + E_TILE - 1) / E_TILE), 2 * N / I / OFFS, groups);
    k_encode<I><<<grid, E_THREADS, smem, st>>>(in, out, (int64_t)db_rows, 1u, 0u - 1u);
    return cudaGetLastError();
}

int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return IPR_OK;
    set_last_error(cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? IPR_E_OOM : IPR_E_CUDA;
}

}  // namespace

// interp^-1 mod 65535 for interp a power of two (2^16 = 1 mod 65535)
uint32_t encode_num_inv(uint64_t interp) {
    uint32_t inv = 1;
    unsigned logi = 0;
    while ((1ull << logi) < interp) logi++;
    for (unsigned b = 0; b < (16 - logi) % 16; b++) inv = (inv * 2) % PMOD;
    return inv;
}

int encode_db_device(const uint16_t* d_raw, uint16_t* d_out, uint64_t db_rows, uint64_t db_cols, uint64_t interp,
                     cudaStream_t st) {
    if (!d_raw || !d_out || !interp || (interp & (interp - 1)) || interp > 32 || db_rows % E_ROWS ||
        db_cols % (interp * N) || (reinterpret_cast<uintptr_t>(d_raw) | reinterpret_cast<uintptr_t>(d_out)) % 16) {
        set_last_error("encode: interp must be a power of two <= 32, db_rows a multiple of 32, db_cols of "
                       "interp*2048, buffers 16-byte aligned");
        return IPR_E_ARGS;
    }
    if (d_raw == d_out) {
        set_last_error("encode: input and output must differ");
        return IPR_E_ARGS;
    }
    const uint64_t c = db_cols / (interp * N);
    if (c > 65535 || 2 * N / interp > 65535) {
        set_last_error("encode: shape too large for one launch");
        return IPR_E_ARGS;
    }
    if (interp == 1) {
        k_encode_scale1<<<148 * 8, 256, 0, st>>>(d_raw, d_out, (int64_t)(db_rows * db_cols));
    } else {
        cudaError_t e;
        switch (interp) {
            case 2: e = launch_encode<2>(d_raw, d_out, db_rows, (unsigned)c, st); break;
            case 4: e = launch_encode<4>(d_raw, d_out, db_rows, (unsigned)c, st); break;
            case 8: e = launch_encode<8>(d_raw, d_out, db_rows, (unsigned)c, st); break;
            case 16: e = launch_encode<16>(d_raw, d_out, db_rows, (unsigned)c, st); break;
            default: e = launch_encode<32>(d_raw, d_out, db_rows, (unsigned)c, st); break;
        }
        if (e != cudaSuccess) return cuda_status(e);
    }
    return cuda_status(cudaGetLastError());
}

int raw_db_device(const uint8_t* d_entries, const uint8_t* d_occupied, uint64_t num_buckets, uint64_t entry_size,
                  uint64_t db_rows, uint64_t db_cols, uint64_t per, uint16_t* d_raw, cudaStream_t st) {
    if (!d_entries || !d_occupied || !d_raw || entry_size < 2 || entry_size % 2 || entry_size > 6144 || !per ||
        per * (entry_size / 2) > db_cols || per > 65535) {
        set_last_error("cuckoo_to_raw_db: bad shape (entry size even and <= 6144, per * entry_size/2 <= db_cols)");
        return IPR_E_ARGS;
    }
    // every column of an item is written whole; the columns past the last item are zero
    const uint64_t used = per * (entry_size / 2) * db_rows, all = db_rows * db_cols;
    int st0 = used < all ? cuda_status(cudaMemsetAsync(d_raw + used, 0, (all - used) * sizeof(uint16_t), st)) : IPR_OK;
    if (st0) return st0;
    if (entry_size % 16 == 0 && db_rows % 8 == 0 &&
        (reinterpret_cast<uintptr_t>(d_entries) | reinterpret_cast<uintptr_t>(d_raw)) % 16 == 0) {
        const dim3 grid((unsigned)((db_rows + RT_ROWS - 1) / RT_ROWS), (unsigned)per,
                        (unsigned)((entry_size + RT_BYTES - 1) / RT_BYTES));
        k_raw_db_vec<<<grid, RT_THREADS, 0, st>>>(d_entries, d_occupied, (int64_t)num_buckets, (int)entry_size,
                                                  (int64_t)db_rows, (int64_t)per, d_raw);
        return cuda_status(cudaGetLastError());
    }
    const int smem = 32 * ((int)(entry_size + 3) / 4 * 4 + 4);
    st0 = cuda_status(cudaFuncSetAttribute(k_raw_db, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (st0) return st0;
    const dim3 grid((unsigned)((db_rows + 31) / 32), (unsigned)per);
    k_raw_db<<<grid, 256, smem, st>>>(d_entries, d_occupied, (int64_t)num_buckets, (int)entry_size, (int64_t)db_rows,
                                      (int64_t)per, d_raw);
    return cuda_status(cudaGetLastError());
}

}  // namespace ipr

extern "C" {

int ipr_encode_db(int device, const uint16_t* d_raw, uint16_t* d_encoded, uint64_t db_rows, uint64_t db_cols,
                  uint64_t interp, void* stream) {
    int st = ipr::cuda_status(cudaSetDevice(device));
    if (st) return st;
    return ipr::encode_db_device(d_raw, d_encoded, db_rows, db_cols, interp, static_cast<cudaStream_t>(stream));
}

int ipr_cuckoo_to_raw_db(int device, const uint8_t* d_entries, const uint8_t* d_occupied, uint64_t num_buckets,
                         uint64_t entry_size, uint64_t db_rows, uint64_t db_cols, uint64_t per, uint16_t* d_raw,
                         void* stream) {
    int st = ipr::cuda_status(cudaSetDevice(device));
    if (st) return st;
    return ipr::raw_db_device(d_entries, d_occupied, num_buckets, entry_size, db_rows, db_cols, per, d_raw,
                              static_cast<cudaStream_t>(stream));
}

}  // extern "C"
