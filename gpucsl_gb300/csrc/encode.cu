// Ordinal encoding of discrete samples on the device (replaces the host OrdinalEncoder
// and the dims computation of gpucsl/pc/discover_skeleton_discrete.py:38-49): per
// column, the observed values in ascending order get codes 0..k-1 and dims = k.
//
// Integer-valued inputs (int32, int64, uint8, or float64 holding integers) whose column
// range is below ENC_RANGE are encoded in two passes over X, each over a grid of (32-column
// block, row chunk) tiles so that every SM streams its share with eight loads a thread in
// flight:
//   1. column minimum / maximum, integrality and the presence bitmap.  Value v has bit
//      v mod ENC_RANGE: distinct values of a column within the range have distinct bits
//      whatever the minimum turns out to be, so no earlier pass has to find it.  A tile whose
//      columns span at most 64 values each keeps bit v mod 64 in a register and spreads the
//      word when its minimum is known; other tiles go over their rows once more, into
//      bitmaps in shared memory;
//   2. codes = number of present values from the minimum up to the value, around the
//      circular bitmap: a popcount under a mask of one word where the block's columns span
//      at most 32 (or 64) values, otherwise the rank of the bit's word plus a popcount.
//      Transposed through shared memory into the column-major layout of the discrete solver
//      (column j at codes + j * ldc).  The first row chunk writes dims and the status.
// What bounds it: X is read twice (the second time partly from L2) and the codes written
// once.  n = 50000, p = 200, int64: 272 -> 78 us a call.  Three passes with four loads in
// flight, bitmaps of stride 128 words (every lane in one bank) and four memsets took that.
// A column with more than 255 distinct values, a wider range, or a non-integer value sets
// GCSL_ERR_UNSUPPORTED in the status word (bits and words are taken modulo their range, so
// nothing is read or written out of bounds whatever the values).
#include "common.cuh"

namespace gcsl {

constexpr int ENC_RANGE = 4096;  // values per column: min .. min + 4095
constexpr int ENC_WORDS = ENC_RANGE / 32;
// Tiles of at most this many rows have the bitmaps (words) and ranks (bytes) of pass 2 in shared
// memory at a pitch of 33 words and 36 bytes: loading and ranking them, word by word along a
// column, is then free of bank conflicts, and the rows' look-ups, at random words, share a bank
// three ways.  At 32 it is the other way round, which pays off over many rows.  Columns over 100
// values, int32, 33 against 32: 5000 x 1000 (192 rows) 97, 126 us; 50000 x 200 (448 rows) 87, 122;
// 50000 x 2000 (3648 rows) 509, 401.
constexpr int ENC_PAD_ROWS = 1024;
constexpr int ENC_STEP = 64;     // rows per step of a block: 8 warps x 8 loads a thread
constexpr int ENC_BLOCKS = 6;    // blocks an SM that the row chunks are sized for: six of the eight it holds

// Per-column scratch of the encoder.
struct EncWs {
    long long *mn, *mx;  // column minimum / maximum
    int *bad;            // column has a non-integer value
    unsigned *bits;      // presence bitmap, ENC_WORDS words per column (8-byte aligned)
    int *status;
};

// The integer type a sample's value is held in.
template <typename T>
struct EncInt {
    using type = int;
};
template <>
struct EncInt<long long> {
    using type = long long;
};
template <>
struct EncInt<double> {
    using type = long long;
};

template <typename T, typename V>
__device__ __forceinline__ bool enc_value(T x, V &v) {
    if constexpr (sizeof(T) == 8 && (T)0.5 != 0) {  // double
        // on the bits: conversions run on the FP64 pipe (1/64 of the integer rate)
        const long long u = __double_as_longlong((double)x);
        const int e = (int)((u >> 52) & 0x7ff) - 1023;
        const unsigned long long m = ((unsigned long long)u & 0xfffffffffffffull) | 0x10000000000000ull;
        if (e < 0) {  // |x| < 1
            v = 0;
            return (u << 1) == 0;
        }
        if (e <= 52) {
            const long long a = (long long)(m >> (52 - e));
            v = u < 0 ? -a : a;
            return (m << 11 << (1 + e)) == 0;  // the fraction's 52 - e bits
        }
        const double d = (double)x;
        v = (long long)d;
        return (double)v == d;  // integral (NaN fails)
    } else {
        v = (V)x;
        return true;
    }
}

__global__ void __launch_bounds__(256) enc_init_kernel(long long n, int p, uint8_t *__restrict__ dims, EncWs w) {
    pdl_trigger();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const long long words = (long long)p * ENC_WORDS;
    for (long long q = k; q < words; q += gridDim.x * blockDim.x) w.bits[q] = 0u;
    for (int j = k; j < p; j += gridDim.x * blockDim.x) {
        w.mn[j] = 0x7fffffffffffffffll;
        w.mx[j] = (long long)0x8000000000000000ull;
        w.bad[j] = 0;
        if (n == 0) dims[j] = 1;
    }
    if (k == 0) *w.status = 0;
}

// Pass 1: tile (blockIdx.x: 32 columns, blockIdx.y: rows); lane = column.
template <typename T>
__global__ void __launch_bounds__(256) enc_scan_kernel(const T *__restrict__ X, long long n, int p, long long ld,
                                                      int rows, EncWs w) {
    using V = typename EncInt<T>::type;
    __shared__ V smin[8][32], smax[8][32];
    __shared__ unsigned long long smask[8][32];
    __shared__ int sbad[32];
    __shared__ unsigned bits[ENC_WORDS][32];
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + lane;
    const long long t0 = (long long)blockIdx.y * rows, t1 = min(n, t0 + rows);
    if (threadIdx.x < 32) sbad[threadIdx.x] = 0;
    V mn = 0, mx = 0;
    unsigned long long mask = 0ull;  // 0: no value seen
    bool ok = true;
    auto take = [&](T x) {
        V v;
        ok = enc_value(x, v) && ok;
        mn = mask == 0ull || v < mn ? v : mn;
        mx = mask == 0ull || v > mx ? v : mx;
        mask |= 1ull << ((int)v & 63);
    };
    if (j < p) {
        long long t = t0 + warp;
        for (; t + 56 < t1; t += ENC_STEP) {
            T x[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = X[(t + 8 * e) * ld + j];
#pragma unroll
            for (int e = 0; e < 8; ++e) take(x[e]);
        }
        for (; t < t1; t += 8) take(X[t * ld + j]);
    }
    __syncthreads();
    smin[warp][lane] = mn;
    smax[warp][lane] = mx;
    smask[warp][lane] = mask;
    if (!ok) sbad[lane] = 1;
    __syncthreads();
    // every warp finds its columns' span over the block
    mask = 0ull;
    for (int q = 0; q < 8; ++q) {
        const unsigned long long m = smask[q][lane];
        if (m == 0ull) continue;
        mn = mask == 0ull || smin[q][lane] < mn ? smin[q][lane] : mn;
        mx = mask == 0ull || smax[q][lane] > mx ? smax[q][lane] : mx;
        mask |= m;
    }
    const bool wide = mask != 0ull && (unsigned long long)(long long)mx - (unsigned long long)(long long)mn >= 64ull;
    const bool any_wide = __any_sync(GCSL_FULL_MASK, wide);  // (the same in every warp)
    pdl_wait();  // the scratch is initialised
    if (warp == 0 && j < p) {  // (mask != 0: a tile has at least one row)
        atomicMin(w.mn + j, (long long)mn);
        atomicMax(w.mx + j, (long long)mx);
        if (sbad[lane]) atomicOr(w.bad + j, 1);
        if (!any_wide) {
            // bits from the minimum's up lie in its word, those below it in the next one
            unsigned long long *g = reinterpret_cast<unsigned long long *>(w.bits + (size_t)j * ENC_WORDS);
            const int wd = (int)(mn >> 6) & (ENC_RANGE / 64 - 1);
            const unsigned long long up = ~0ull << ((int)mn & 63);
            if (mask & up) atomicOr(g + wd, mask & up);
            if (mask & ~up) atomicOr(g + ((wd + 1) & (ENC_RANGE / 64 - 1)), mask & ~up);
        }
    }
    if (!any_wide) return;
    for (int k = threadIdx.x; k < 32 * ENC_WORDS; k += blockDim.x) (&bits[0][0])[k] = 0u;
    __syncthreads();
    if (j < p) {
        for (long long t = t0 + warp; t < t1; t += 8) {
            V v;
            enc_value(X[t * ld + j], v);
            // values repeat: set a bit only when it is not set yet (few atomics)
            const int o = (int)v & (ENC_RANGE - 1);
            const unsigned bit = 1u << (o & 31);
            if (!(bits[o >> 5][lane] & bit)) atomicOr(&bits[o >> 5][lane], bit);
        }
    }
    __syncthreads();
    for (int wd = warp; wd < ENC_WORDS; wd += 8) {
        const unsigned b = bits[wd][lane];
        if (b != 0u && j < p) atomicOr(w.bits + (size_t)j * ENC_WORDS + wd, b);
    }
}

// Codes of the tile's rows, ENC_STEP x 32 columns at a time, written column-major; `code_of`
// gives the code of a sample of the thread's column.
template <typename T, typename F>
__device__ __forceinline__ void enc_write(const T *__restrict__ X, int p, long long ld, long long t0, long long t1,
                                          uint8_t *__restrict__ codes, long long ldc,
                                          unsigned long long (*tile)[32][9], F code_of) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j0 = blockIdx.x * 32, j = j0 + lane;
    const int c = threadIdx.x >> 3, g = threadIdx.x & 7;  // column and 8-sample group written out
    int buf = 0;
    for (long long ts = t0; ts < t1; ts += ENC_STEP, buf ^= 1) {
        const long long r0 = ts + warp * 8;
        T x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = j < p && r0 + e < t1 ? X[(r0 + e) * ld + j] : T(0);
        unsigned lo = 0u, hi = 0u;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            lo |= (code_of(x[e]) & 0xffu) << (8 * e);
            hi |= (code_of(x[e + 4]) & 0xffu) << (8 * e);
        }
        tile[buf][lane][warp] = ((unsigned long long)hi << 32) | lo;
        __syncthreads();  // (two buffers: the next step's writes cannot reach this step's reads)
        const long long t = ts + g * 8;
        if (j0 + c < p && t < t1) {
            const unsigned long long v = tile[buf][c][g];
            uint8_t *dst = codes + (size_t)(j0 + c) * ldc + t;
            if (t + 8 <= t1 && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0) {
                *reinterpret_cast<unsigned long long *>(dst) = v;
            } else {
                for (int e = 0; e < 8 && t + e < t1; ++e) dst[e] = (uint8_t)(v >> (8 * e));
            }
        }
    }
}

// Pass 2: codes, dims and status.
template <typename T, bool PAD>
__global__ void __launch_bounds__(256) enc_codes_kernel(const T *__restrict__ X, long long n, int p, long long ld,
                                                       int rows, uint8_t *__restrict__ codes, long long ldc,
                                                       uint8_t *__restrict__ dims, EncWs w) {
    using V = typename EncInt<T>::type;
    __shared__ unsigned long long tile[2][32][9];
    __shared__ unsigned bits[ENC_WORDS][PAD ? 33 : 32];
    __shared__ uint8_t rank[ENC_WORDS][PAD ? 36 : 32];
    __shared__ int total[32];
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j0 = blockIdx.x * 32, j = j0 + lane;
    const bool col = j < p;
    const long long base = col ? w.mn[j] : 0, top = col ? w.mx[j] : 0;
    const unsigned long long span = (unsigned long long)top - (unsigned long long)base;  // values less one
    const long long t0 = (long long)blockIdx.y * rows, t1 = min(n, t0 + rows);
    const bool narrow = __all_sync(GCSL_FULL_MASK, span < 64ull);  // (the same in every warp)
    auto finish = [&](int count) {  // one warp of the first row chunk, lane = column
        if (count > 255 || span >= ENC_RANGE || w.bad[j]) atomicCAS(w.status, 0, GCSL_ERR_UNSUPPORTED);
        dims[j] = (uint8_t)(count > 0 ? (count > 255 ? 255 : count) : 1);
    };
    if (narrow) {
        unsigned long long m = 0ull;  // bit k: the value base + k is present
        if (col) {
            const unsigned long long *g =
                reinterpret_cast<const unsigned long long *>(w.bits + (size_t)j * ENC_WORDS);
            const int wd = (int)(base >> 6) & (ENC_RANGE / 64 - 1), sh = (int)base & 63;
            m = g[wd] >> sh;
            if (sh) m |= g[(wd + 1) & (ENC_RANGE / 64 - 1)] << (64 - sh);
            if (blockIdx.y == 0 && warp == 0) finish(__popcll(m));
        }
        const int b = (int)base;
        if (__all_sync(GCSL_FULL_MASK, span < 32ull)) {
            const unsigned m32 = (unsigned)m;
            enc_write(X, p, ld, t0, t1, codes, ldc, tile, [&](T x) -> unsigned {
                V v;
                enc_value(x, v);
                return __popc(m32 & ((1u << (((int)v - b) & 31)) - 1u));
            });
        } else {
            enc_write(X, p, ld, t0, t1, codes, ldc, tile, [&](T x) -> unsigned {
                V v;
                enc_value(x, v);
                return __popcll(m & ((1ull << (((int)v - b) & 63)) - 1ull));
            });
        }
        return;
    }
    for (int k = threadIdx.x; k < 32 * ENC_WORDS; k += blockDim.x) {
        const int c = k / ENC_WORDS, wd = k - c * ENC_WORDS;
        bits[wd][c] = j0 + c < p ? w.bits[(size_t)(j0 + c) * ENC_WORDS + wd] : 0u;
    }
    __syncthreads();
    // rank of a word's first bit, counted from the minimum's bit around the circle, mod 256
    // (codes below 255 are exact)
    for (int c = warp; c < 32; c += 8) {
        const int o0 = (int)__shfl_sync(GCSL_FULL_MASK, base, c) & (ENC_RANGE - 1);
        int carry = 0;
        for (int w0 = 0; w0 < ENC_WORDS; w0 += 32) {
            const int cnt = __popc(bits[w0 + lane][c]);
            int x = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(GCSL_FULL_MASK, x, o);
                if (lane >= o) x += y;
            }
            rank[w0 + lane][c] = (uint8_t)(carry + x - cnt);
            carry += __shfl_sync(GCSL_FULL_MASK, x, 31);
        }
        __syncwarp();
        const int below = rank[o0 >> 5][c] + __popc(bits[o0 >> 5][c] & ((1u << (o0 & 31)) - 1u));
        __syncwarp();
        for (int w0 = 0; w0 < ENC_WORDS; w0 += 32) rank[w0 + lane][c] = (uint8_t)(rank[w0 + lane][c] - below);
        if (lane == 0) total[c] = carry;
    }
    __syncthreads();
    if (blockIdx.y == 0 && warp == 0 && col) finish(total[lane]);
    const int o0 = (int)base & (ENC_RANGE - 1), count = total[lane];
    enc_write(X, p, ld, t0, t1, codes, ldc, tile, [&](T x) -> unsigned {
        V v;
        enc_value(x, v);
        const int o = (int)v & (ENC_RANGE - 1), wd = o >> 5;
        // bits below the minimum's come after the last one's
        return rank[wd][lane] + __popc(bits[wd][lane] & ((1u << (o & 31)) - 1u)) + (o < o0 ? count : 0);
    });
}

namespace host {

size_t encode_workspace_bytes(int p) {
    const size_t per = 2 * sizeof(long long) + sizeof(int) + ENC_WORDS * sizeof(unsigned);
    return 256 + ((size_t)p * per + 255) / 256 * 256;
}

static EncWs enc_ws(void *ws, int p) {
    uint8_t *c = static_cast<uint8_t *>(ws);
    EncWs w;
    w.status = reinterpret_cast<int *>(c);
    c += 256;
    w.mn = reinterpret_cast<long long *>(c);
    c += (size_t)p * sizeof(long long);
    w.mx = reinterpret_cast<long long *>(c);
    c += (size_t)p * sizeof(long long);
    w.bits = reinterpret_cast<unsigned *>(c);
    c += (size_t)p * ENC_WORDS * sizeof(unsigned);
    w.bad = reinterpret_cast<int *>(c);
    return w;
}

template <typename T>
static cudaError_t encode_typed(const T *X, long long n, int p, long long ld, uint8_t *codes, long long ldc,
                                uint8_t *dims, const EncWs &w, int num_sms, cudaStream_t s) {
    const int strips = (p + 31) / 32, all = ENC_BLOCKS * num_sms;
    const int init_blocks = std::min((p + 7) / 8, all);
    enc_init_kernel<<<(unsigned)init_blocks, 256, 0, s>>>(n, p, dims, w);
    note_launch(1);
    cudaError_t e = cudaGetLastError();
    if (n == 0 || e != cudaSuccess) return e;
    // whole steps a tile, about `all` tiles in all, at most 65535 along the rows
    const long long want = std::min(65535, std::max(1, all / strips));
    long long rows = (n + want - 1) / want;
    rows = (rows + ENC_STEP - 1) / ENC_STEP * ENC_STEP;
    const dim3 grid((unsigned)strips, (unsigned)((n + rows - 1) / rows));
    const bool pad = rows <= ENC_PAD_ROWS;
    e = launch_pdl(enc_scan_kernel<T>, grid, dim3(256), 0, s, X, n, p, ld, (int)rows, w);
    if (e == cudaSuccess)
        e = launch_pdl(pad ? enc_codes_kernel<T, true> : enc_codes_kernel<T, false>, grid, dim3(256), 0, s, X, n, p, ld,
                       (int)rows, codes, ldc, dims, w);
    note_launch(2);
    return e != cudaSuccess ? e : cudaGetLastError();
}

// status: the first int of the workspace (cleared here); the caller reads it back.
cudaError_t encode_columns(const void *X, int dtype, long long n, int p, long long ld, uint8_t *codes, long long ldc,
                           uint8_t *dims, void *workspace, int num_sms, cudaStream_t s) {
    const EncWs w = enc_ws(workspace, p);
    switch (dtype) {
    case GCSL_DTYPE_I32: return encode_typed(static_cast<const int *>(X), n, p, ld, codes, ldc, dims, w, num_sms, s);
    case GCSL_DTYPE_I64: return encode_typed(static_cast<const long long *>(X), n, p, ld, codes, ldc, dims, w, num_sms, s);
    case GCSL_DTYPE_U8: return encode_typed(static_cast<const uint8_t *>(X), n, p, ld, codes, ldc, dims, w, num_sms, s);
    case GCSL_DTYPE_F64: return encode_typed(static_cast<const double *>(X), n, p, ld, codes, ldc, dims, w, num_sms, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace host
}  // namespace gcsl
