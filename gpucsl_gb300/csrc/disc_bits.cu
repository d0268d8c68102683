// Levels 0 and 1 of the discrete skeleton on bit planes.
//
// A level-0 or level-1 test needs the table N[s][a][b] over all n samples, and the same
// column takes part in hundreds of tests.  Each value a of a variable becomes one bit
// plane (bit = the sample has that value), and a cell is the population count of the AND
// of two or three planes.  A variable of d values has d - 1 planes: the cells of its last
// value follow from the tables one variable smaller.  So the counts of a level are small
// matrix products over bits, between all pairs of planes (level 0) or, for a centre i and
// each value a of i but the last, between all pairs of planes of i's neighbours masked by
// plane (i, a) (level 1: one table serves the tests (i, j | s) and (i, s | j)).
//
// A warp multiplies 4 planes by 4, lane = word pair: 8 loads feed 16 cells, the next pass's
// loads in flight.  Population counts run at 16 lanes a clock (64 for LOP3), so two words
// of a cell are first added as bits to a kept word (carry-save: sum = x ^ y ^ z stays,
// majority has weight two) and one count per two words remains; counting and logic then
// take the same time.
//
// Statistics: every count is an exact integer; a test's chi-squared is first bounded from
// below in FP32, and a test whose p-value is certainly zero (the series cuts terms below
// exp(-20) off) ends there: it can neither raise the pair's largest p-value nor remove the
// edge.  The others, packed densely, are evaluated in FP64 from the integers
// q = N N_s - N_a N_b, which are exact: chi^2 = sum q^2 / (N_a N_b N_s); those on a jump of the
// p-value once more in the published order (pvalue_tie).
//
// Measured against one block per test with shared-memory atomics (level 0, level 1):
// p = 200, n = 50000, cardinality 2..5: 476, 1805 -> 104, 409 us; p = 299, n = 99991,
// cardinality 2..6: 1836, 8095 -> 381, 2146 us.  Level 1 is bound by the integer pipe (LOP3
// and the population counts, about 60 % busy) and the latency of the plane loads.
#include <algorithm>

#include "disc_stat.cuh"

namespace gcsl {

constexpr int BP_SIDE = 4;         // planes on each side of a warp's block
constexpr int BP_GROUP = 24;       // planes of a neighbour group of a level-1 task
constexpr int BP_LANES = 8;        // lanes that share one test's statistic
constexpr int BP_LEVEL1_DIM = 10;  // level 1: values of a variable up to which planes may pay
constexpr int BP_ROUND = 64;       // words of one pass of a warp (2 a lane): slices are multiples

// Words of a plane: whole passes, zero past the samples.
__host__ __device__ inline long long bp_words(long long n) {
    return (n + 32 * BP_ROUND - 1) / (32 * BP_ROUND) * BP_ROUND;
}

// Neighbours of one level-1 group: as many as surely fit in BP_GROUP planes.
__host__ __device__ inline int bp_group_vars(int max_dim) { return max_dim > 1 ? BP_GROUP / (max_dim - 1) : BP_GROUP; }

// ------------------------------------------------------------------ bit planes
// Item (chunk, v): planes of variable v.  A lane takes 32 samples (two 16-byte loads) and
// makes one word of every plane: four codes at a time, a byte of (w ^ aaaa) + 0x7f.. has its
// high bit clear exactly where the code is a (codes below 128), and the eight steps' bits
// are shifted together.  A word holds its samples in the order this gives, the same for every
// plane, which is all that counts need.  Codes at or above the cardinality set
// GCSL_ERR_INVALID_ARG.  The first item of a variable also stores its cardinality (1 ..
// max_dim, the bound all buffers are sized by; a larger one sets DISC_STATUS_WIDE, ends the
// solve's levels, whose sepsets would come from the clamped counts, and the solve is repeated
// on the general path), off[v] planes before it (d - 1 each) and foff[v] values before it (d
// each).  LG_BLOCKS extra items build the ln Gamma tables.
//
// Bound by the integer pipe: 4 instructions per 4 codes and value (a ballot per sample took
// three times as many: 66 us at p = 299, n = 99991, cardinality 2..6).
__device__ __forceinline__ void planes_item(int item, const uint8_t *__restrict__ data, long long ld, long long n,
                                            int p, const uint8_t *__restrict__ dims, int max_dim, int chunks,
                                            uint32_t *__restrict__ planes, long long words, uint8_t *__restrict__ card,
                                            int *__restrict__ off, int *__restrict__ foff, double *__restrict__ lg,
                                            DevState *st) {
    __shared__ int s_sum[8][2];
    if (item >= chunks * p) {
        lgam_build(lg, item - chunks * p);
        return;
    }
    const int v = item / chunks, chunk = item - v * chunks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // planes and values before v
    int po = 0, fo = 0;
    for (int u = threadIdx.x; u < v; u += blockDim.x) {
        const int d = max(1, min((int)dims[u], max_dim));
        po += d - 1;
        fo += d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        po += __shfl_xor_sync(GCSL_FULL_MASK, po, o);
        fo += __shfl_xor_sync(GCSL_FULL_MASK, fo, o);
    }
    if (lane == 0) {
        s_sum[warp][0] = po;
        s_sum[warp][1] = fo;
    }
    __syncthreads();
    po = fo = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        po += s_sum[w][0];
        fo += s_sum[w][1];
    }
    const int d = max(1, min((int)dims[v], max_dim));
    if (chunk == 0 && threadIdx.x == 0) {
        if (dims[v] > max_dim) {
            set_status(st, DISC_STATUS_WIDE);
            st->done = 1;
        }
        card[v] = (uint8_t)d;
        off[v] = po;
        foff[v] = fo;
        if (v == p - 1) {
            off[p] = po + d - 1;
            foff[p] = fo + d;
        }
    }
    const uint32_t dv = dims[v];
    const uint32_t above = dv <= 128 ? (0x80u - dv) * 0x01010101u : 0u;
    uint32_t bad = 0;
    for (long long w = (long long)chunk * blockDim.x + threadIdx.x; w < words; w += (long long)chunks * blockDim.x) {
        const long long t = 32 * w;
        uint32_t c[8];
        if (t + 32 <= n) {
            const uint4 *src = reinterpret_cast<const uint4 *>(data + (size_t)v * ld + t);
            const uint4 x = __ldg(src), y = __ldg(src + 1);
            c[0] = x.x, c[1] = x.y, c[2] = x.z, c[3] = x.w;
            c[4] = y.x, c[5] = y.y, c[6] = y.z, c[7] = y.w;
#pragma unroll
            for (int q = 0; q < 8; ++q) bad |= ((c[q] + above) | c[q]) & 0x80808080u;
        } else {  // the last samples byte by byte; 0x7f matches no value
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                c[q] = 0x7f7f7f7fu;
                for (int e = 0; e < 4; ++e)
                    if (t + 4 * q + e < n) {
                        const uint32_t x = data[(size_t)v * ld + t + 4 * q + e];
                        bad |= x >= dv;
                        c[q] = (c[q] & ~(0xffu << (8 * e))) | ((x < 128u ? x : 0x7fu) << (8 * e));
                    }
            }
        }
        for (int a = 0; a + 1 < d; ++a) {
            const uint32_t rep = 0x01010101u * (uint32_t)a;
            uint32_t word = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) word = (word >> 1) | (~((c[q] ^ rep) + 0x7f7f7f7fu) & 0x80808080u);
            planes[(size_t)(po + a) * words + w] = word;
        }
    }
    if (dv > 128) bad = 0;  // more than max_dim values: the general path checks them
    if (__any_sync(GCSL_FULL_MASK, bad != 0) && lane == 0) set_status(st, GCSL_ERR_INVALID_ARG);
}

// One item a block, or with a cap on the resident blocks several.  The blocks also clear the pair
// counts (`cells` words on a 16-byte boundary), which the next kernel adds to.
__global__ void __launch_bounds__(256) disc_planes_kernel(const uint8_t *__restrict__ data, long long ld, long long n,
                                                          int p, const uint8_t *__restrict__ dims, int max_dim,
                                                          int chunks, uint32_t *__restrict__ planes, long long words,
                                                          uint8_t *__restrict__ card, int *__restrict__ off,
                                                          int *__restrict__ foff, double *__restrict__ lg,
                                                          uint32_t *__restrict__ counts, long long cells,
                                                          DevState *st) {
    const long long thread = (long long)blockIdx.x * blockDim.x + threadIdx.x,
                    threads = (long long)gridDim.x * blockDim.x;
    for (long long k = thread; k < cells / 4; k += threads)
        reinterpret_cast<uint4 *>(counts)[k] = make_uint4(0u, 0u, 0u, 0u);
    if (thread < cells % 4) counts[cells - 1 - thread] = 0u;
    for (int item = (int)blockIdx.x; item < chunks * p + LG_BLOCKS; item += (int)gridDim.x) {
        planes_item(item, data, ld, n, p, dims, max_dim, chunks, planes, words, card, off, foff, lg, st);
        __syncthreads();  // its shared sums are read
    }
}

// ------------------------------------------------------------ counts of a block
// Words of one pass of a warp: two consecutive words of 4 + 4 planes per lane.  The planes
// are given by their first words' offsets, 32 bits each (host: all planes below 2^32 words).
struct PopcWords {
    uint2 r[BP_SIDE], c[BP_SIDE];
    __device__ __forceinline__ void load(const uint32_t *__restrict__ planes, const uint32_t (&ro)[BP_SIDE],
                                         const uint32_t (&co)[BP_SIDE]) {
#pragma unroll
        for (int i = 0; i < BP_SIDE; ++i) r[i] = __ldg(reinterpret_cast<const uint2 *>(planes + ro[i]));
#pragma unroll
        for (int j = 0; j < BP_SIDE; ++j) c[j] = __ldg(reinterpret_cast<const uint2 *>(planes + co[j]));
    }
};

// Carry-save step of one cell: `kept` gains the bits of x and y; returns the count of the
// carries (weight two).
__device__ __forceinline__ uint32_t csa_count(uint32_t &kept, uint32_t x, uint32_t y) {
    uint32_t carry;
    asm("lop3.b32 %0, %1, %2, %3, 0xe8;" : "=r"(carry) : "r"(kept), "r"(x), "r"(y));  // majority
    asm("lop3.b32 %0, %1, %2, %3, 0x96;" : "=r"(kept) : "r"(kept), "r"(x), "r"(y));   // sum
    return __popc(carry);
}

// Counts of the planes at word offsets ro x co, masked by the plane at mo with MASKED, over
// `passes` passes from word w0; lane l returns the count of (row l / 4 % 4, column l % 4).
template <bool MASKED>
__device__ __forceinline__ uint32_t popc_block(const uint32_t *__restrict__ planes, uint32_t (&ro)[BP_SIDE],
                                               uint32_t (&co)[BP_SIDE], uint32_t mo, int w0, int passes) {
    const int lane = threadIdx.x & 31;
    const uint32_t first = (uint32_t)w0 + 2u * lane;
#pragma unroll
    for (int k = 0; k < BP_SIDE; ++k) ro[k] += first, co[k] += first;
    mo += first;
    uint32_t kept[BP_SIDE * BP_SIDE], twos[BP_SIDE * BP_SIDE];
#pragma unroll
    for (int k = 0; k < BP_SIDE * BP_SIDE; ++k) kept[k] = twos[k] = 0;
    PopcWords next;
    uint2 m, mask = make_uint2(0u, 0u);
    next.load(planes, ro, co);
    if (MASKED) mask = __ldg(reinterpret_cast<const uint2 *>(planes + mo));
    for (int t = 0; t < passes; ++t) {
        PopcWords now = next;
        m = mask;
        if (t + 1 < passes) {
#pragma unroll
            for (int k = 0; k < BP_SIDE; ++k) ro[k] += BP_ROUND, co[k] += BP_ROUND;
            next.load(planes, ro, co);
            if (MASKED) {
                mo += BP_ROUND;
                mask = __ldg(reinterpret_cast<const uint2 *>(planes + mo));
            }
        }
        if (MASKED) {
#pragma unroll
            for (int j = 0; j < BP_SIDE; ++j) now.c[j].x &= m.x, now.c[j].y &= m.y;
        }
#pragma unroll
        for (int i = 0; i < BP_SIDE; ++i)
#pragma unroll
            for (int j = 0; j < BP_SIDE; ++j) {
                const int k = BP_SIDE * i + j;
                twos[k] += csa_count(kept[k], now.r[i].x & now.c[j].x, now.r[i].y & now.c[j].y);
            }
    }
#pragma unroll
    for (int k = 0; k < BP_SIDE * BP_SIDE; ++k) kept[k] = 2 * twos[k] + __popc(kept[k]);
    // 16 sums over 32 lanes: halve the values and add the other half's at each step
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < o; ++k) {
            const uint32_t send = up ? kept[k] : kept[k + o];
            const uint32_t mine = up ? kept[k + o] : kept[k];
            kept[k] = mine + __shfl_xor_sync(GCSL_FULL_MASK, send, o);
        }
    }
    return kept[0] + __shfl_xor_sync(GCSL_FULL_MASK, kept[0], 16);
}

// Words per slice when `blocks` blocks are to give about `want` work items: the slices are
// whole passes, at least four of them.
__device__ __forceinline__ int slice_words(long long words, long long blocks, long long want) {
    long long slices = (want + blocks - 1) / (blocks > 0 ? blocks : 1);
    const long long most = words / (4 * BP_ROUND) > 1 ? words / (4 * BP_ROUND) : 1;
    slices = slices < 1 ? 1 : slices > most ? most : slices;
    return (int)(((words + slices - 1) / slices + BP_ROUND - 1) / BP_ROUND * BP_ROUND);
}

// ------------------------------------------------------------------- level 0
// Counts of all pairs of planes (x <= y), both triangles of `counts` (cleared before).  The
// blocks of the upper triangle, each cut into K slices when they alone would not fill the
// resident warps a few times over.
__global__ void __launch_bounds__(256, 2) disc_pair_counts_kernel(const uint32_t *__restrict__ planes, long long words,
                                                                  const int *__restrict__ off, int p,
                                                                  uint32_t *__restrict__ counts, int ldc,
                                                                  DevState *st) {
    const int lane = threadIdx.x & 31;
    const int S = off[p];
    const long long nb = (S + BP_SIDE - 1) / BP_SIDE;
    const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long blocks = nb * (nb + 1) / 2;  // block row r pairs with block columns r .. nb - 1
    const long long per = slice_words(words, blocks, 6 * warps), slices = (words + per - 1) / per;
    for (long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < blocks * slices; t += warps) {
        const long long b = t / slices, sl = t - b * slices;
        // first block of row r: r nb - r (r - 1) / 2
        const float h = (float)nb + 0.5f;
        long long r = (long long)(h - sqrtf(fmaxf(h * h - 2.0f * (float)b, 0.0f)));
        r = r < nb ? r : nb - 1;
        while (r > 0 && r * nb - r * (r - 1) / 2 > b) --r;
        while (r + 1 < nb && (r + 1) * nb - (r + 1) * r / 2 <= b) ++r;
        const long long c = r + (b - (r * nb - r * (r - 1) / 2));
        uint32_t ro[BP_SIDE], co[BP_SIDE];
#pragma unroll
        for (int i = 0; i < BP_SIDE; ++i) {
            ro[i] = (uint32_t)(min((int)(BP_SIDE * r) + i, S - 1) * words);
            co[i] = (uint32_t)(min((int)(BP_SIDE * c) + i, S - 1) * words);
        }
        const long long w0 = sl * per, w1 = w0 + per < words ? w0 + per : words;
        if (!dcheck(st, S <= ldc && c < nb && w0 < w1 && (w1 - w0) % BP_ROUND == 0, GCSL_DCHECK_CELL)) continue;
        const uint32_t got = popc_block<false>(planes, ro, co, 0u, (int)w0, (int)(w1 - w0) / BP_ROUND);
        const int x = (int)(BP_SIDE * r) + lane / 4, y = (int)(BP_SIDE * c) + lane % 4;
        if (lane < 16 && x <= y && y < S && got != 0) {
            atomicAdd(counts + (size_t)x * ldc + y, got);
            if (x != y) atomicAdd(counts + (size_t)y * ldc + x, got);
        }
    }
}

// The cells of one test's table, shared by the BP_LANES lanes of its group: body(s, a, b).
// Quotients of the small cell indices by multiplication (exact below 2^12 cells with the
// half added).
template <class F>
__device__ __forceinline__ void group_cells(int ds, int di, int dj, int gl, F &&body) {
    const int per = di * dj, cells = ds * per;
    const float rp = 1.0f / (float)per, rj = 1.0f / (float)dj;
    for (int k = gl; k < cells; k += BP_LANES) {
        const int s = (int)(((float)k + 0.5f) * rp), r = k - s * per;
        const int a = (int)(((float)r + 0.5f) * rj);
        body(s, a, r - a * dj);
    }
}

template <typename V>
__device__ __forceinline__ V group_sum(V v, unsigned mask) {
#pragma unroll
    for (int o = BP_LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
    return v;
}

// chi^2 of one test by the lanes of its group: q = N N_s - N_a N_b is an exact integer
// (n < 2^30) and a cell adds q^2 / (N_a N_b N_s), by the reciprocals of the pair tables that
// all tests share (zero for an empty entry).  T supplies the counts strata(), rows(),
// cols(), cell(s, a, b), row(s, a), col(s, b), total(s) and 1 / row, 1 / col, 1 / total.
template <class T>
__device__ double chi2_exact(const T &t, int gl, unsigned mask) {
    double chi = 0.0;
    group_cells(t.strata(), t.rows(), t.cols(), gl, [&](int s, int a, int b) {
        const double q = (double)((long long)t.cell(s, a, b) * t.total(s) - (long long)t.row(s, a) * t.col(s, b));
        chi = fma(q * q, t.inv_row(s, a) * t.inv_col(s, b) * t.inv_total(s), chi);
    });
    return group_sum(chi, mask);
}

// A lower bound of chi^2 in FP32 (chi2_floor_term).
template <class T>
__device__ float chi2_floor(const T &t, int gl, unsigned mask) {
    float chi = 0.f;
    group_cells(t.strata(), t.rows(), t.cols(), gl, [&](int s, int a, int b) {
        const float e = __fdividef((float)t.row(s, a) * (float)t.col(s, b), (float)t.total(s));
        if (!(e > 0.f)) return;  // also a stratum without samples (0 / 0)
        chi += chi2_floor_term((float)t.cell(s, a, b), e);
    });
    return 0.999f * group_sum(chi, mask);
}

// P-value of a test in the published order, by one thread (tests on a jump of the p-value).
template <class T>
__device__ __noinline__ double pvalue_ordered(const T &t) {
    double chi = 0.0;
    for (int s = 0; s < t.strata(); ++s) {
        const double n = (double)t.total(s);
        if (n == 0.0) continue;
        double part = 0.0;
        for (int a = 0; a < t.rows(); ++a)
            for (int b = 0; b < t.cols(); ++b) {
                const double e = __ddiv_rn(__dmul_rn((double)t.row(s, a), (double)t.col(s, b)), n);
                if (e == 0.0) continue;
                const double d = __dsub_rn((double)t.cell(s, a, b), e);
                part = __dadd_rn(part, __ddiv_rn(__dmul_rn(d, d), e));
            }
        chi = __dadd_rn(chi, part);
    }
    return pchisq_dev(chi, (long long)(t.rows() - 1) * (t.cols() - 1) * t.strata());
}

// One pair's full table in shared memory with its marginals.
struct PairTable {
    const uint32_t *tab, *nr, *nc;  // di x dj cells (row stride dj), row and column counts
    const double *ir, *ic;          // reciprocals of the row and column counts
    int di, dj;
    uint32_t n;
    double in;
    __device__ __forceinline__ int strata() const { return 1; }
    __device__ __forceinline__ int rows() const { return di; }
    __device__ __forceinline__ int cols() const { return dj; }
    __device__ __forceinline__ uint32_t total(int) const { return n; }
    __device__ __forceinline__ uint32_t row(int, int a) const { return nr[a]; }
    __device__ __forceinline__ uint32_t col(int, int b) const { return nc[b]; }
    __device__ __forceinline__ uint32_t cell(int, int a, int b) const { return tab[a * dj + b]; }
    __device__ __forceinline__ double inv_row(int, int a) const { return ir[a]; }
    __device__ __forceinline__ double inv_col(int, int b) const { return ic[b]; }
    __device__ __forceinline__ double inv_total(int) const { return in; }
};

// Level 0, a group of BP_LANES lanes per pair (vi >= vj): its full table F (all values, both
// triangles, the counts of single values on the diagonal) with the reciprocals, for level 1
// (where `full` is given), and its test.  The last row and column of a table come from the counts
// of single values.
// p-values are evaluated a thread per test at the end of a round.
constexpr int BP_L0_THREADS = 128, BP_L0_GROUPS = BP_L0_THREADS / BP_LANES;
__global__ void __launch_bounds__(BP_L0_THREADS) disc_level0_kernel(
    const uint32_t *__restrict__ counts, int ldc, int p, const uint8_t *__restrict__ dims, const int *__restrict__ off,
    const int *__restrict__ foff, uint32_t n, uint32_t *__restrict__ full, double *__restrict__ inv, int ldf,
    double alpha, const double *__restrict__ lg, uint16_t *__restrict__ G, double *__restrict__ pmax, DevState *st,
    unsigned long long order) {
    __shared__ uint32_t s_tab[BP_L0_GROUPS][256];
    __shared__ uint32_t s_nr[BP_L0_GROUPS][16], s_nc[BP_L0_GROUPS][16];
    __shared__ double s_ir[BP_L0_GROUPS][16], s_ic[BP_L0_GROUPS][16];
    __shared__ double s_chi[BP_L0_GROUPS];
    __shared__ int s_df[BP_L0_GROUPS], s_vi[BP_L0_GROUPS], s_vj[BP_L0_GROUPS];
    const int gl = threadIdx.x & (BP_LANES - 1), gw = threadIdx.x / BP_LANES;
    const unsigned mask = ((1u << BP_LANES) - 1u) << (threadIdx.x & 31 & ~(BP_LANES - 1));
    const long long total = (long long)p * (p + 1) / 2;
    const double rn = 1.0 / (double)n;
    for (long long t0 = (long long)blockIdx.x * BP_L0_GROUPS; t0 < total; t0 += (long long)gridDim.x * BP_L0_GROUPS) {
        const long long t1 = t0 + gw;
        if (t1 < total) {
            const long long t = work_order(t1, total, order);
            long long u = (long long)((sqrtf(1.0f + 8.0f * (float)t) - 1.0f) * 0.5f);  // t = u (u + 1) / 2 + v, v <= u
            while (u > 0 && u * (u + 1) / 2 > t) --u;
            while ((u + 1) * (u + 2) / 2 <= t) ++u;
            const int vi = (int)u, vj = (int)(t - u * (u + 1) / 2);
            int x = off[vi], y = off[vj], di = dims[vi], dj = dims[vj], fi = foff[vi], fj = foff[vj];
            if (!dcheck(st, vi < p && min(di, dj) >= 1 && max(di, dj) <= 16 && max(x + di, y + dj) - 1 <= ldc &&
                                max(fi + di, fj + dj) <= ldf, GCSL_DCHECK_CELL)) {
                x = y = fi = fj = 0;
                di = dj = 1;
            }
            uint32_t *tab = s_tab[gw], *nr = s_nr[gw], *nc = s_nc[gw];
            for (int a = gl; a < di - 1; a += BP_LANES) nr[a] = __ldg(counts + (size_t)(x + a) * (ldc + 1));
            for (int b = gl; b < dj - 1; b += BP_LANES) nc[b] = __ldg(counts + (size_t)(y + b) * (ldc + 1));
            group_cells(1, di - 1, dj - 1, gl, [&](int, int a, int b) {
                tab[a * dj + b] = __ldg(counts + (size_t)(x + a) * ldc + y + b);
            });
            __syncwarp(mask);
            if (gl == 0 && di > 0) {
                uint32_t s = n;
                for (int a = 0; a < di - 1; ++a) s -= nr[a];
                nr[di - 1] = s;
            }
            if (gl == 1 && dj > 0) {
                uint32_t s = n;
                for (int b = 0; b < dj - 1; ++b) s -= nc[b];
                nc[dj - 1] = s;
            }
            __syncwarp(mask);
            for (int a = gl; a < di - 1; a += BP_LANES) {  // last column
                uint32_t s = nr[a];
                for (int b = 0; b < dj - 1; ++b) s -= tab[a * dj + b];
                tab[a * dj + dj - 1] = s;
            }
            __syncwarp(mask);
            for (int b = gl; b < dj; b += BP_LANES) {  // last row
                uint32_t s = nc[b];
                for (int a = 0; a < di - 1; ++a) s -= tab[a * dj + b];
                tab[(di - 1) * dj + b] = s;
            }
            __syncwarp(mask);
            double chi = 0.0;
            int df = -1;  // no p-value to evaluate
            if (vi == vj) {
                for (int a = gl; a < di; a += BP_LANES) {
                    if (full == nullptr) break;
                    full[(size_t)(fi + a) * ldf + fi + a] = nr[a];
                    inv[(size_t)(fi + a) * ldf + fi + a] = nr[a] ? 1.0 / (double)nr[a] : 0.0;
                }
            } else {
                group_cells(1, di, dj, gl, [&](int, int a, int b) {
                    if (full == nullptr) return;
                    const uint32_t c = tab[a * dj + b];
                    const double r = c ? 1.0 / (double)c : 0.0;
                    full[(size_t)(fi + a) * ldf + fj + b] = c;
                    full[(size_t)(fj + b) * ldf + fi + a] = c;
                    inv[(size_t)(fi + a) * ldf + fj + b] = r;
                    inv[(size_t)(fj + b) * ldf + fi + a] = r;
                });
                df = (di - 1) * (dj - 1);
                const PairTable T{tab, nr, nc, s_ir[gw], s_ic[gw], di, dj, n, rn};
                const bool zero = alpha > 0.0 && df > 0 && pvalue_zero(chi2_floor(T, gl, mask), df);
                if (zero) {
                    df = -2;
                } else if (df > 0) {
                    for (int k = gl; k < di + dj; k += BP_LANES) {
                        const uint32_t c = k < di ? nr[k] : nc[k - di];
                        (k < di ? s_ir[gw][k] : s_ic[gw][k - di]) = c ? 1.0 / (double)c : 0.0;
                    }
                    __syncwarp(mask);
                    chi = chi2_exact(T, gl, mask);
                } else {
                    df = 0;
                }
            }
            if (gl == 0) {
                s_chi[gw] = chi;
                s_df[gw] = df;
                s_vi[gw] = vi;
                s_vj[gw] = vj;
            }
        }
        __syncthreads();
        if (threadIdx.x < BP_L0_GROUPS && t0 + threadIdx.x < total && s_df[threadIdx.x] != -1) {
            const int vi = s_vi[threadIdx.x], vj = s_vj[threadIdx.x], df = s_df[threadIdx.x];
            double pv = df == -2 ? 0.0 : pchisq_tab(s_chi[threadIdx.x], df, lg);  // df 0: 1
            if (df > 0 && pvalue_tie(s_chi[threadIdx.x], pv, alpha))
                pv = pvalue_ordered(PairTable{s_tab[threadIdx.x], s_nr[threadIdx.x], s_nc[threadIdx.x], nullptr, nullptr,
                                              (int)dims[vi], (int)dims[vj], n, rn});
            pmax[(size_t)vj * p + vi] = pv;
            const uint16_t keep = pv >= alpha ? 0 : 1;
            G[(size_t)vi * p + vj] = keep;
            G[(size_t)vj * p + vi] = keep;
        }
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) st->tests[0] = (unsigned long long)p * (p - 1) / 2;
}

// ------------------------------------------------------------------- level 1
// Test (i, u | w) of a task from its shared tables.
struct TripleTable {
    const uint32_t *cnt;   // N[a of i][value of u][value of w]
    int su, sw, sa;        // strides of u's and w's values and of i's in cnt
    const uint32_t *uw;    // counts of the pair (u, w) with strides fu, fw, their reciprocals
    const double *ruw;
    int fu, fw;
    const uint32_t *iw;    // counts of the pair (i, w), lw per value of i, their reciprocals
    const double *riw;
    int lw;
    const uint32_t *nw;    // counts of w's values, their reciprocals
    const double *rnw;
    int di, du, dw;
    __device__ __forceinline__ int strata() const { return dw; }
    __device__ __forceinline__ int rows() const { return di; }
    __device__ __forceinline__ int cols() const { return du; }
    __device__ __forceinline__ uint32_t total(int s) const { return nw[s]; }
    __device__ __forceinline__ uint32_t row(int s, int a) const { return iw[a * lw + s]; }
    __device__ __forceinline__ uint32_t col(int s, int b) const { return uw[b * fu + s * fw]; }
    __device__ __forceinline__ uint32_t cell(int s, int a, int b) const { return cnt[a * sa + b * su + s * sw]; }
    __device__ __forceinline__ double inv_total(int s) const { return rnw[s]; }
    __device__ __forceinline__ double inv_row(int s, int a) const { return riw[a * lw + s]; }
    __device__ __forceinline__ double inv_col(int s, int b) const { return ruw[b * fu + s * fw]; }
};

// Shared-memory layout of a level-1 task (4-byte words; the doubles come first) for tables
// of max_dim values.
struct BitTaskLayout {
    int vars, values, ld, ruw, riu, riw, rnu, rnw, chi, cnt, uw, iu, iw, nu, nw, queue, words;
    __host__ __device__ explicit BitTaskLayout(int max_dim) {
        vars = bp_group_vars(max_dim);
        values = vars * max_dim;
        ld = values | 1;
        int o = 0;
        ruw = o, o += 2 * values * ld;
        riu = o, o += 2 * max_dim * values;
        riw = o, o += 2 * max_dim * values;
        rnu = o, o += 2 * values;
        rnw = o, o += 2 * values;
        chi = o, o += 2 * 2 * vars * vars;
        cnt = o, o += max_dim * values * ld;
        uw = o, o += values * ld;
        iu = o, o += max_dim * values;
        iw = o, o += max_dim * values;
        nu = o, o += values;
        nw = o, o += values;
        queue = o, o += 2 * vars * vars;
        words = o;
    }
};

constexpr int BP_MAX_VARS = BP_GROUP;
constexpr int BP_L1_THREADS = 128;

// A level-1 task: centre i and two groups g <= h of its neighbours; the tests (i, u | w) and
// (i, w | u) of every pair of neighbours u (group g) before w (group h).  Tasks are taken
// from a counter, so that the uneven ones (degrees and cardinalities differ) even out.
__global__ void __launch_bounds__(BP_L1_THREADS, 512 / BP_L1_THREADS) disc_bits_level1_kernel(const uint32_t *__restrict__ planes, long long words,
                                                                  const int *__restrict__ off,
                                                                  const int *__restrict__ foff,
                                                                  const uint32_t *__restrict__ full,
                                                                  const double *__restrict__ inv, int ldf,
                                                                  const long long *__restrict__ tasks,
                                                                  const int *__restrict__ rows, int max_dim,
                                                                  const double *__restrict__ lg, DiscLevelArgs A) {
    extern __shared__ __align__(8) uint32_t sm[];
    __shared__ long long s_task;
    __shared__ int s_var[2][BP_MAX_VARS], s_pl[2][BP_MAX_VARS + 1], s_va[2][BP_MAX_VARS + 1];
    __shared__ int s_plane[2][BP_GROUP], s_at[2][BP_GROUP];  // planes of a group, their places among its values
    __shared__ int s_value[2][2 * BP_GROUP];
    __shared__ int s_queued;
    DevState *st = A.st;
    if (st->done) return;
    if (st->max_degree[1] - 1 < 1) {
        if (blockIdx.x == 0 && threadIdx.x == 0) st->done = 1;
        return;
    }
    if (st->disc_route != 0) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->last_level = 1;
        st->tests[1] = (unsigned long long)A.prefix[A.p];
    }
    const BitTaskLayout Ly(max_dim);
    uint32_t *cnt = sm + Ly.cnt, *uw = sm + Ly.uw, *iu = sm + Ly.iu, *iw = sm + Ly.iw, *nu = sm + Ly.nu,
             *nw = sm + Ly.nw;
    double *ruw = reinterpret_cast<double *>(sm + Ly.ruw), *riu = reinterpret_cast<double *>(sm + Ly.riu),
           *riw = reinterpret_cast<double *>(sm + Ly.riw), *rnu = reinterpret_cast<double *>(sm + Ly.rnu),
           *rnw = reinterpret_cast<double *>(sm + Ly.rnw), *s_chi = reinterpret_cast<double *>(sm + Ly.chi);
    int *queue = reinterpret_cast<int *>(sm + Ly.queue);
    const int p = A.p, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const long long total = tasks[p];
    for (;;) {
        if (tid == 0) {
            s_task = (long long)atomicAdd(&st->units[1], 1ull);
            s_queued = 0;
        }
        __syncthreads();
        if (s_task >= total) return;
        const long long t = work_order(s_task, total, A.order);
        const int ri = upper_row(tasks, p, t), i = rows[ri];
        const int *nbrs = A.adj + (size_t)i * p + 1;
        const int deg = nbrs[-1];
        int di = A.dims[i];
        const int ng = (deg + Ly.vars - 1) / Ly.vars;
        int h = (int)(t - tasks[ri]), g = 0;
        while (h >= ng - g) h -= ng - g, ++g;
        h += g;
        if (!dcheck(st, g < ng && h < ng && deg < p, GCSL_DCHECK_SET)) g = h = 0;
        if (!dcheck(st, di >= 1 && di <= max_dim && off[i] + di - 1 <= off[p] && foff[i] + di <= ldf, GCSL_DCHECK_CELL))
            di = 1;
        // the two groups' variables, planes and values (warps 0 and 1)
        if (warp < 2) {
            const int g0 = (warp ? h : g) * Ly.vars, cntv = min(Ly.vars, deg - g0);
            int pc = 0, vc = 0;
            for (int k0 = 0; k0 < cntv; k0 += 32) {
                const int k = k0 + lane;
                int v = k < cntv ? nbrs[g0 + k] : 0;
                if (!dcheck(st, v >= 0 && v < p && (k >= cntv || v != i), GCSL_DCHECK_SET)) v = 0;
                int d = k < cntv ? A.dims[v] : 0;
                if (!dcheck(st, k >= cntv || (d >= 1 && d <= max_dim && off[v] + d - 1 <= off[p] && foff[v] + d <= ldf),
                            GCSL_DCHECK_CELL))
                    d = 0;
                int a = d > 1 ? d - 1 : 0, b = d;
                const int a1 = a, b1 = b;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int x = __shfl_up_sync(GCSL_FULL_MASK, a, o), y = __shfl_up_sync(GCSL_FULL_MASK, b, o);
                    if (lane >= o) a += x, b += y;
                }
                if (k < cntv) {
                    s_var[warp][k] = v;
                    s_pl[warp][k + 1] = pc + a;
                    s_va[warp][k + 1] = vc + b;
                    for (int e = 0; e < a1; ++e) {
                        s_plane[warp][pc + a - a1 + e] = off[v] + e;
                        s_at[warp][pc + a - a1 + e] = vc + b - b1 + e;
                    }
                    for (int e = 0; e < b1; ++e) s_value[warp][vc + b - b1 + e] = foff[v] + e;
                }
                pc += __shfl_sync(GCSL_FULL_MASK, a, 31);
                vc += __shfl_sync(GCSL_FULL_MASK, b, 31);
            }
            if (lane == 0) s_pl[warp][0] = s_va[warp][0] = 0;
        }
        const int vr = min(Ly.vars, deg - g * Ly.vars), vc = min(Ly.vars, deg - h * Ly.vars);
        __syncthreads();
        const int nr = s_pl[0][vr], nc = s_pl[1][vc], fr = s_va[0][vr], fc = s_va[1][vc];
        // pair tables of the task and their reciprocals
        const int fi = foff[i], ld = Ly.ld, vals = Ly.values, plane_sz = vals * ld;
        for (int k = tid; k < fr * fc; k += blockDim.x) {
            const int x = k / fc, y = k - x * fc;
            const size_t at = (size_t)s_value[0][x] * ldf + s_value[1][y];
            uw[x * ld + y] = __ldg(full + at);
            ruw[x * ld + y] = __ldg(inv + at);
        }
        for (int k = tid; k < di * fr; k += blockDim.x) {
            const int a = k / fr, x = k - a * fr;
            const size_t at = (size_t)(fi + a) * ldf + s_value[0][x];
            iu[a * vals + x] = __ldg(full + at);
            riu[a * vals + x] = __ldg(inv + at);
        }
        for (int k = tid; k < di * fc; k += blockDim.x) {
            const int a = k / fc, x = k - a * fc;
            const size_t at = (size_t)(fi + a) * ldf + s_value[1][x];
            iw[a * vals + x] = __ldg(full + at);
            riw[a * vals + x] = __ldg(inv + at);
        }
        for (int k = tid; k < fr; k += blockDim.x) {
            const size_t at = (size_t)s_value[0][k] * (ldf + 1);
            nu[k] = __ldg(full + at);
            rnu[k] = __ldg(inv + at);
        }
        for (int k = tid; k < fc; k += blockDim.x) {
            const size_t at = (size_t)s_value[1][k] * (ldf + 1);
            nw[k] = __ldg(full + at);
            rnw[k] = __ldg(inv + at);
        }
        for (int k = tid; k < (di - 1) * plane_sz; k += blockDim.x) cnt[k] = 0;
        __syncthreads();
        // counts: blocks of 4 x 4 planes per value of i; of a group with itself those of the
        // upper triangle.  Few blocks are cut into slices of the words.
        {
            const int br = (nr + BP_SIDE - 1) / BP_SIDE, bc = (nc + BP_SIDE - 1) / BP_SIDE;
            const int blocks = g == h ? br * (br + 1) / 2 : br * bc;
            const int items0 = blocks * (di - 1);
            if (items0 > 0) {
                const int per = slice_words(words, items0, 4 * nwarps), slices = (int)((words + per - 1) / per);
                const uint32_t mo = (uint32_t)((size_t)off[i] * words);
                for (int it = warp; it < items0 * slices; it += nwarps) {
                    const int sl = it % slices, ab = it / slices;
                    const int a = ab / blocks;
                    int b = ab - a * blocks, r = 0, c;
                    if (g == h) {
                        while (b >= bc - r) b -= bc - r, ++r;
                        c = r + b;
                    } else {
                        r = b / bc;
                        c = b - r * bc;
                    }
                    uint32_t ro[BP_SIDE], co[BP_SIDE];
#pragma unroll
                    for (int k = 0; k < BP_SIDE; ++k) {
                        ro[k] = (uint32_t)(s_plane[0][min(BP_SIDE * r + k, nr - 1)] * words);
                        co[k] = (uint32_t)(s_plane[1][min(BP_SIDE * c + k, nc - 1)] * words);
                    }
                    const int w0 = sl * per, w1 = (int)min((long long)w0 + per, words);
                    if (!dcheck(st, w0 < w1 && (w1 - w0) % BP_ROUND == 0, GCSL_DCHECK_CELL)) continue;
                    const uint32_t got =
                        popc_block<true>(planes, ro, co, mo + (uint32_t)(a * words), w0, (w1 - w0) / BP_ROUND);
                    const int x = BP_SIDE * r + lane / 4, y = BP_SIDE * c + lane % 4;
                    if (lane < 16 && x < nr && y < nc &&
                        dcheck(st, s_at[0][x] < fr && s_at[1][y] < fc, GCSL_DCHECK_CELL))
                        atomicAdd(cnt + a * plane_sz + s_at[0][x] * ld + s_at[1][y], got);
                }
            }
        }
        __syncthreads();
        // the last value of the column variable, of the row variable, and of i (of a group with
        // itself the pairs x >= y hold nothing of meaning and are not read)
        for (int k = tid; k < (di - 1) * nr * vc; k += blockDim.x) {
            const int y = k % vc, ar = k / vc, r = ar % nr, a = ar / nr;
            const int x0 = s_at[0][r], y0 = s_va[1][y], y1 = s_va[1][y + 1] - 1;
            uint32_t *row = cnt + a * plane_sz + x0 * ld, v = iu[a * vals + x0];
            for (int e = y0; e < y1; ++e) v -= row[e];
            if (y1 >= y0) row[y1] = v;
        }
        __syncthreads();
        for (int k = tid; k < (di - 1) * vr * fc; k += blockDim.x) {
            const int y = k % fc, ax = k / fc, x = ax % vr, a = ax / vr;
            const int x0 = s_va[0][x], x1 = s_va[0][x + 1] - 1;
            uint32_t *col = cnt + a * plane_sz + y, v = iw[a * vals + y];
            for (int e = x0; e < x1; ++e) v -= col[e * ld];
            if (x1 >= x0) col[x1 * ld] = v;
        }
        __syncthreads();
        for (int k = tid; k < fr * fc; k += blockDim.x) {
            const int x = k / fc, at = x * ld + (k - x * fc);
            uint32_t v = uw[at];
            for (int a = 0; a < di - 1; ++a) v -= cnt[a * plane_sz + at];
            cnt[(di - 1) * plane_sz + at] = v;
        }
        __syncthreads();
        // tests: pair (x, y) of neighbours, direction 0 (i, x | y), 1 (i, y | x)
        auto table = [&](int x, int y, int dir) {
            TripleTable T;
            const int vx = s_va[0][x], vy = s_va[1][y];
            const int dx = s_va[0][x + 1] - vx, dy = s_va[1][y + 1] - vy;
            T.cnt = cnt + vx * ld + vy;
            T.sa = plane_sz;
            T.uw = uw + vx * ld + vy;
            T.ruw = ruw + vx * ld + vy;
            T.di = di;
            T.lw = vals;
            if (dir == 0) {
                T.su = T.fu = ld, T.sw = T.fw = 1;
                T.iw = iw + vy, T.riw = riw + vy, T.nw = nw + vy, T.rnw = rnw + vy;
                T.du = dx, T.dw = dy;
            } else {
                T.su = T.fu = 1, T.sw = T.fw = ld;
                T.iw = iu + vx, T.riw = riu + vx, T.nw = nu + vx, T.rnw = rnu + vx;
                T.du = dy, T.dw = dx;
            }
            return T;
        };
        auto record = [&](int x, int y, int dir, double pv) {
            const int posx = g * Ly.vars + x, posy = h * Ly.vars + y;
            const int j = dir ? s_var[1][y] : s_var[0][x];
            const int pj = dir ? posy : posx, ps = dir ? posx : posy;
            const int lo = i < j ? i : j, hi = i < j ? j : i;
            const size_t ix = (size_t)lo * p + hi;
            atomic_max_nonneg(&A.pmax[ix], pv);
            if (pv >= A.alpha) {
                const unsigned long long rank = (unsigned long long)(ps - (ps > pj ? 1 : 0));
                atomicMin(&A.win[ix], (rank << 1) | (i < j ? 0ull : 1ull));
            }
        };
        const int gl = tid & (BP_LANES - 1), gw = tid / BP_LANES, groups = blockDim.x / BP_LANES;
        const unsigned mask = ((1u << BP_LANES) - 1u) << (lane & ~(BP_LANES - 1));
        const int pairs = g == h ? vr * (vr - 1) / 2 : vr * vc;
        for (int k = gw; k < 2 * pairs; k += groups) {
            int x, y, q = k >> 1;
            if (g == h) {
                x = 0;
                while (q >= vr - 1 - x) q -= vr - 1 - x, ++x;
                y = x + 1 + q;
            } else {
                x = q / vc;
                y = q - x * vc;
            }
            const TripleTable T = table(x, y, k & 1);
            const int df = (T.di - 1) * (T.du - 1) * T.dw;
            if (A.alpha > 0.0 && df > 0 && pvalue_zero(chi2_floor(T, gl, mask), df)) continue;
            if (gl == 0) {
                const int slot = atomicAdd(&s_queued, 1);
                if (dcheck(st, x < vr && y < vc && slot < 2 * Ly.vars * Ly.vars, GCSL_DCHECK_CELL))
                    queue[slot] = (x << 16) | (y << 1) | (k & 1);
            }
        }
        __syncthreads();
        const int queued = s_queued;
        for (int k = gw; k < queued; k += groups) {
            const int x = queue[k] >> 16, y = (queue[k] & 0xffff) >> 1, dir = queue[k] & 1;
            const double chi = chi2_exact(table(x, y, dir), gl, mask);
            if (gl == 0) s_chi[k] = chi;
        }
        __syncthreads();
        for (int k = tid; k < queued; k += blockDim.x) {
            const int x = queue[k] >> 16, y = (queue[k] & 0xffff) >> 1, dir = queue[k] & 1;
            const int dx = s_va[0][x + 1] - s_va[0][x], dy = s_va[1][y + 1] - s_va[1][y];
            const int df = (di - 1) * ((dir ? dy : dx) - 1) * (dir ? dx : dy);
            double pv = pchisq_tab(s_chi[k], df, lg);  // df < 1: 1
            if (df > 0 && pvalue_tie(s_chi[k], pv, A.alpha)) pv = pvalue_ordered(table(x, y, dir));
            record(x, y, dir, pv);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------- host
namespace host {

// The bit-plane path takes tables whose values all fit 16 x 16 pair tables and whose plane
// counts fit a 256 MB matrix; counts stay below 2^30 so that q is exact, and the planes
// (16 GB at most) below 2^32 words.
bool disc_bits_ok(long long n, int p, int max_dim) {
    return max_dim >= 2 && max_dim <= 16 && (long long)p * max_dim <= 8192 && n < (1ll << 30) &&
           (long long)p * (max_dim - 1) * bp_words(n) < (1ll << 32);
}

// Whether level 0 is counted on planes (three kernels, the first of them with the planes' words
// rounded up to whole passes) or with a table for each pair (two, cheap while the pairs are few).
// Where level 1 may follow on planes the lines lie where a solve of both levels takes the same,
// in the median over samples and graphs (planes with the better level 1, tables, us): 4 values:
// 16 variables 138, 133, 23 variables 185, 235; 8 values: 32 variables 349, 333; 10 values: 48
// variables 644, 604, 80 variables 1018, 1028.  With more values level 1 has its tables, and
// level 0 alone takes, 12 values, n = 2000: 40 variables 141, 98, 100 variables 168, 205; 16
// values, 200 variables: n = 10000 624, 644, n = 50000 1416, 928.
bool disc_bits_level0(long long n, int p, int max_dim) {
    if (max_dim <= 8) return p >= 10 + 4 * (max_dim - 2);
    return max_dim <= BP_LEVEL1_DIM ? p >= 64 : p >= 128 && n <= 16384;
}

// Whether level 1 may run on planes (the plan of the level decides, disc_level1_route).  With 12
// values it never paid (all tests of 23 .. 200 variables: 1.08 to 3.2 times the tables' time), with
// 10 it does where the graph is dense and n small (32 variables, n = 1000: 1521, 2562 us).
bool disc_bits_level1(int max_dim) { return max_dim <= BP_LEVEL1_DIM; }

int disc_bits_group(int max_dim) { return bp_group_vars(max_dim); }

size_t disc_lgam_doubles() { return 2 * LG_TERMS; }

size_t disc_bits_words(long long n, int p, int max_dim) { return (size_t)p * (max_dim - 1) * (size_t)bp_words(n); }

cudaError_t launch_disc_bits_level0(const DiscBits &b, const DiscLevelArgs &A, int num_sms, cudaStream_t s) {
    const int p = A.p, ldc = p * (b.max_dim - 1), ldf = p * b.max_dim;
    const long long words = bp_words(A.n);
    // 256 words a block and pass; about eight blocks per SM over all variables
    const long long want = (8ll * num_sms + p - 1) / p, most = (words + 255) / 256;
    const int chunks = (int)(want < 1 ? 1 : want > most ? most : want);
    // room left on every SM for concurrent solves: at most `cap` blocks of 256 threads on each
    const int cap = blocks_per_sm_cap();
    const int items = chunks * p + LG_BLOCKS;
    disc_planes_kernel<<<cap > 0 ? std::min(items, num_sms * cap) : items, 256, 0, s>>>(A.data, A.ld, A.n, p, A.dims, b.max_dim, chunks, b.planes,
                                                              words, b.card, b.off, b.foff, b.lg, b.counts,
                                                              (long long)ldc * ldc, A.st);
    disc_pair_counts_kernel<<<num_sms * (cap == 1 ? 1 : 2), 256, 0, s>>>(b.planes, words, b.off, p, b.counts, ldc, A.st);
    const long long pairs = (long long)p * (p + 1) / 2, lb = (pairs + BP_L0_GROUPS - 1) / BP_L0_GROUPS;
    const long long l0_per_sm = cap > 0 ? std::min(16, cap * (256 / BP_L0_THREADS)) : 16;
    disc_level0_kernel<<<(unsigned)std::min(lb, num_sms * l0_per_sm), BP_L0_THREADS, 0, s>>>(
        b.counts, ldc, p, b.card, b.off, b.foff, (uint32_t)A.n, b.full, b.inv, ldf, A.alpha, b.lg, A.G, A.pmax, A.st, A.order);
    note_launch(3);
    return note_error("discrete level 0 launch", cudaGetLastError());
}

cudaError_t launch_disc_bits_level1(const DiscBits &b, const DiscLevelArgs &A, const long long *tasks,
                                    const int *rows, int num_sms, cudaStream_t s) {
    const BitTaskLayout Ly(b.max_dim);
    const size_t smem = (size_t)Ly.words * sizeof(uint32_t);
    static std::atomic<unsigned long long> limit_set{0};
    const cudaError_t ea = raise_dyn_smem_limit(disc_bits_level1_kernel, limit_set);
    if (ea != cudaSuccess) return note_error("disc_bits_level1_kernel shared memory", ea);
    int per_sm = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, disc_bits_level1_kernel, BP_L1_THREADS, smem) !=
            cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    const int cap = blocks_per_sm_cap();  // room left on every SM for concurrent solves
    if (cap > 0 && per_sm > cap * (256 / BP_L1_THREADS)) per_sm = cap * (256 / BP_L1_THREADS);  // blocks of 256 threads
    DiscLevelArgs B = A;
    B.dims = b.card;
    disc_bits_level1_kernel<<<num_sms * per_sm, BP_L1_THREADS, smem, s>>>(b.planes, bp_words(A.n), b.off, b.foff, b.full, b.inv,
                                                                A.p * b.max_dim, tasks, rows, b.max_dim, b.lg, B);
    note_launch(1);
    return note_error("disc_bits_level1_kernel launch", cudaGetLastError());
}

}  // namespace host
}  // namespace gcsl
