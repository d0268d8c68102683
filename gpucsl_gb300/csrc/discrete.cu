// Discrete (chi-squared) PC-stable skeleton kernels for sm_103a (kernel d + write-back e).
//
//   tests          disc_test_kernel      (reference: gpucsl/pc/cuda/discrete_ci.cu:37-246,
//                                         helpers/discrete_helpers.cu:25-186)
//   p-value        disc_stat.cuh         (reference: helpers/math_helpers.cu:54-175)
//   write-back     disc_finalize_kernel  (reference: helpers/graph_helpers.cu:81-101)
//
// Levels 0 and 1 run on bit planes (disc_bits.cu) where those are faster (disc_bits_level0,
// disc_level1_route); the kernels here take the other levels, and these ones otherwise.
//
// One CTA evaluates one test at a time (grid-stride over the level's flattened test
// list): the l+2 uint8 columns are streamed with 16-byte loads and counted into a
// shared-memory table N[s][a][b] (several copies when the table is small, so that
// lanes of a warp rarely hit the same counter), the copies are merged, the threads take the
// table's cells one each at a time (table_chi2; tables wider than 32 values one stratum each, in
// the oracle's order), and a warp evaluates the p-value.  Counts are exact integers; the order of
// the chi^2 sum follows from the block's size alone, so results do not depend on scheduling.
//
// As in the reference every rank of every direction is tested (discrete_ci.cu:221-244
// has no effective early exit) and pmax folds all of them.  The removing test with the
// smallest key (rank, dir) is the canonical remover; its set becomes the sepset.
#include <algorithm>

#include "disc_stat.cuh"
#include "gauss_dev.cuh"  // block_scan_rows

namespace gcsl {

// ------------------------------------------------------------ test kernel

__device__ __forceinline__ void tri_pair(long long t, int &vi, int &vj) {
    // t -> (vi > vj), t = vi (vi - 1) / 2 + vj
    long long i = (long long)((1.0 + sqrt(1.0 + 8.0 * (double)t)) * 0.5);
    while (i * (i - 1) / 2 > t) --i;
    while ((i + 1) * i / 2 <= t) ++i;
    vi = (int)i;
    vj = (int)(t - i * (i - 1) / 2);
}

// Count the table N[s][a][b] of one test into shared memory (all threads of the CTA).
// S / mult live in shared memory; `copies` replicas of T counters are merged into the
// first one before returning.
//
// `trusted`: every code of every column is below its cardinality (checked once per
// solve by disc_validate_kernel), so no sample needs a range check.  Tables of at most
// 256 cells then take the packed path: with every code in range each byte lane of
// ((sum_k s_k m_k) * di + a) * dj + b stays below T <= 256, so 32-bit multiplies and
// adds on four samples' bytes at once carry nothing between lanes and give the four
// cell indices of the scalar formula.
__device__ void count_table(const uint8_t *__restrict__ data, long long ld, long long n, int vi, int vj,
                            const int *S, const int *mult, int L, int di, int dj, int T, int copies,
                            uint32_t *sm_tab, int *bad, bool trusted) {
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int k = tid; k < T * copies; k += nt) sm_tab[k] = 0;
    __syncthreads();
    uint32_t *tab = sm_tab + (size_t)(tid % copies) * T;
    const uint4 *ci = reinterpret_cast<const uint4 *>(data + (size_t)vi * ld);
    const uint4 *cj = reinterpret_cast<const uint4 *>(data + (size_t)vj * ld);
    const long long nvec = (n + 15) >> 4;
    // the debug build always takes the checked path below (every cell index is checked)
    if (trusted && T <= 256 && !GCSL_DEBUG_CHECKS) {
        const long long nfull = n >> 4;  // vectors of 16 samples, all valid
        for (long long v = tid; v < nfull; v += nt) {
            uint32_t s4[4] = {0u, 0u, 0u, 0u};
            for (int k = 0; k < L; ++k) {
                const uint4 w = __ldg(reinterpret_cast<const uint4 *>(data + (size_t)S[k] * ld) + v);
                const uint32_t mk = (uint32_t)mult[k];
                s4[0] += w.x * mk;
                s4[1] += w.y * mk;
                s4[2] += w.z * mk;
                s4[3] += w.w * mk;
            }
            const uint4 xi = __ldg(ci + v), xj = __ldg(cj + v);
            const uint32_t idx4[4] = {(s4[0] * (uint32_t)di + xi.x) * (uint32_t)dj + xj.x,
                                      (s4[1] * (uint32_t)di + xi.y) * (uint32_t)dj + xj.y,
                                      (s4[2] * (uint32_t)di + xi.z) * (uint32_t)dj + xj.z,
                                      (s4[3] * (uint32_t)di + xi.w) * (uint32_t)dj + xj.w};
#pragma unroll
            for (int q = 0; q < 16; ++q) atomicAdd(&tab[(idx4[q >> 2] >> (8 * (q & 3))) & 0xffu], 1u);
        }
        // the last, partial vector
        if (tid == 0 && (n & 15)) {
            const long long v = nfull;
            const int nvalid = (int)(n & 15);
            for (int q = 0; q < nvalid; ++q) {
                const size_t off = (size_t)(v << 4) + q;
                int sidx = 0;
                for (int k = 0; k < L; ++k) sidx += (int)data[(size_t)S[k] * ld + off] * mult[k];
                const int a = data[(size_t)vi * ld + off], b = data[(size_t)vj * ld + off];
                atomicAdd(&tab[(sidx * di + a) * dj + b], 1u);
            }
        }
    } else
    for (long long v = tid; v < nvec; v += nt) {
        int sidx[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) sidx[q] = 0;
        for (int k = 0; k < L; ++k) {
            const uint4 w = __ldg(reinterpret_cast<const uint4 *>(data + (size_t)S[k] * ld) + v);
            const int mk = mult[k];
            const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int q = 0; q < 16; ++q) sidx[q] += (int)((ww[q >> 2] >> (8 * (q & 3))) & 0xffu) * mk;
        }
        const uint4 xi = __ldg(ci + v), xj = __ldg(cj + v);
        const uint32_t wi[4] = {xi.x, xi.y, xi.z, xi.w};
        const uint32_t wj[4] = {xj.x, xj.y, xj.z, xj.w};
        const long long rem = n - (v << 4);
        const int nvalid = rem >= 16 ? 16 : (int)rem;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            if (q < nvalid) {
                const int a = (int)((wi[q >> 2] >> (8 * (q & 3))) & 0xffu);
                const int b = (int)((wj[q >> 2] >> (8 * (q & 3))) & 0xffu);
                const int idx = (sidx[q] * di + a) * dj + b;
                // codes at or above their cardinality are invalid input: never written
                if ((unsigned)idx < (unsigned)T && a < di && b < dj) atomicAdd(&tab[idx], 1u);
                else *bad = 1;
            }
        }
    }
    __syncthreads();
    if (copies > 1) {
        for (int k = tid; k < T; k += nt) {
            uint32_t s = 0;
            for (int c = 0; c < copies; ++c) s += sm_tab[(size_t)c * T + k];
            sm_tab[k] = s;
        }
        __syncthreads();
    }
}

// chi^2 partial sum of one stratum, (a, b) order; E = N_a+ N_+b / N_++, terms with
// N_++ == 0 or E == 0 skipped (discrete_helpers.cu:164-186).
__device__ double stratum_chi2(const uint32_t *Ts, int di, int dj) {
    double part = 0.0;
    if (di <= 16 && dj <= 16) {
        uint32_t ma[16], mb[16];
        uint32_t mt = 0;
#pragma unroll
        for (int a = 0; a < 16; ++a) ma[a] = mb[a] = 0;
        for (int a = 0; a < di; ++a)
            for (int b = 0; b < dj; ++b) {
                const uint32_t o = Ts[a * dj + b];
                ma[a] += o;
                mb[b] += o;
                mt += o;
            }
        if (mt == 0) return 0.0;
        for (int a = 0; a < di; ++a)
            for (int b = 0; b < dj; ++b) {
                const double e = __ddiv_rn(__dmul_rn((double)ma[a], (double)mb[b]), (double)mt);
                if (e == 0.0) continue;
                const double d = __dsub_rn((double)Ts[a * dj + b], e);
                part = __dadd_rn(part, __ddiv_rn(__dmul_rn(d, d), e));
            }
        return part;
    }
    // wide tables: the marginals are recomputed from the table (same integers)
    uint32_t mt = 0;
    for (int k = 0; k < di * dj; ++k) mt += Ts[k];
    if (mt == 0) return 0.0;
    for (int a = 0; a < di; ++a) {
        uint32_t ma = 0;
        for (int b = 0; b < dj; ++b) ma += Ts[a * dj + b];
        for (int b = 0; b < dj; ++b) {
            uint32_t mb = 0;
            for (int a2 = 0; a2 < di; ++a2) mb += Ts[a2 * dj + b];
            const double e = __ddiv_rn(__dmul_rn((double)ma, (double)mb), (double)mt);
            if (e == 0.0) continue;
            const double d = __dsub_rn((double)Ts[a * dj + b], e);
            part = __dadd_rn(part, __ddiv_rn(__dmul_rn(d, d), e));
        }
    }
    return part;
}

// Statistic of the counted table in the oracle's order: strata by one thread each, then
// added in ascending order; every thread returns the sum.  The unit entry point's, and the
// test kernel's for tables too wide for table_chi2.
__device__ double table_chi2_ordered(const uint32_t *sm_tab, int dim_s, int di, int dj, double *s_part) {
    for (int s = threadIdx.x; s < dim_s; s += blockDim.x)
        s_part[s] = stratum_chi2(sm_tab + (size_t)s * di * dj, di, dj);
    __syncthreads();
    double chi = 0.0;
    for (int s = 0; s < dim_s; ++s) chi = __dadd_rn(chi, s_part[s]);
    __syncthreads();
    return chi;
}

// Statistic of the counted table, all threads of the block; every thread returns the sum.
// With di, dj <= 32 a thread takes one cell at a time, its marginals summed from the table
// (integers) and the stratum totals from s_part: q = N N_s - N_a N_b is an exact integer and
// the cell adds q^2 / (N_a N_b N_s).  A cell costs one FP64 division (GB300's FP64 pipe is
// 1/64 of its FP32 pipe) and all lanes stay busy; a warp per stratum with its terms added in
// order took two divisions and a serial chain of additions.  Before that, a lower bound of
// the sum in FP32 ends tests whose p-value is certainly zero (pvalue_zero; `zero_ok`: a zero
// p-value changes nothing): *zero is set and 0 returned.
__device__ double table_chi2(const uint32_t *sm_tab, int dim_s, int di, int dj, double *s_part, bool zero_ok,
                             bool *zero) {
    __shared__ double s_red[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    *zero = false;
    if (di > 32 || dj > 32) return table_chi2_ordered(sm_tab, dim_s, di, dj, s_part);
    double chi = 0.0;
    uint32_t *s_mt = reinterpret_cast<uint32_t *>(s_part);
    const int per = di * dj, cells = dim_s * per;
    for (int s = warp; s < dim_s; s += nwarps) {
        uint32_t m = 0;
        for (int k = lane; k < per; k += 32) m += sm_tab[s * per + k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(GCSL_FULL_MASK, m, o);
        if (lane == 0) s_mt[s] = m;
    }
    __syncthreads();
    auto marginals = [&](int k, int &s, uint32_t &ma, uint32_t &mb) {
        s = k / per;
        const int r = k - s * per, a = r / dj, b = r - a * dj;
        const uint32_t *t = sm_tab + s * per;
        ma = mb = 0;
        for (int y = 0; y < dj; ++y) ma += t[a * dj + y];
        for (int x = 0; x < di; ++x) mb += t[x * dj + b];
    };
    const int df = (di - 1) * (dj - 1) * dim_s;
    if (zero_ok && df > 0) {
        float f = 0.f;
        for (int k = tid; k < cells; k += blockDim.x) {
            int s;
            uint32_t ma, mb;
            marginals(k, s, ma, mb);
            if (ma == 0 || mb == 0) continue;
            const float e = __fdividef((float)ma * (float)mb, (float)s_mt[s]), o = (float)sm_tab[k];
            f += chi2_floor_term(o, e);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(GCSL_FULL_MASK, f, o);
        if (lane == 0) s_red[warp] = (double)f;
        __syncthreads();
        float sum = 0.f;
        for (int w = 0; w < nwarps; ++w) sum += (float)s_red[w];
        __syncthreads();
        if (pvalue_zero(0.999f * sum, df)) {
            *zero = true;
            return 0.0;
        }
    }
    for (int k = tid; k < cells; k += blockDim.x) {
        int s;
        uint32_t ma, mb;
        marginals(k, s, ma, mb);
        if (ma == 0 || mb == 0) continue;
        // unsigned: a product of two counts of up to 2^32 samples; |q| is at most a quarter of it
        const unsigned long long e = (unsigned long long)ma * mb;
        const long long q = (long long)((unsigned long long)sm_tab[k] * s_mt[s] - e);
        chi += (double)q * (double)q / ((double)e * (double)s_mt[s]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) chi += __shfl_xor_sync(GCSL_FULL_MASK, chi, o);
    if (lane == 0) s_red[warp] = chi;
    __syncthreads();
    chi = 0.0;
    for (int w = 0; w < nwarps; ++w) chi += s_red[w];
    __syncthreads();
    return chi;
}

// P-value of the counted table in the published order, by one thread (tests on a jump of the
// p-value).
__device__ __noinline__ double table_pvalue_ordered(const uint32_t *sm_tab, int dim_s, int di, int dj) {
    double chi = 0.0;
    for (int s = 0; s < dim_s; ++s) chi = __dadd_rn(chi, stratum_chi2(sm_tab + (size_t)s * di * dj, di, dj));
    return pchisq_dev(chi, (long long)(di - 1) * (long long)(dj - 1) * (long long)dim_s);
}

// Per-test header prepared by thread 0: table geometry and replica count.
__device__ __forceinline__ bool table_geometry(const uint8_t *dims, const int *S, int *mult, int L, int vi, int vj,
                                               int table_cap, int part_cap, int &dim_s, int &di, int &dj,
                                               int &copies) {
    long long ds = 1;
    for (int k = 0; k < L; ++k) {
        mult[k] = (int)ds;
        ds *= dims[S[k]];
        if (ds > table_cap) return false;
    }
    di = dims[vi];
    dj = dims[vj];
    const long long T = ds * di * dj;
    if (T > table_cap || ds > part_cap) return false;
    dim_s = (int)ds;
    copies = 1;
    if (T <= table_cap / 8) copies = 8;
    else if (T <= table_cap / 4) copies = 4;
    else if (T <= table_cap / 2) copies = 2;
    return true;
}

// Threads of the test kernel: 256 at level 0 (many small tests), 512 above, where the tests
// are few and large and the block is the parallelism of a test.
constexpr int DISC_THREADS = 512;

__global__ void __launch_bounds__(DISC_THREADS) disc_test_kernel(DiscLevelArgs A) {
    extern __shared__ uint32_t sm_tab[];
    struct Header {
        int S[GCSL_MAX_LEVELS + 2], mult[GCSL_MAX_LEVELS + 2];
        int vi, vj, di, dj, dim_s, copies, ok;
        long long rank;
    };
    __shared__ Header s_hdr[2];
    __shared__ int s_bad;
    // per-stratum statistics follow the counters (8-byte aligned)
    double *s_part = reinterpret_cast<double *>(sm_tab + ((A.table_cap + 1) & ~1));
    __shared__ int s_trusted;
    DevState *st = A.st;
    pdl_wait();  // every thread: what follows this kernel must find the one before it complete
    if (threadIdx.x == 0) {
        s_bad = 0;
        // codes checked in range for this solve: disc_validate_kernel (or the plane writer) ran
        // before level 0 and leaves the status 0 only then (any other error also selects the
        // checked path); read once per CTA, seen by all threads after the first barrier below
        s_trusted = *(volatile const int32_t *)&st->status == 0;
    }
    const int L = A.level;
    if (L > 0) {
        if (st->done) return;
        const int md = st->max_degree[L];
        if (md - 1 < L) {
            if (blockIdx.x == 0 && threadIdx.x == 0) st->done = 1;
            return;
        }
        if (A.routed && st->disc_route == 0) return;
        if (blockIdx.x == 0 && threadIdx.x == 0) st->last_level = L;
    }
    const long long total = (L == 0) ? (long long)A.p * (A.p - 1) / 2 : A.prefix[A.p];
    const int tid = threadIdx.x;

    // test t0's variables and table geometry (one thread)
    auto prepare = [&](long long t0, Header &H) {
        const long long t = work_order(t0, total, A.order);
        int vi, vj;
        long long rank = 0;
        if (L == 0) {
            tri_pair(t, vi, vj);
        } else {
            vi = upper_row(A.prefix, A.p, t);
            const long long off = t - A.prefix[vi];
            const int deg = A.adj[(size_t)vi * A.p];
            const long long R = binom_rt(deg - 1, L);
            const int m = (int)(off / R);
            rank = off - (long long)m * R;
            vj = A.adj[(size_t)vi * A.p + 1 + m];
            unrank_positions_rt(L, deg - 1, rank, H.S);
            const int *nbrs = A.adj + (size_t)vi * A.p + 1;
            for (int c = 0; c < L; ++c) H.S[c] = resolve_position(nbrs, vj, H.S[c]);
        }
        int dim_s = 0, di = 0, dj = 0, copies = 1;
        const bool ok =
            table_geometry(A.dims, H.S, H.mult, L, vi, vj, A.table_cap, A.part_cap, dim_s, di, dj, copies);
        H.vi = vi;
        H.vj = vj;
        H.di = di;
        H.dj = dj;
        H.dim_s = dim_s;
        H.copies = copies;
        H.ok = ok;
        H.rank = rank;
        if (!ok) set_status(st, GCSL_ERR_UNSUPPORTED);
    };

    // the next test's header is prepared by the last warp while the others start on this one's
    // statistic
    if (tid == 0 && blockIdx.x < total) prepare(blockIdx.x, s_hdr[0]);
    int cur = 0;
    for (long long t0 = blockIdx.x; t0 < total; t0 += gridDim.x, cur ^= 1) {
        __syncthreads();
        const Header &H = s_hdr[cur];
        const bool more = t0 + gridDim.x < total;
        const int ahead = blockDim.x - 32;  // the thread that prepares
        if (!H.ok) {
            if (tid == ahead && more) prepare(t0 + gridDim.x, s_hdr[cur ^ 1]);
            continue;
        }
        const int vi = H.vi, vj = H.vj, di = H.di, dj = H.dj, dim_s = H.dim_s;
        count_table(A.data, A.ld, A.n, vi, vj, H.S, H.mult, L, di, dj, dim_s * di * dj, H.copies, sm_tab, &s_bad,
                    s_trusted != 0);
        if (tid == ahead && more) prepare(t0 + gridDim.x, s_hdr[cur ^ 1]);
        bool zero;
        const double chi = table_chi2(sm_tab, dim_s, di, dj, s_part, A.alpha > 0.0, &zero);
        if (tid == 0 && s_bad) set_status(st, GCSL_ERR_INVALID_ARG);
        double pv = 0.0;
        if (!zero && tid < 32) {  // warp 0: the p-value's series split over the lanes
            const long long df = (long long)(di - 1) * (long long)(dj - 1) * (long long)dim_s;
            pv = pchisq_tab_warp(chi, df, A.lg);
            if (tid == 0 && df > 0 && pvalue_tie(chi, pv, A.alpha)) pv = table_pvalue_ordered(sm_tab, dim_s, di, dj);
        }
        if (tid == 0) {
            const int lo = vi < vj ? vi : vj, hi = vi < vj ? vj : vi;
            const size_t ix = (size_t)lo * A.p + hi;
            if (L == 0) {
                A.pmax[ix] = pv;
                const uint16_t keep = (pv >= A.alpha) ? 0 : 1;
                A.G[(size_t)vi * A.p + vj] = keep;
                A.G[(size_t)vj * A.p + vi] = keep;
            } else if (!zero) {
                atomic_max_nonneg(&A.pmax[ix], pv);
                if (pv >= A.alpha) {
                    const unsigned long long key = ((unsigned long long)H.rank << 1) | (vi < vj ? 0ull : 1ull);
                    atomicMin(&A.win[ix], key);
                }
            }
        }
    }
    if (blockIdx.x == 0 && tid == 0) st->tests[L] = (unsigned long long)total;
}

// One test for the unit entry point: counts and (chi^2, p-value) to global memory.
struct UnitSet {
    int S[GCSL_MAX_LEVELS];
};

__global__ void __launch_bounds__(256) disc_table_kernel(const uint8_t *data, long long ld, long long n,
                                                         const uint8_t *dims, int vi, int vj, UnitSet us, int L,
                                                         int table_cap, uint32_t *counts, long long counts_cap,
                                                         double *out2) {
    extern __shared__ uint32_t sm_tab[];
    __shared__ int s_S[GCSL_MAX_LEVELS + 2];
    __shared__ int s_mult[GCSL_MAX_LEVELS + 2];
    __shared__ int s_hdr[4];
    __shared__ double s_part[1024];
    if (threadIdx.x == 0) {
        for (int k = 0; k < L; ++k) s_S[k] = us.S[k];
        int dim_s = 0, di = 0, dj = 0, copies = 1;
        bool ok = table_geometry(dims, s_S, s_mult, L, vi, vj, table_cap, 1024, dim_s, di, dj, copies);
        if (ok && (long long)dim_s * di * dj > counts_cap) ok = false;  // never write past the caller's buffer
        s_hdr[0] = ok ? dim_s : -1;
        s_hdr[1] = di;
        s_hdr[2] = dj;
        s_hdr[3] = copies;
    }
    __syncthreads();
    const int dim_s = s_hdr[0], di = s_hdr[1], dj = s_hdr[2];
    if (dim_s < 0) {
        if (threadIdx.x == 0) out2[0] = out2[1] = -1.0;
        return;
    }
    const int T = dim_s * di * dj;
    __shared__ int s_bad;
    if (threadIdx.x == 0) s_bad = 0;
    count_table(data, ld, n, vi, vj, s_S, s_mult, L, di, dj, T, s_hdr[3], sm_tab, &s_bad, false);
    for (int k = threadIdx.x; k < T; k += blockDim.x) counts[k] = sm_tab[k];
    const double chi = table_chi2_ordered(sm_tab, dim_s, di, dj, s_part);
    if (threadIdx.x == 0) {
        if (s_bad) {
            out2[0] = out2[1] = -1.0;
            return;
        }
        out2[0] = chi;
        out2[1] = pchisq_dev(chi, (long long)(di - 1) * (long long)(dj - 1) * (long long)dim_s);
    }
}

// Codes in range: every code of columns 0..p-1 (samples 0..n-1) below its cardinality.
// Sets GCSL_ERR_INVALID_ARG otherwise, which makes the test kernels check every sample.
// A byte x of a word is >= d (1 <= d <= 128) iff the high bit of (x + 128 - d) | x is
// set; with all bytes below d nothing carries between bytes, and a byte >= 128 (which
// may carry) has its own high bit set, so the word test is exact.
__global__ void __launch_bounds__(256) disc_validate_kernel(const uint8_t *__restrict__ data, long long ld,
                                                            long long n, int p, const uint8_t *__restrict__ dims,
                                                            double *__restrict__ lg, DevState *st) {
    if (blockIdx.x < LG_BLOCKS) lgam_build(lg, (int)blockIdx.x);
    const long long nvec = (n + 15) >> 4;
    const long long total = nvec * p;
    bool bad = false;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int col = (int)(i / nvec);
        const long long v = i - (long long)col * nvec;
        const uint32_t d = dims[col];
        const uint4 w = __ldg(reinterpret_cast<const uint4 *>(data + (size_t)col * ld) + v);
        const long long rem = n - (v << 4);
        if (d == 0 || d > 128 || rem < 16) {  // rare: byte by byte
            const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
            const int nvalid = rem >= 16 ? 16 : (int)rem;
            for (int q = 0; q < nvalid; ++q) bad |= ((ww[q >> 2] >> (8 * (q & 3))) & 0xffu) >= d;
        } else {
            const uint32_t add = (0x80u - d) * 0x01010101u;
            const uint32_t hit = (((w.x + add) | w.x) | ((w.y + add) | w.y) | ((w.z + add) | w.z) |
                                  ((w.w + add) | w.w)) & 0x80808080u;
            bad |= hit != 0;
        }
    }
    if (__any_sync(GCSL_FULL_MASK, bad) && (threadIdx.x & 31) == 0) set_status(st, GCSL_ERR_INVALID_ARG);
}

// Level 1: 0 when its `tests` are faster on bit planes, 1 when a table for each is.  Times in
// microseconds of both ways, from what bounds each.  Planes: the longest task (`task` passes of
// 64 words by one block, which waits for its loads) or all tasks' passes (`passes`), and the
// statistics: their cells, or one test's series, whose terms a thread adds one by one.  Tables:
// one test's pass over the samples, or all tests'.
//
// The constants fit both ways' times over 594 problems of 2 .. 10 values, 10 .. 300 variables,
// 200 .. 500000 samples and sparse to complete graphs: by this rule a solve takes 0.4 % longer
// than by the better way on average, 24 % in the worst of them.  Levels 0 and 1 on planes and by
// tables: 8 values, 23 variables, n = 200000, 354 tests: 2176, 251 us; 40 variables, n = 10000,
// all 59280 tests: 890, 1904 us.
__device__ __forceinline__ int disc_level1_route(float tests, float task, float passes, int max_dim, float mean_planes,
                                                 float n) {
    const float d = (float)max_dim, m = mean_planes + 1.0f;
    const float planes = 8.0f + fmaxf(0.14f * task, passes * (1.0f / 4600.0f)) +
                         fmaxf(1.2e-5f * tests * m * m * m, 0.26f * d * d * d);
    const float tables = 15.0f + fmaxf(1.7e-4f * n, tests * (0.05f + 7.3e-7f * n));
    return planes < tables ? 0 : 1;
}

// One block plans a level: per-row test counts deg C(deg - 1, L) and their exclusive prefix,
// the edge and test totals, and with group > 0 the bit-plane path's tasks (pairs of a row's
// neighbour groups of `group` variables): `rows` lists the rows by falling work, about d deg^2,
// so that the uneven tasks are started largest first, and `tasks` is the prefix of their task
// counts in that order.  From these it chooses the level's route (max_dim: the largest
// cardinality; planes: the planes before each variable).
__global__ void __launch_bounds__(1024) disc_plan_kernel(const int *__restrict__ adj, int p, int L, int group,
                                                         int max_dim, long long n, const int *__restrict__ planes,
                                                         const uint8_t *__restrict__ dims, long long *__restrict__ w,
                                                         long long *__restrict__ prefix, long long *__restrict__ tasks,
                                                         int *__restrict__ rows, DevState *st) {
    extern __shared__ long long s_key[];
    __shared__ unsigned long long s_task, s_passes;
    if (st->done) return;
    if (threadIdx.x == 0) s_task = s_passes = 0ull;
    unsigned long long edges = 0;
    for (int r = threadIdx.x; r < p; r += blockDim.x) {
        const int deg = adj[(size_t)r * p];
        const long long R = (deg - 1 >= L) ? binom_rt(deg - 1, L) : 0;
        if (R >= GCSL_RANK_LIMIT) set_status(st, GCSL_ERR_UNSUPPORTED);
        w[r] = (long long)deg * R;
        edges += (unsigned long long)deg;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) edges += __shfl_xor_sync(GCSL_FULL_MASK, edges, o);
    if ((threadIdx.x & 31) == 0 && edges) atomicAdd(&st->edges[L], edges);  // directed count; halved on the host
    __syncthreads();
    block_scan_rows(w, p, prefix);
    __syncthreads();
    if (threadIdx.x == 0) st->tests_full[L] = (unsigned long long)prefix[p];
    if (group <= 0) return;
    const float mean = (float)planes[p] / (float)p;  // planes of a variable
    const long long words = (n + 2047) / 2048;       // passes of 64 words over the samples
    unsigned long long longest = 0ull, passes = 0ull;
    for (int r = threadIdx.x; r < p; r += blockDim.x) {
        const long long deg = adj[(size_t)r * p];
        s_key[r] = w[r] > 0 ? deg * deg * dims[r] : 0;
        if (w[r] > 0) {  // blocks of 4 x 4 planes of two groups, for every value of the row's variable but the last
            const long long side = (long long)ceilf(0.25f * mean * (float)min((long long)group, deg));
            const long long ng = (deg + group - 1) / group, task = side * side * (dims[r] - 1) * words;
            longest = max(longest, (unsigned long long)task);
            passes += (unsigned long long)(task * (ng * (ng + 1) / 2));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        longest = max(longest, __shfl_xor_sync(GCSL_FULL_MASK, longest, o));
        passes += __shfl_xor_sync(GCSL_FULL_MASK, passes, o);
    }
    if ((threadIdx.x & 31) == 0 && passes) {
        atomicMax(&s_task, longest);
        atomicAdd(&s_passes, passes);
    }
    __syncthreads();
    if (threadIdx.x == 0)
        st->disc_route = disc_level1_route((float)prefix[p], (float)s_task, (float)s_passes, max_dim, mean, (float)n);
    for (int r = threadIdx.x; r < p; r += blockDim.x) {
        const long long key = s_key[r];
        int rank = 0;
        for (int q = 0; q < p; ++q) rank += s_key[q] > key || (s_key[q] == key && q < r);
        const long long ng = key > 0 ? (adj[(size_t)r * p] + group - 1) / group : 0;
        rows[rank] = r;
        w[rank] = ng * (ng + 1) / 2;
    }
    __syncthreads();
    block_scan_rows(w, p, tasks);
}

// Write-back of a level: canonical remover -> skeleton, sepsets, records.
__global__ void disc_finalize_kernel(const int *__restrict__ adj, int p, int L, uint16_t *G,
                                     unsigned long long *win, int *sep_dense, int max_level, int *rec_pool,
                                     long long rec_cap, DevState *st) {
    if (st->done) return;
    if (st->max_degree[L] - 1 < L) return;
    const long long total = (long long)p * p;
    unsigned long long removed = 0;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
         k += (long long)gridDim.x * blockDim.x) {
        const unsigned long long key = win[k];
        if (key == GCSL_KEY_NONE) continue;
        win[k] = GCSL_KEY_NONE;
        const int lo = (int)(k / p), hi = (int)(k - (long long)lo * p);
        const long long rank = (long long)(key >> 1);
        const int vi = (key & 1) ? hi : lo, vj = (key & 1) ? lo : hi;
        const int *row = adj + (size_t)vi * p;
        int S[GCSL_MAX_LEVELS];
        unrank_positions_rt(L, row[0] - 1, rank, S);
        for (int c = 0; c < L; ++c) S[c] = resolve_position(row + 1, vj, S[c]);
        G[(size_t)lo * p + hi] = 0;
        G[(size_t)hi * p + lo] = 0;
        if (sep_dense != nullptr && L <= max_level) {
            for (int c = 0; c < L; ++c) {
                sep_dense[((size_t)lo * p + hi) * max_level + c] = S[c];
                sep_dense[((size_t)hi * p + lo) * max_level + c] = S[c];
            }
        }
        if (rec_pool != nullptr) {
            const unsigned long long off = atomicAdd(&st->n_rec_ints, (unsigned long long)(3 + L));
            if ((long long)(off + 3 + L) <= rec_cap) {
                rec_pool[off] = lo;
                rec_pool[off + 1] = hi;
                rec_pool[off + 2] = L;
                for (int c = 0; c < L; ++c) rec_pool[off + 3 + c] = S[c];
            } else {
                set_status(st, GCSL_ERR_CAPACITY);
            }
        }
        ++removed;
    }
    if (removed) atomicAdd(&st->removed[L], removed);
}

__global__ void pmax_finish_kernel(double *pmax, int p) {
    const long long total = (long long)p * p;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
         k += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(k / p), j = (int)(k - (long long)i * p);
        if (i >= j) pmax[k] = -1.0;
    }
}

// Unit entry point kernels -------------------------------------------------
__global__ void pchisq_kernel(const double *x, const long long *df, long long count, double *out) {
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < count;
         k += (long long)gridDim.x * blockDim.x)
        out[k] = pchisq_dev(x[k], df[k]);
}

namespace host {

int disc_table_cap(int device) {
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    // leave room for the static shared arrays of the kernels and 1024 strata statistics
    const int dyn = optin - 16 * 1024;
    return dyn / (int)sizeof(uint32_t);
}

// Shared memory of one level's tables: the largest table of the level has at most
// max_dim^(L+2) counters; small tables get replicas (fewer atomic collisions) while the
// footprint stays small enough for several CTAs per SM.  Levels whose largest table
// would not fit take the whole budget.
void disc_level_caps(int cap_full, int max_dim, int L, int &table_cap, int &part_cap) {
    long long need = 1, ds = 1;
    for (int k = 0; k < L + 2 && need <= cap_full; ++k) {
        need *= max_dim;
        if (k < L) ds *= max_dim;
    }
    if (need > cap_full || ds > 1024) {
        table_cap = cap_full;
        part_cap = 1024;
        return;
    }
    const long long reps = need <= 512 ? 8 : need <= 2048 ? 4 : need <= 8192 ? 2 : 1;
    table_cap = (int)(need * reps < cap_full ? need * reps : cap_full);
    part_cap = (int)ds;
}

cudaError_t launch_disc_tests(const DiscLevelArgs &A, int num_sms, cudaStream_t s) {
    const size_t smem = (size_t)((A.table_cap + 1) & ~1) * sizeof(uint32_t) + (size_t)A.part_cap * sizeof(double);
    static std::atomic<unsigned long long> limit_set{0};
    const cudaError_t ea = raise_dyn_smem_limit(disc_test_kernel, limit_set);
    if (ea != cudaSuccess) return note_error("disc_test_kernel shared memory", ea);
    int per_sm = 1;
    const int threads = A.level == 0 ? DISC_THREADS / 2 : DISC_THREADS;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, disc_test_kernel, threads, smem) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    const int cap = blocks_per_sm_cap();  // room left on every SM for concurrent solves
    if (cap > 0 && per_sm > cap) per_sm = cap;
    note_launch(1);
    // behind the bit-plane kernel it often has nothing to do: its launch overlaps that one's end
    if (A.routed)
        return note_error("disc_test_kernel launch", launch_pdl(disc_test_kernel, dim3((unsigned)(num_sms * per_sm)),
                                                                dim3((unsigned)threads), smem, s, A));
    disc_test_kernel<<<num_sms * per_sm, threads, smem, s>>>(A);
    return note_error("disc_test_kernel launch", cudaGetLastError());
}

// Also builds the ln Gamma tables (at least LG_BLOCKS blocks: num_sms >= 1).
cudaError_t launch_disc_validate(const uint8_t *data, long long ld, long long n, int p, const uint8_t *dims,
                                 double *lg, DevState *st, int num_sms, cudaStream_t s) {
    disc_validate_kernel<<<std::max(num_sms * 4, LG_BLOCKS), 256, 0, s>>>(data, ld, n, p, dims, lg, st);
    note_launch(1);
    return note_error("disc_validate_kernel launch", cudaGetLastError());
}

// group: neighbours per group of the bit-plane path's level 1 (0: no tasks).
cudaError_t launch_disc_plan(const int *adj, int p, int L, int group, int max_dim, long long n, const int *planes,
                             const uint8_t *dims, long long *w, long long *prefix, long long *tasks, int *rows,
                             DevState *st, cudaStream_t s) {
    const size_t smem = group > 0 ? (size_t)p * sizeof(long long) : 0;  // p <= 4096 with groups
    disc_plan_kernel<<<1, 1024, smem, s>>>(adj, p, L, group, max_dim, n, planes, dims, w, prefix, tasks, rows, st);
    note_launch(1);
    return cudaGetLastError();
}

cudaError_t launch_disc_finalize(const int *adj, int p, int L, uint16_t *G, unsigned long long *win, int *sep,
                                 int max_level, int *rec, long long rec_cap, DevState *st, int num_sms,
                                 cudaStream_t s) {
    disc_finalize_kernel<<<num_sms * 2, 256, 0, s>>>(adj, p, L, G, win, sep, max_level, rec, rec_cap, st);
    note_launch(1);
    return cudaGetLastError();
}

cudaError_t launch_pmax_finish(double *pmax, int p, int num_sms, cudaStream_t s) {
    pmax_finish_kernel<<<num_sms * 2, 256, 0, s>>>(pmax, p);
    note_launch(1);
    return cudaGetLastError();
}

cudaError_t launch_disc_table(const uint8_t *data, long long ld, long long n, const uint8_t *dims, int vi, int vj,
                              const int *S, int L, int table_cap, uint32_t *counts, long long counts_cap, double *out2,
                              cudaStream_t s) {
    UnitSet us;
    for (int k = 0; k < GCSL_MAX_LEVELS; ++k) us.S[k] = k < L ? S[k] : 0;
    const size_t smem = (size_t)table_cap * sizeof(uint32_t);
    cudaFuncSetAttribute(disc_table_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    disc_table_kernel<<<1, 256, smem, s>>>(data, ld, n, dims, vi, vj, us, L, table_cap, counts, counts_cap, out2);
    note_launch(1);
    return cudaGetLastError();
}

cudaError_t launch_pchisq(const double *x, const long long *df, long long count, double *out, cudaStream_t s) {
    const int blocks = (int)((count + 255) / 256);
    pchisq_kernel<<<blocks > 0 ? blocks : 1, 256, 0, s>>>(x, df, count, out);
    note_launch(1);
    return cudaGetLastError();
}

}  // namespace host
}  // namespace gcsl
