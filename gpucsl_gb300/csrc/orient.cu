// Edge orientation of the skeleton on the GPU: v-structures, then Meek's rules R1-R3 to
// a fixed point, with the result of the reference's sequential CPU code
// (gpucsl/pc/edge_orientation/v_structures.py:8-35, orientation_rules.py:7-89).
//
// The reference visits ordered edges (v1, v2) in column-major order (key v2 * p + v1)
// and inner vertices ascending, writing a live graph.  Its outcome is reproduced in
// parallel from the structure of those writes:
//
// * v-structures read only the skeleton and the sepsets, so every unshielded triple's
//   decision is fixed; a triple with middle b orienting a -> b writes "a -> b present,
//   b -> a absent".  The last writer of a directed pair wins, and the visiting order is
//   by the middle vertex first, so with P[a][b] = "some triple orients a -> b":
//   a -> b is absent at the end iff P[b][a] and (not P[a][b] or a > b).
// * R1 checks the live graph before writing: on each edge the earliest firing (smallest
//   visiting key (v2 p + v1) p + v3) decides the direction (atomicMin per edge).
// * R2 and R3 write without a live check: on each edge the latest firing (largest key
//   v2 p + v1, the smallest complement) decides the direction (atomicMin per edge).
// Each rule reads a snapshot (the graph after the previous rule's firings are applied).
//
// D[a * p + b] = 1 means the directed graph has a -> b; an undirected edge has both.
//
// A step is a few dependent loads on a few thousand edges, so what bounds the whole is the
// number of steps times the cost of separating them.  orient_kernel runs them all in one
// cooperative launch with barriers between (about 1 us), skips the applications of rules
// that fired nowhere and counts the passes itself: on a skeleton of 1000 vertices with the
// sets of its solve 116 us a call, where sweeps over p^2 entries, six launches and a host read
// a pass took 296 us.
// The barriers' waits have a time limit, so a step has to be short against it: where the sum of
// cubed degrees (a bound on a step's work) is above OR_MAX_WORK, the same steps run as separate
// kernels.  Close to the line the two cost about the same (1000 vertices of degree 39: 169 us
// in one kernel; of degree 60, in separate ones: 152).
#include "common.cuh"
#include "gauss_dev.cuh"

namespace gcsl {

constexpr unsigned long long OR_NONE = 0xffffffffffffffffull;
constexpr unsigned long long OR_MAX_WORK = 1ull << 26;
constexpr long long OR_WAIT_NS = 4000000000ll;  // a barrier's limit
constexpr int OR_MAX_PASSES = 1 << 20;          // of one cooperative launch
// Warps per row of a dense graph's neighbours (for_edges), as far as the SMs hold them: with one,
// 300 vertices of degree 150 kept 38 blocks busy.  One kernel (at most a block an SM) against
// one warp a row: 100 vertices of degree 40: 178 -> 85 us, of degree 5: 66 -> 67; separate kernels:
// 300 of degree 150: 1061 -> 197 us, 1000 of degree 200: 1565 -> 374.
constexpr int OR_SHARE = 4, OR_SHARE_STEPS = 16;

enum OrStatus { OR_UNFINISHED = 0, OR_DONE = 1 };

// Control words of the cooperative kernel, zero at its start.
struct OrCtl {
    unsigned arrived;    // blocks that reached a barrier, over all barriers
    unsigned fired[2];   // last odd / even phase in which a rule fired
    int status, passes;  // read by the host
    int changed;         // separate kernels: a rule of the pass fired
    unsigned long long work;  // sum of degree^3
};

__device__ __forceinline__ bool in_sepset(const int *__restrict__ sep, int L, int p, int a, int c, int v) {
    const int *s1 = sep + ((size_t)a * p + c) * L, *s2 = sep + ((size_t)c * p + a) * L;
    bool in = false;
#pragma unroll 4
    for (int k = 0; k < L; ++k) in |= s1[k] == v || s2[k] == v;
    return in;
}

// A directed edge's presence and the lists change between the steps of one kernel: read
// from L2.
__device__ __forceinline__ bool arc(const uint8_t *D, int p, int a, int b) {
    return __ldcg(D + (size_t)a * p + b) != 0;
}

// A warp's rows first, first + step, ..; with more warps than rows several share one and take
// turns in its neighbours.
struct RowShare {
    int first, step, part, share;
    __device__ __forceinline__ RowShare(int p, int warp, int warps) {
        share = warps > p ? warps / p : 1;
        step = warps / share;
        part = warp / step;
        first = part < share ? warp - part * step : p;  // the last few warps: no rows
    }
};

// f(a, b, list of a, degree of a, lane of the group, group mask) for every directed pair
// (a, b) of adjacent vertices: eight lanes per neighbour b.
template <typename F>
__device__ __forceinline__ void for_edges(const int *adj, int p, const RowShare &rs, F f) {
    const int lane = threadIdx.x & 31, sub = lane & 7;
    const unsigned group = 0xffu << (lane & 24);
    for (int a = rs.first; a < p; a += rs.step) {
        const int *ra = adj + (size_t)a * p;
        const int da = __ldcg(ra);
        for (int t = 4 * rs.part + (lane >> 3); t < da; t += 4 * rs.share) f(a, __ldcg(ra + 1 + t), ra, da, sub, group);
    }
}

// P[a][b] for every skeleton edge: some neighbour v != a of b, non-adjacent to a, with b
// in neither sepset(a, v) nor sepset(v, a).
__device__ __forceinline__ void vstruct_flags(const uint16_t *__restrict__ S, const int *adj, int p,
                                              const int *__restrict__ sep, int L, uint8_t *P, const RowShare &rs) {
    for_edges(adj, p, rs, [&](int a, int b, const int *, int, int sub, unsigned group) {
        const int *rb = adj + (size_t)b * p;
        const int db = __ldcg(rb);
        bool hit = false;
        for (int k = sub; k < db && !hit; k += 8) {
            const int v = __ldcg(rb + 1 + k);
            hit = v != a && S[(size_t)a * p + v] == 0 && !in_sepset(sep, L, p, a, v, b);
        }
        const bool any = __any_sync(group, hit);
        if (sub == 0) P[(size_t)a * p + b] = any ? 1 : 0;
    });
}

// Directions of the v-structures; D is zero elsewhere.  The keys of the edges start empty
// (those of a < b are used).
__device__ __forceinline__ void vstruct_apply(const int *adj, int p, const uint8_t *P, uint8_t *D,
                                              unsigned long long *key, int warp, int warps) {
    const int lane = threadIdx.x & 31;
    for (int a = warp; a < p; a += warps) {
        const int *ra = adj + (size_t)a * p;
        const int da = __ldcg(ra);
        for (int t = lane; t < da; t += 32) {
            const int b = __ldcg(ra + 1 + t);
            const bool pab = arc(P, p, a, b), pba = arc(P, p, b, a);
            D[(size_t)a * p + b] = pba && (!pab || a > b) ? 0 : 1;
            if (a < b) key[(size_t)a * p + b] = OR_NONE;
        }
    }
}

__device__ __forceinline__ void fire_edge(unsigned long long *key, int p, int from, int to, unsigned long long seq,
                                          bool latest) {
    const int lo = min(from, to), hi = max(from, to);
    const unsigned long long k = seq * 2 + (from < to ? 0 : 1);
    atomicMin(&key[(size_t)lo * p + hi], latest ? ~k : k);
}

// R1 on snapshot D: v1 -> v2 (directed only), v2 - v3 undirected, v1 and v3
// non-adjacent: orient v2 -> v3.  Earliest key per edge.  True if the thread fired one.
__device__ __forceinline__ bool rule1(const int *adj, int p, const uint8_t *D, unsigned long long *key,
                                      const RowShare &rs) {
    bool fired = false;
    for_edges(adj, p, rs, [&](int v1, int v2, const int *, int, int sub, unsigned) {
        const int *r2 = adj + (size_t)v2 * p;
        const int d2 = __ldcg(r2);
        if (!arc(D, p, v1, v2) || arc(D, p, v2, v1)) return;
        for (int k = sub; k < d2; k += 8) {
            const int v3 = __ldcg(r2 + 1 + k);
            const bool a = arc(D, p, v2, v3), b = arc(D, p, v3, v2), c = arc(D, p, v1, v3), d = arc(D, p, v3, v1);
            if (v3 != v1 && a && b && !c && !d) {
                fire_edge(key, p, v2, v3, ((unsigned long long)v2 * p + v1) * p + v3, false);
                fired = true;
            }
        }
    });
    return fired;
}

// v1 - v2 undirected in D: R2 some v3 with v1 -> v3 -> v2 directed only; R3 two non-adjacent
// v3, v4 with v1 - v3 -> v2, v1 - v4 -> v2.  Orient v1 -> v2, latest key per edge.
template <int RULE>
__device__ __forceinline__ bool rule23(const int *adj, int p, const uint8_t *D, unsigned long long *key,
                                       const RowShare &rs) {
    bool fired = false;
    for_edges(adj, p, rs, [&](int v1, int v2, const int *r1, int d1, int sub, unsigned group) {
        if (!arc(D, p, v1, v2) || !arc(D, p, v2, v1)) return;
        bool fire = false;
        for (int k0 = 0; k0 < d1 && !fire; k0 += 8) {
            const int v3 = k0 + sub < d1 ? __ldcg(r1 + 1 + k0 + sub) : v2;
            const bool out = arc(D, p, v1, v3), in = arc(D, p, v3, v1), on = arc(D, p, v3, v2),
                       off = arc(D, p, v2, v3);
            const bool hit = v3 != v2 && out && in == (RULE == 3) && on && !off;
            unsigned found = __ballot_sync(group, hit) & group;
            if constexpr (RULE == 2) {
                fire = found != 0u;
            } else {
                // each member against the members after it in the list
                for (; found != 0u && !fire; found &= found - 1u) {
                    const int src = __ffs(found) - 1;
                    const int u = __shfl_sync(group, v3, src);
                    bool pair = false;
                    for (int k = k0 + (src & 7) + 1 + sub; k < d1 && !pair; k += 8) {
                        const int v4 = __ldcg(r1 + 1 + k);
                        pair = v4 != v2 && arc(D, p, v1, v4) && arc(D, p, v4, v1) && arc(D, p, v4, v2) &&
                               !arc(D, p, v2, v4) && !arc(D, p, u, v4) && !arc(D, p, v4, u);
                    }
                    fire = __any_sync(group, pair);
                }
            }
        }
        if (fire && sub == 0) {
            fire_edge(key, p, v1, v2, (unsigned long long)v2 * p + v1, true);
            fired = true;
        }
    });
    return fired;
}

// Orient every edge whose key is set and empty the key; `latest`: the keys are complements.
__device__ __forceinline__ void rule_apply(const int *adj, int p, uint8_t *D, unsigned long long *key, bool latest,
                                           int warp, int warps) {
    const int lane = threadIdx.x & 31;
    for (int lo = warp; lo < p; lo += warps) {
        const int *r = adj + (size_t)lo * p;
        const int d = __ldcg(r);
        for (int t = lane; t < d; t += 32) {
            const int hi = __ldcg(r + 1 + t);
            if (hi <= lo) continue;
            const size_t k = (size_t)lo * p + hi;
            const unsigned long long v = __ldcg(key + k);
            if (v == OR_NONE) continue;
            const bool up = ((latest ? ~v : v) & 1ull) == 0;  // lo -> hi
            D[k] = up ? 1 : 0;
            D[(size_t)hi * p + lo] = up ? 0 : 1;
            key[k] = OR_NONE;
        }
    }
}

// Grid barrier of the cooperative kernel: phase = its number from 1.  *fired: whether any
// thread of the grid came with f.  False if the wait passed its limit; every block then
// runs into the same limit at this barrier or the next and returns.
__device__ __forceinline__ bool or_barrier(OrCtl *ctl, unsigned phase, bool f, bool *fired) {
    __shared__ int s_ok, s_fired;
    const int any = __syncthreads_or(f);
    if (threadIdx.x == 0) {
        if (any) atomicMax(&ctl->fired[phase & 1], phase);
        __threadfence();
        atomicAdd(&ctl->arrived, 1u);
        const unsigned target = phase * gridDim.x;
        long long t0 = 0;
        bool ok = true;
        for (unsigned polls = 0;; ++polls) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&ctl->arrived) : "memory");
            if (v >= target) break;
            if ((polls & 255u) == 255u) {
                long long now;
                asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
                if (t0 == 0) t0 = now;
                if (now - t0 > OR_WAIT_NS) {
                    ok = false;
                    break;
                }
            }
        }
        __threadfence();
        s_ok = ok;
        // (a block ahead of this one is in the next phase at most, which has the other word)
        s_fired = __ldcg(&ctl->fired[phase & 1]) == phase;
    }
    __syncthreads();
    const bool ok = s_ok != 0;
    *fired = s_fired != 0;
    __syncthreads();
    return ok;
}

__global__ void __launch_bounds__(256, 1) orient_kernel(const uint16_t *__restrict__ S, int p,
                                                    const int *__restrict__ sep, int L, int *adj, uint8_t *P,
                                                    uint8_t *D, unsigned long long *key, OrCtl *ctl) {
    const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), warps = (int)(gridDim.x * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    const long long pp = (long long)p * p, tid = (long long)blockIdx.x * blockDim.x + threadIdx.x,
                    threads = (long long)gridDim.x * blockDim.x;
    const RowShare rs(p, warp, warps);
    unsigned phase = 0;
    bool fired;
    const long long vec = (reinterpret_cast<uintptr_t>(D) & 15u) == 0 ? pp / 16 : 0;
    for (long long k = tid; k < vec; k += threads) reinterpret_cast<uint4 *>(D)[k] = make_uint4(0u, 0u, 0u, 0u);
    for (long long k = vec * 16 + tid; k < pp; k += threads) D[k] = 0;
    unsigned long long work = 0ull;
    for (int r = warp; r < p; r += warps) {
        const unsigned long long d = (unsigned long long)compact_row(S, p, adj, nullptr, r, lane);
        work += d * d * d;
    }
    if (lane == 0 && work != 0ull) atomicAdd(&ctl->work, work);
    if (!or_barrier(ctl, ++phase, false, &fired)) return;
    if (__ldcg(&ctl->work) > OR_MAX_WORK) return;  // (every block alike)
    vstruct_flags(S, adj, p, sep, L, P, rs);
    if (!or_barrier(ctl, ++phase, false, &fired)) return;
    vstruct_apply(adj, p, P, D, key, warp, warps);
    if (!or_barrier(ctl, ++phase, false, &fired)) return;
    const long long max_passes = pp / 2 + 2;  // every pass orients an edge
    for (int n = 1;; ++n) {
        bool changed = false;
        for (int rule = 1; rule <= 3; ++rule) {
            const bool f = rule == 1   ? rule1(adj, p, D, key, rs)
                           : rule == 2 ? rule23<2>(adj, p, D, key, rs)
                                       : rule23<3>(adj, p, D, key, rs);
            if (!or_barrier(ctl, ++phase, f, &fired)) return;
            if (!fired) continue;
            changed = true;
            rule_apply(adj, p, D, key, rule != 1, warp, warps);
            if (!or_barrier(ctl, ++phase, false, &fired)) return;
        }
        if (!changed || n >= max_passes) {
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                ctl->passes = n;
                ctl->status = OR_DONE;
            }
            return;
        }
        if (n >= OR_MAX_PASSES) return;
    }
}

// The same steps as separate kernels.
__global__ void __launch_bounds__(256) orient_step_kernel(const uint16_t *__restrict__ S, int p,
                                                         const int *__restrict__ sep, int L, const int *adj,
                                                         uint8_t *P, uint8_t *D, unsigned long long *key, OrCtl *ctl,
                                                         int step) {
    const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), warps = (int)(gridDim.x * blockDim.x) >> 5;
    const RowShare rs(p, warp, warps);
    bool fired = false;
    switch (step) {
    case 0: vstruct_flags(S, adj, p, sep, L, P, rs); break;
    case 1: vstruct_apply(adj, p, P, D, key, warp, warps); break;
    case 2: fired = rule1(adj, p, D, key, rs); break;
    case 3: rule_apply(adj, p, D, key, false, warp, warps); break;
    case 4: fired = rule23<2>(adj, p, D, key, rs); break;
    case 6: fired = rule23<3>(adj, p, D, key, rs); break;
    default: rule_apply(adj, p, D, key, true, warp, warps); break;  // 5, 7
    }
    if (fired) ctl->changed = 1;
}

namespace host {

size_t orient_workspace_bytes(int p) {
    const size_t pp = (size_t)p * p;
    auto al = [](size_t x) { return (x + 255) / 256 * 256; };
    return al(pp * sizeof(int)) + al(pp) + al(pp * sizeof(unsigned long long)) + al(sizeof(OrCtl));
}

cudaError_t launch_compact(const uint16_t *G, int p, int *adj, int *up, DevState *st, int level, int2 *elist,
                           cudaStream_t s);

// Returns the number of rule passes in *passes; `host_words` is pinned host memory (2 ints).
cudaError_t orient_edges(const uint16_t *S, int p, const int *sep, int L, uint8_t *D, void *ws, int num_sms,
                         int *host_words, int *passes, cudaStream_t s) {
    const size_t pp = (size_t)p * p;
    auto al = [](size_t x) { return (x + 255) / 256 * 256; };
    char *w = static_cast<char *>(ws);
    int *adj = reinterpret_cast<int *>(w);
    uint8_t *P = reinterpret_cast<uint8_t *>(w + al(pp * sizeof(int)));
    unsigned long long *key = reinterpret_cast<unsigned long long *>(w + al(pp * sizeof(int)) + al(pp));
    OrCtl *ctl = reinterpret_cast<OrCtl *>(w + al(pp * sizeof(int)) + al(pp) + al(pp * 8));
    const int rows_blocks = (p + 7) / 8;
    const int step_blocks = std::max(rows_blocks, std::min(rows_blocks * OR_SHARE_STEPS, num_sms * 8));
    int coop_blocks = std::min(rows_blocks * OR_SHARE, num_sms);
    if (coop_blocks < 2 * rows_blocks) coop_blocks = std::min(rows_blocks, num_sms);  // no two warps for every row
    cudaError_t e = cudaMemsetAsync(ctl, 0, sizeof(OrCtl), s);
    if (e != cudaSuccess) return e;
    void *args[] = {&S, &p, &sep, &L, &adj, &P, &D, &key, &ctl};
    // at most one block an SM: all resident
    e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(orient_kernel),
                                    dim3((unsigned)coop_blocks), dim3(256), args, 0, s);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs than the device's for this context
        cudaGetLastError();
        host_words[0] = OR_UNFINISHED;
    } else {
        note_launch(1);
        if (e != cudaSuccess ||
            (e = cudaMemcpyAsync(host_words, &ctl->status, 2 * sizeof(int), cudaMemcpyDeviceToHost, s)) !=
                cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
            return e;
    }
    if (host_words[0] == OR_DONE) {
        *passes = host_words[1];
        return cudaSuccess;
    }
    if ((e = launch_compact(S, p, adj, nullptr, nullptr, 0, nullptr, s)) != cudaSuccess ||
        (e = cudaMemsetAsync(D, 0, pp, s)) != cudaSuccess)
        return e;
    const long long max_passes = (long long)pp / 2 + 2;  // every pass orients an edge
    for (int n = 0, first = 0;; first = 2) {
        ++n;
        if ((e = cudaMemsetAsync(&ctl->changed, 0, sizeof(int), s)) != cudaSuccess) return e;
        for (int step = first; step < 8; ++step)
            orient_step_kernel<<<step_blocks, 256, 0, s>>>(S, p, sep, L, adj, P, D, key, ctl, step);
        note_launch(8 - first);
        if ((e = cudaMemcpyAsync(host_words, &ctl->changed, sizeof(int), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
            return e;
        if (!host_words[0] || n >= max_passes) {
            *passes = n;
            break;
        }
    }
    return cudaGetLastError();
}

}  // namespace host
}  // namespace gcsl
