// The float64 certificate of a check: phi, the feasibility push (upper bound) and the Frank-Wolfe longest
// path (lower bound), for one iterate or for a batch's slots together (grid.y = slot).
//
// Reference behaviour (mingxiz/rum-testing-gpu): push solver/common/transforms.py:94-98,
// solver/common/arcflow_kernels.py:357-434; lower bound solver/common/transforms.py:101-114,
// solver/common/arcflow_kernels.py:388-448.
//
// The push works on q = Mobius(x) and recomputes the clipped weights w = max(q, 0) + eps where they
// are read, instead of storing a w slab. The two layered recursions (the push's masses and the
// longest path) read different arrays and go layer by layer in the same launches. Every sum keeps
// one order whatever the launch shape: members ascending, rows by residue mod 1024, then the
// shuffle tree over the 32 warps of residues.
#pragma once
#include "xform.cuh"

namespace rumb {

// Result slots of one check (device doubles)
enum { R_PHI2 = 0, R_RY = 1, R_UB_NOW = 2, R_UB_BEST = 3, R_LB_NOW = 4, R_LB_SEED = 5, R_BETTER = 6, R_SLOTS = 8 };

constexpr double CERT_EPS = 1e-12;
constexpr int CERT_PART = 64;                 // per slot: 32 warp sums each of two quantities

struct CertArgs {
    int n;
    ll Nloc, mp;
    double *qa, *qb, *outw, *mass, *dp;       // slabs and node arrays, one per slot
    const ll *obs;                            // observed positions
    const double *p;                          // the rows' values
    double *pfit, *best;                      // the pushed point on the rows: current and best (or nullptr)
    double *res, *part;
    unsigned *count;                          // finished CTAs, two words per slot (zero between launches)
    ll pstride;                               // between slots' rows (p, pfit, best)
    const int *active, *lb;                   // slot flags (nullptr: all): solved at all, with the lower bound
};

__device__ __forceinline__ double wclip(double q) { return (q > 0.0 ? q : 0.0) + CERT_EPS; }

// The last CTA of `total` to come here (uniform in the CTA; the others' writes before it are visible).
__device__ __forceinline__ bool cert_last(unsigned *count, unsigned total) {
    __threadfence();
    unsigned c = 0;
    if (threadIdx.x == 0) c = atomicAdd(count, 1u);
    c = __shfl_sync(0xffffffffu, c, 0);                       // CTAs of one warp
    if (c + 1u != total) return false;
    if (threadIdx.x == 0) *count = 0u;                        // ready for the next launch
    __threadfence();
    return true;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// phi^2 = sum (p - y)^2 and sum (p - y) y over the rows, y = x2[obs] or given directly; with the lower bound
// also g[obs] = p - y (into qb). 32 CTAs of one warp, CTA b the rows with residue 32 b .. 32 b + 31 mod
// 1024, eight rows' loads in flight per lane: 39 us as one CTA of 1024 threads at n = 18 (23,650 rows).
constexpr int CERT_U = 8;
template <class T>
__global__ void __launch_bounds__(32) obs_stats_kernel(CertArgs A, const T *x2, ll xstride, const double *yv, int with_lb) {
    const int slot = blockIdx.y, lane = threadIdx.x;
    if (A.active && !A.active[slot]) return;
    x2 += slot * xstride;
    const double *p = A.p + slot * A.pstride;
    double *g = with_lb && !(A.lb && !A.lb[slot]) ? A.qb + (ll)slot * A.n * A.Nloc : nullptr;
    double f = 0.0, ry = 0.0;
    for (ll j0 = blockIdx.x * 32 + lane; j0 < A.mp; j0 += 1024 * CERT_U) {
        ll o[CERT_U];
        double y[CERT_U], pj[CERT_U];
#pragma unroll
        for (int u = 0; u < CERT_U; ++u) {
            const ll j = j0 + 1024 * u;
            o[u] = j < A.mp ? A.obs[j] : 0;
            pj[u] = j < A.mp ? p[j] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < CERT_U; ++u) {
            const ll j = j0 + 1024 * u;
            y[u] = j < A.mp ? (yv ? yv[j] : (double)x2[o[u]]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < CERT_U; ++u) {
            if (j0 + 1024 * u >= A.mp) break;
            const double r = pj[u] - y[u];
            f += r * r;
            ry += r * y[u];
            if (g) g[o[u]] = r;
        }
    }
    f = warp_sum(f);
    ry = warp_sum(ry);
    double *part = A.part + slot * CERT_PART;
    if (lane == 0) {
        part[blockIdx.x] = f;
        part[32 + blockIdx.x] = ry;
    }
    if (!cert_last(A.count + 2 * slot, gridDim.x)) return;
    f = warp_sum(__ldcg(part + lane));
    ry = warp_sum(__ldcg(part + 32 + lane));
    if (lane == 0) {
        A.res[slot * R_SLOTS + R_PHI2] = f;
        A.res[slot * R_SLOTS + R_RY] = ry;
    }
}

// The pushed point on the rows and its distance; the last CTA keeps the running minimum.
__global__ void __launch_bounds__(32) ub_eval_kernel(CertArgs A) {
    const int slot = blockIdx.y, lane = threadIdx.x;
    if (A.active && !A.active[slot]) return;
    const double *x = A.qa + (ll)slot * A.n * A.Nloc, *p = A.p + slot * A.pstride;
    double *pfit = A.pfit + slot * A.pstride;
    double f = 0.0;
    for (ll j0 = blockIdx.x * 32 + lane; j0 < A.mp; j0 += 1024 * CERT_U) {
        ll o[CERT_U];
        double v[CERT_U], pj[CERT_U];
#pragma unroll
        for (int u = 0; u < CERT_U; ++u) {
            const ll j = j0 + 1024 * u;
            o[u] = j < A.mp ? A.obs[j] : 0;
            pj[u] = j < A.mp ? p[j] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < CERT_U; ++u) v[u] = x[o[u]];
#pragma unroll
        for (int u = 0; u < CERT_U; ++u) {
            const ll j = j0 + 1024 * u;
            if (j >= A.mp) break;
            pfit[j] = v[u];
            const double d = v[u] - pj[u];
            f += d * d;
        }
    }
    f = warp_sum(f);
    double *part = A.part + slot * CERT_PART, *res = A.res + slot * R_SLOTS;
    if (lane == 0) part[blockIdx.x] = f;
    if (!cert_last(A.count + 2 * slot + 1, gridDim.x)) return;
    f = warp_sum(__ldcg(part + lane));
    if (lane == 0) {
        const double ub = sqrt(f);
        const bool better = ub < res[R_UB_BEST];
        res[R_UB_NOW] = ub;
        res[R_BETTER] = better ? 1.0 : 0.0;
        if (better) res[R_UB_BEST] = ub;
    }
}

__global__ void ub_commit_kernel(CertArgs A) {
    const int slot = blockIdx.y;
    if (A.active && !A.active[slot]) return;
    const ll j = blockIdx.x * (ll)blockDim.x + threadIdx.x;
    if (j < A.mp && A.res[slot * R_SLOTS + R_BETTER] != 0.0) A.best[slot * A.pstride + j] = A.pfit[slot * A.pstride + j];
}

// outw[D] = sum of w(x, D) over the x not in D; also the masses' start, 1 at the empty set.
__global__ void __launch_bounds__(256) outw_kernel(CertArgs A) {
    const int slot = blockIdx.y, n = A.n;
    if (A.active && !A.active[slot]) return;
    const ll D = blockIdx.x * (ll)blockDim.x + threadIdx.x, N = 1LL << n;
    if (D >= N) return;
    const double *q = A.qa + (ll)slot * n * A.Nloc;
    double s = 0.0;
    constexpr int U = 8;
    unsigned out = ~(unsigned)D & (unsigned)(N - 1);
    while (out) {
        double w[U];
        int k = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            w[u] = 0.0;
            if (out) {
                const int x = __ffs((int)out) - 1;
                out &= out - 1u;
                w[u] = q[(ll)x * A.Nloc + (ll)compress_bit((ull)D, x)];
                k = u + 1;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < k) s += wclip(w[u]);
    }
    A.outw[slot * N + D] = s;
    if (D == 0) A.mass[slot * N] = 1.0;
}

// Node C of a layer: the mass pushed into it, mass[C] = sum over x in C of mass[P] w(x, P) / outw[P], P = C \ x.
// Six members' loads are in flight together (one at a time the loads' latency was the layer's time:
// 20 us a layer at n = 18, 8.8 us at n = 8, now 5 and 3).
constexpr int CERT_E = 6;
__device__ __forceinline__ double mass_node(const CertArgs &A, const double *q, const double *outw, const double *mass,
                                            unsigned C) {
    double s = 0.0;
    for (unsigned rem = C; rem;) {
        double ow[CERT_E], m[CERT_E], w[CERT_E];
        int k = 0;
#pragma unroll
        for (int u = 0; u < CERT_E; ++u) {
            if (rem) {
                const int x = __ffs((int)rem) - 1;
                rem &= rem - 1u;
                const unsigned P = C ^ (1u << x);
                ow[u] = outw[P];
                m[u] = mass[P];
                w[u] = q[(ll)x * A.Nloc + (ll)compress_bit((ull)P, x)];
                k = u + 1;
            }
        }
#pragma unroll
        for (int u = 0; u < CERT_E; ++u)
            if (u < k && ow[u] > 0.0) s += m[u] * wclip(w[u]) / ow[u];
    }
    return s;
}
// The longest path into C: dp[C] = max over x in C of dp[P] + R(x, P).
__device__ __forceinline__ double path_node(const CertArgs &A, const double *R, const double *dp, unsigned C) {
    double best = -1e300;
    for (unsigned rem = C; rem;) {
        double d[CERT_E], r[CERT_E];
        int k = 0;
#pragma unroll
        for (int u = 0; u < CERT_E; ++u) {
            if (rem) {
                const int x = __ffs((int)rem) - 1;
                rem &= rem - 1u;
                const unsigned P = C ^ (1u << x);
                d[u] = dp[P];
                r[u] = R[(ll)x * A.Nloc + (ll)compress_bit((ull)P, x)];
                k = u + 1;
            }
        }
#pragma unroll
        for (int u = 0; u < CERT_E; ++u)
            if (u < k) {
                const double v = d[u] + r[u];
                if (v > best) best = v;
            }
    }
    return best;
}
__device__ __forceinline__ void lb_final(double *res, double top) {
    const double rc = top - res[R_RY];
    const double v = res[R_PHI2] - 2.0 * rc;
    res[R_LB_NOW] = sqrt(v > 0.0 ? v : 0.0);
}

// One popcount layer: the first `mb` CTAs of a slot its masses, the others its longest paths. The full set
// ends the lower bound.
__global__ void __launch_bounds__(128) cert_layer_kernel(CertArgs A, const int *nodes, int ns, unsigned mb) {
    const int slot = blockIdx.y, n = A.n;
    if (A.active && !A.active[slot]) return;
    const ll N = 1LL << n, S = (ll)n * A.Nloc;
    if (blockIdx.x < mb) {
        const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
        if (i >= ns) return;
        const unsigned C = (unsigned)nodes[i];
        double *mass = A.mass + slot * N;
        mass[C] = mass_node(A, A.qa + slot * S, A.outw + slot * N, mass, C);
    } else {
        if (A.lb && !A.lb[slot]) return;
        const int i = (int)((blockIdx.x - mb) * blockDim.x + threadIdx.x);
        if (i >= ns) return;
        const unsigned C = (unsigned)nodes[i];
        double *dp = A.dp + slot * N;
        // layer 1 starts from the empty set's 0
        const double v = (C & (C - 1u)) == 0u ? 0.0 + A.qb[slot * S + (ll)(__ffs((int)C) - 1) * A.Nloc]
                                             : path_node(A, A.qb + slot * S, dp, C);
        dp[C] = v;
        if ((ll)C == N - 1) lb_final(A.res + slot * R_SLOTS, v);
    }
}

// All layers of a small lattice in one CTA per slot and recursion (blockIdx.x 0: masses, 1: longest paths),
// the nodes' values in shared memory: at most CERT_SMALL_N alternatives (a launch per layer costs more than
// the layer there).
constexpr int CERT_SMALL_N = 12;
__global__ void __launch_bounds__(1024) cert_small_kernel(CertArgs A, const int *nodes, int push, int with_lb) {
    __shared__ double val[1 << CERT_SMALL_N];
    const int slot = blockIdx.y, n = A.n;
    if (A.active && !A.active[slot]) return;
    const int N = 1 << n;
    const ll S = (ll)n * A.Nloc;
    const bool mass = blockIdx.x == 0;
    if (mass ? !push : (!with_lb || (A.lb && !A.lb[slot]))) return;
    const double *q = (mass ? A.qa : A.qb) + slot * S, *outw = A.outw + (ll)slot * N;
    double *out = (mass ? A.mass : A.dp) + (ll)slot * N;
    if (threadIdx.x == 0) val[0] = mass ? 1.0 : 0.0;
    __syncthreads();
    int lo = 1, cnt = n;                                      // layer c: nodes[lo .. lo + C(n, c))
    for (int c = 1; c <= n; ++c) {
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
            const unsigned C = (unsigned)nodes[lo + i];
            const double v = mass ? mass_node(A, q, outw, val, C) : path_node(A, q, val, C);
            val[C] = v;
            out[C] = v;
        }
        __syncthreads();
        lo += cnt;
        cnt = cnt * (n - c) / (c + 1);
    }
    if (!mass && threadIdx.x == 0) lb_final(A.res + slot * R_SLOTS, val[N - 1]);
}

// rf(x, T) = mass[T] w(x, T) / outw[T] on the slab (into qb)
__global__ void __launch_bounds__(256) extract_kernel(CertArgs A) {
    const int slot = blockIdx.y, n = A.n;
    if (A.active && !A.active[slot]) return;
    const ll a = blockIdx.x * (ll)blockDim.x + threadIdx.x, S = (ll)n * A.Nloc, N = 1LL << n;
    if (a >= S) return;
    const int x = (int)(a >> (n - 1));
    const ll T = (ll)expand_bit((ull)(a & (A.Nloc - 1)), x);
    const double ow = A.outw[slot * N + T];
    A.qb[slot * S + a] = (ow > 0.0) ? A.mass[slot * N + T] * wclip(A.qa[slot * S + a]) / ow : 0.0;
}

}  // namespace rumb
