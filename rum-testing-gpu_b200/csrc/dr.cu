// The float64 iteration's kernels (formulas and windows in dr.cuh).
#include "dr.cuh"

namespace rumb {

// ---------------------------------------------------------------- runs of 2^B values in a warp
// A run is held by G = 2^(B - 4) lanes, 16 values each. Top layout: register j of lane g is value
// g | j << (B - 4) (lanes on consecutive values: every global access is contiguous); low layout:
// value 16 g + j. The stages of bits 0..3 run in the low layout, those of bits max(4, B - 4)..B - 1
// in the top layout, and with B = 9 bit 4 is a lane bit of the top layout (one shuffle stage). The
// layouts are exchanged through shared memory padded by one value in 16, which keeps both sides of
// the exchange free of bank conflicts.
constexpr int DR_R = 16;
__device__ __forceinline__ int dr_pad(int i) { return i + (i >> 4); }

template <int B>
__device__ __forceinline__ void run_to_low(double (&v)[DR_R], double *w, int g) {
#pragma unroll
    for (int j = 0; j < DR_R; ++j) w[dr_pad(g | (j << (B - 4)))] = v[j];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < DR_R; ++j) v[j] = w[17 * g + j];
    __syncwarp();
}
template <int B>
__device__ __forceinline__ void run_to_top(double (&v)[DR_R], double *w, int g) {
#pragma unroll
    for (int j = 0; j < DR_R; ++j) w[17 * g + j] = v[j];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < DR_R; ++j) v[j] = w[dr_pad(g | (j << (B - 4)))];
    __syncwarp();
}

// the top layout's register stages (and bit 4's lane stage when B = 9)
template <int B, int MODE>
__device__ __forceinline__ void run_top_stages(double (&v)[DR_R], int lane, const Co<double> &k) {
    constexpr int NB = B - 4 < 4 ? B - 4 : 4;               // the highest NB bits
    xf_regs<double, DR_R, 4 - NB, NB, MODE>(v, k);
    if constexpr (B == 9) {
        const bool hi = (lane >> 4) & 1;
        const double c0 = hi ? k.d : k.a, c1 = hi ? k.c : k.b;
#pragma unroll
        for (int i = 0; i < DR_R; ++i) {
            const double o = __shfl_xor_sync(0xffffffffu, v[i], 16);
            if (MODE == XF_APRIME) {
                if (hi) v[i] = k.d * v[i] - o;
            } else if (MODE == XF_UNIT) {
                v[i] = c1 * o + (hi ? -v[i] : v[i]);
            } else {
                v[i] = c0 * v[i] + c1 * o;
            }
        }
    }
}
template <int MODE>
__device__ __forceinline__ void run_low_stages(double (&v)[DR_R], const Co<double> &k) {
    xf_regs<double, DR_R, 0, 4, MODE>(v, k);
}

// Asks L2 for memory that is read later (no registers held meanwhile): `bytes` from p, both multiples of
// 16, or the line at p.
__device__ __forceinline__ void prefetch_run(const double *p, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_line(const double *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ unsigned dr_cb(unsigned m, int x) { return (m & ((1u << x) - 1u)) | ((m >> (x + 1)) << x); }

// ---------------------------------------------------------------- the t stream's low window
// One warp on 512 consecutive values of alternative x's block (2^(9 - B) runs): t' = d + alpha (A Q)_L e,
// d' = min(t', 0) + (1 - alpha) max(t', 0), e' = (Q^T A')_L |t'|. w: the warp's 544 values of shared memory.
template <int B, bool OUT>
__device__ __forceinline__ void dr_low_t(const DrArgs &P, ll at, double *w, int lane) {
    constexpr int G = 1 << (B - 4);
    const int g = lane & (G - 1), run = lane / G;
    w += run * (17 << (B - 4));
    const ll p0 = at + ((ll)run << B) + g;
    double v[DR_R], dd[DR_R];
#pragma unroll
    for (int j = 0; j < DR_R; ++j) v[j] = P.e[p0 + (j << (B - 4))];
    run_top_stages<B, XF_GEN>(v, lane, P.kAQ);
    run_to_low<B>(v, w, g);
    run_low_stages<XF_GEN>(v, P.kAQ);
    run_to_top<B>(v, w, g);
#pragma unroll
    for (int j = 0; j < DR_R; ++j) dd[j] = P.d[p0 + (j << (B - 4))];
#pragma unroll
    for (int j = 0; j < DR_R; ++j) {
        const double t = dd[j] + P.alpha * v[j];
        const double neg = t < 0.0 ? t : 0.0, pos = t > 0.0 ? t : 0.0;
        P.d[p0 + (j << (B - 4))] = neg + (1.0 - P.alpha) * pos;
        if (OUT) P.t_out[p0 + (j << (B - 4))] = t;
        v[j] = pos - neg;
    }
    run_top_stages<B, XF_APRIME>(v, lane, P.kAp);
    run_top_stages<B, XF_UNIT>(v, lane, P.kQ);
    run_to_low<B>(v, w, g);
    run_low_stages<XF_APRIME>(v, P.kAp);
    run_low_stages<XF_UNIT>(v, P.kQ);
    run_to_top<B>(v, w, g);
#pragma unroll
    for (int j = 0; j < DR_R; ++j) P.e[p0 + (j << (B - 4))] = v[j];
}

// ---------------------------------------------------------------- the v stream's low window and the prox
// The exchanges of a v run: a lane group without a run (act false) computes on another run's values and
// stores nothing.
template <int B>
__device__ __forceinline__ void vrun_to_low(double (&v)[DR_R], double *w, int g, bool act) {
#pragma unroll
    for (int j = 0; j < DR_R; ++j)
        if (act) w[dr_pad(g | (j << (B - 4)))] = v[j];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < DR_R; ++j) v[j] = w[17 * g + j];
    __syncwarp();
}
template <int B>
__device__ __forceinline__ void vrun_to_top(double (&v)[DR_R], double *w, int g, bool act) {
#pragma unroll
    for (int j = 0; j < DR_R; ++j)
        if (act) w[17 * g + j] = v[j];
    __syncwarp();
}

// Phase 1 on one run: v' = c + alpha Q_L a, left in the tile.
template <int B>
__device__ __forceinline__ void dr_low_v1(const DrArgs &P, ll p0, double *w, int g, int lane, bool act) {
    double v[DR_R], cc[DR_R];
#pragma unroll
    for (int j = 0; j < DR_R; ++j) v[j] = P.a[p0 + (j << (B - 4))];
    run_top_stages<B, XF_UNIT>(v, lane, P.kQ);
    vrun_to_low<B>(v, w, g, act);
    run_low_stages<XF_UNIT>(v, P.kQ);
    vrun_to_top<B>(v, w, g, act);
#pragma unroll
    for (int j = 0; j < DR_R; ++j) cc[j] = P.c[p0 + (j << (B - 4))];
#pragma unroll
    for (int j = 0; j < DR_R; ++j) {
        const int i = dr_pad(g | (j << (B - 4)));
        cc[j] += P.alpha * w[i];
        if (act) w[i] = cc[j];                               // slot i is this lane's from here on
    }
}

// Phase 3 on one run: u = max(v - tau, 0), c' = v - alpha u, a' = Q^T_L (2 u - v). A threshold of
// NaN marks a menu finished in phase 2 (the tile then holds 2 u - v).
template <int B, bool HALF, bool OUT>
__device__ __forceinline__ void dr_low_v3(const DrArgs &P, ll p0, double *w, const double *stau, int alt, int g, int lane,
                                          bool act) {
    double v[DR_R];
#pragma unroll
    for (int j = 0; j < DR_R; ++j) {
        const int i = g | (j << (B - 4));
        const int m = HALF ? (((i >> alt) << (alt + 1)) | (1 << alt) | (i & ((1 << alt) - 1))) : i;
        const double tau = stau[m];
        double x = w[dr_pad(i)];
        if (tau == tau) {
            double u = x - tau;
            u = u > 0.0 ? u : 0.0;
            if (act) {
                P.c[p0 + (j << (B - 4))] = x - P.alpha * u;
                if (OUT) P.u_out[p0 + (j << (B - 4))] = u;
            }
            x = 2.0 * u - x;
        }
        v[j] = x;
    }
    run_top_stages<B, XF_UNIT>(v, lane, P.kQ);
    __syncwarp();
    vrun_to_low<B>(v, w, g, act);
    run_low_stages<XF_UNIT>(v, P.kQ);
    vrun_to_top<B>(v, w, g, act);
#pragma unroll
    for (int j = 0; j < DR_R; ++j)
        if (act) P.a[p0 + (j << (B - 4))] = w[dr_pad(g | (j << (B - 4)))];
}

// Shared memory of a v tile: the runs (padded) and one threshold per menu.
__host__ __device__ constexpr int dr_low_elems(int M, int n) {
    return (M * (1 << (M - 1)) + (n - M) * (1 << M)) / 16 * 17 + (1 << M);
}

// One low CTA: the first 2^(n - M) of a slot are the v tiles (largest base mask first: the longest
// tiles start first), the others the t stream's chunks of 512 values, one per warp.
template <int M, int NT, int GL, bool OUT>
__global__ void __launch_bounds__(NT, 768 / NT) dr_low_kernel(DrArgs P) {
    extern __shared__ __align__(16) double dr_sm[];
    if (P.active && !P.active[blockIdx.y]) return;
    const int tid = threadIdx.x, lane = tid & 31, wi = tid >> 5;
    constexpr int NW = NT / 32;
    const int n = P.n;
    const ll Nloc = P.Nloc;
    const unsigned tiles = 1u << (n - M);
    const ll slot = (ll)blockIdx.y * P.bstride;
    if (blockIdx.x >= tiles) {
        const ll at = ((ll)(blockIdx.x - tiles) * NW + wi) << 9;
        const int x = (int)(at / Nloc);
        if (x >= n) return;
        double *w = dr_sm + wi * 544;
        if (lane == 0) prefetch_run(P.d + slot + at, 4096);
        if (x < M) dr_low_t<M - 1, OUT>(P, slot + at, w, lane);
        else dr_low_t<M, OUT>(P, slot + at, w, lane);
        return;
    }
    P.a += slot; P.c += slot; P.xhat += slot;
    P.tau += (ll)blockIdx.y * P.tstride;
    if (OUT) P.u_out += slot;
    const unsigned base = (tiles - 1u - blockIdx.x) << M;
    const unsigned hi = base >> M;
    const int pc = __popc(hi);
    constexpr int HS = 17 << (M - 5), FS = 17 << (M - 4);        // padded runs
    double *sv = dr_sm, *stau = dr_sm + (M * HS + (n - M) * FS);
    __shared__ int halt[32], nspec;
    __shared__ __align__(16) uint32_t sobs[1 << M];          // per menu: its observed members
    __shared__ uint16_t spec[1 << M];                        // the menus that have some
    if (tid == 0) nspec = 0;
    // the tile's last thresholds and observed members, copied while phase 1 runs
    for (int i = tid; i < (1 << M) / 2; i += NT)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(stau + 2 * i)),
                     "l"(P.tau + base + 2 * i) : "memory");
    for (int i = tid; i < (1 << M) / 4; i += NT)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(sobs + 4 * i)),
                     "l"(P.menu_obs + base + 4 * i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid < n - M && ((hi >> tid) & 1u)) halt[__popc(hi & ((1u << tid) - 1u))] = M + tid;
    __syncthreads();
    for (int q = tid; q < M + pc; q += NT) {
        const int x = q < M ? q : halt[q - M];
        const ll p = (ll)x * Nloc + (q < M ? base >> 1 : dr_cb(base, x));
        const unsigned bytes = 8u << (q < M ? M - 1 : M);
        prefetch_run(P.c + p, bytes);
        if (q >= NW) prefetch_run(P.a + p, bytes);
    }
    // phase 1: the halves (alternatives below M), then the full runs
    constexpr int GH = 1 << (M - 5), GF = 1 << (M - 4);
    constexpr int nh = (M * GH + 31) / 32;
    const int nf = (pc * GF + 31) / 32;
#pragma unroll 1
    for (int it = wi; it < nh + nf; it += NW) {
        if (it < nh) {
            int q = it * (32 / GH) + lane / GH;
            const int g = lane & (GH - 1);
            const bool act = q < M;
            if (!act) q = 0;
            dr_low_v1<M - 1>(P, (ll)q * Nloc + (base >> 1) + g, sv + q * HS, g, lane, act);
        } else {
            int q = (it - nh) * (32 / GF) + lane / GF;
            const int g = lane & (GF - 1);
            const bool act = q < pc;
            if (!act) q = 0;
            const int x = halt[q];
            dr_low_v1<M>(P, (ll)x * Nloc + dr_cb(base, x) + g, sv + M * HS + q * FS, g, lane, act);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int m = tid; m < (1 << M); m += NT)
        if (sobs[m] != 0 && __popc(base | (unsigned)m) > 1) spec[atomicAdd(&nspec, 1)] = (uint16_t)m;
    __syncthreads();
    // phase 2: one thread per menu without observed members. The threshold is the root of
    // sum max(v - tau, 0) = 1; Newton's step on the active set {v > tau} (the mean excess) is the root once
    // the step leaves the set as it was, which the set's smallest value and the others' largest decide
    // in the same walk. From the last iteration's threshold that is one walk for almost every menu;
    // from any start the active set only shrinks after the first step.
    const int total = nspec, gl = lane & (GL - 1);
    const unsigned gm = GL == 32 ? 0xffffffffu : 0xffffu << (lane & 16);
    // this lane's p_hat in the q-th menu with observed members (read ahead of its use)
    auto xhat_of = [&](int q) -> double {
        if (q >= total || gl >= n) return 0.0;
        const int m = spec[q];
        return (sobs[m] >> gl) & 1u ? __ldg(P.xhat + (ll)gl * Nloc + dr_cb(base | (unsigned)m, gl)) : 0.0;
    };
    double xh_next = xhat_of(tid / GL);
#pragma unroll 1
    for (int m = tid; m < (1 << M); m += NT) {
        const unsigned S = base | (unsigned)m;
        const int k = __popc(S);
        if (sobs[m] != 0 && k > 1) continue;
        const double *ph = sv + M * HS + dr_pad(m);
        if (k > 1) {
            double vl[M];
#pragma unroll
            for (int i = 0; i < M; ++i)
                vl[i] = (m >> i) & 1 ? sv[i * HS + dr_pad((int)dr_cb((unsigned)m, i))] : -INFINITY;
            double tau = stau[m];
            for (int round = 0; round < 64; ++round) {
                double s = 0.0, on_min = INFINITY, off_max = -INFINITY;
                int cnt = 0;
                auto take = [&](double x) {
                    const bool on = x > tau;
                    if (on) { s += x; ++cnt; }
                    on_min = on && x < on_min ? x : on_min;
                    off_max = !on && x > off_max ? x : off_max;
                };
#pragma unroll
                for (int i = 0; i < M; ++i) take(vl[i]);
#pragma unroll 4
                for (int h = 0; h < pc; ++h) take(ph[h * FS]);
                if (cnt == 0) {                              // a start above every value, or none yet
                    if (tau == -INFINITY) break;
                    tau = -INFINITY;
                    continue;
                }
                tau = (s - 1.0) / (double)cnt;
                if (on_min > tau && !(off_max > tau)) break;   // the same active set: the root
            }
            stau[m] = tau;
            P.tau[S] = tau;
        } else if (k == 1) {
            // a singleton: u = 1
            const int i = __ffs((int)S) - 1;
            double *p = i < M ? sv + i * HS + dr_pad((int)dr_cb((unsigned)m, i)) : sv + M * HS + dr_pad(m);
            const ll gp = (ll)i * Nloc + dr_cb(S, i);
            const double x = *p;
            P.c[gp] = x - P.alpha;
            if (OUT) P.u_out[gp] = 1.0;
            *p = 2.0 - x;
            stau[m] = __longlong_as_double(0x7ff8000000000000LL);
        }
    }
    // menus with observed members: a group of GL lanes per menu, lane i its member i. They have curvature
    // b + 2 and are pulled to p_hat. Mixed menus (some members unobserved) keep t = b v + 2 xhat and a
    // threshold in t's scale, fully observed ones the equal-curvature value t / (b + 2).
#pragma unroll 1
    for (int q = tid / GL; q < total; q += NT / GL) {
        const int m = spec[q];
        const unsigned S = base | (unsigned)m;
        const uint32_t wb = sobs[m];
        double tau = stau[m];
        const double xh = xh_next;
        xh_next = xhat_of(q + NT / GL);
        const bool in = gl < 31 && ((S >> gl) & 1u), w = (wb >> gl) & 1u;
        const bool mixed = wb != S;
        double *p = gl < M ? sv + gl * HS + dr_pad((int)dr_cb((unsigned)m, gl))
                           : sv + M * HS + dr_pad(m) + __popc(hi & ((1u << (gl - M)) - 1u)) * FS;
        const double x = in ? *p : 0.0;
        const double cw = P.b + 2.0, cu = P.b, icw = mixed ? 1.0 / cw : 1.0, icu = mixed ? 1.0 / cu : 1.0;
        const double t = in ? (P.b * x + 2.0 * xh) * (mixed ? 1.0 : P.inv_c1) : -INFINITY;
        const double tc = in ? t * (w ? icw : icu) : 0.0;
        unsigned A = __ballot_sync(gm, t > tau) & gm;
        for (int round = 0; round < 64; ++round) {
            if (A == 0) {                                    // a start above every value, or none yet
                A = __ballot_sync(gm, in) & gm;
                if (tau == -INFINITY) break;
                tau = -INFINITY;
            }
            double sum = t > tau ? tc : 0.0;
#pragma unroll
            for (int o = 1; o < GL; o <<= 1) sum += __shfl_xor_sync(gm, sum, o);
            const unsigned O = __ballot_sync(gm, t > tau && w) & gm;
            tau = (sum - 1.0) / ((double)__popc(O) * icw + (double)__popc(A ^ O) * icu);
            const unsigned A2 = __ballot_sync(gm, t > tau) & gm;
            if (A2 == A) break;
            A = A2;
        }
        if (in) {
            double u = t - tau;
            if (mixed) u /= w ? cw : cu;
            u = u > 0.0 ? u : 0.0;
            const ll gp = (ll)gl * Nloc + dr_cb(S, gl);
            P.c[gp] = x - P.alpha * u;
            if (OUT) P.u_out[gp] = u;
            *p = 2.0 * u - x;
        }
        if (gl == 0) {
            P.tau[S] = tau;
            stau[m] = __longlong_as_double(0x7ff8000000000000LL);
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int it = wi; it < nh + nf; it += NW) {
        if (it < nh) {
            int q = it * (32 / GH) + lane / GH;
            const int g = lane & (GH - 1);
            const bool act = q < M;
            if (!act) q = 0;
            dr_low_v3<M - 1, true, OUT>(P, (ll)q * Nloc + (base >> 1) + g, sv + q * HS, stau, q, g, lane, act);
        } else {
            int q = (it - nh) * (32 / GF) + lane / GF;
            const int g = lane & (GF - 1);
            const bool act = q < pc;
            if (!act) q = 0;
            const int x = halt[q];
            dr_low_v3<M, false, OUT>(P, (ll)x * Nloc + dr_cb(base, x) + g, sv + M * HS + q * FS, stau, x, g, lane, act);
        }
    }
}

// ---------------------------------------------------------------- the high window
// A tile is 2^B rows of C = 2^CB consecutive values, rows 2^S0 apart (the window reaches the top bit),
// 2^RB values of one column per thread. Layout O: register j holds row bits O..O+RB-1 and the thread's
// index vt the others. Every position is a base of (vt, column) plus a constant of j, in global memory
// (S0 is a template argument: the offsets are immediates) and in shared memory, where 2^RB rows are
// padded by one row so that the lanes of a half-warp in layout 0 (rows 2^RB apart when C < 16) fall on
// different banks.
template <int RB, int O>
__device__ __forceinline__ int high_vrow(int vt) { return (vt & ((1 << O) - 1)) | ((vt >> O) << (O + RB)); }
template <int B, int CB, int RB, int O>
__device__ __forceinline__ int high_base(int vt, int col) {
    const int r = high_vrow<RB, O>(vt);                     // r >> RB and the j part never carry into each other
    return ((r + (r >> RB)) << CB) + col;
}
template <int CB, int RB, int O>
__host__ __device__ constexpr int high_off(int j) { return ((j << O) + ((j << O) >> RB)) << CB; }

template <int B, int CB, int RB, int FROM, int TO>
__device__ __forceinline__ void high_move(double (&v)[1 << RB], double *sm, int vt, int col) {
    double *p = sm + high_base<B, CB, RB, FROM>(vt, col);
#pragma unroll
    for (int j = 0; j < (1 << RB); ++j) p[high_off<CB, RB, FROM>(j)] = v[j];
    __syncthreads();
    p = sm + high_base<B, CB, RB, TO>(vt, col);
#pragma unroll
    for (int j = 0; j < (1 << RB); ++j) v[j] = p[high_off<CB, RB, TO>(j)];
    __syncthreads();
}

// layout 0 -> the last layout (up) or back (down), every row bit's stage once
template <int B, int CB, int RB, int MODE>
__device__ __forceinline__ void high_up(double (&v)[1 << RB], double *sm, int vt, int col, const Co<double> &k) {
    xf_regs<double, 1 << RB, 0, RB, MODE>(v, k);
    if constexpr (B > 2 * RB) {
        high_move<B, CB, RB, 0, RB>(v, sm, vt, col);
        xf_regs<double, 1 << RB, 0, RB, MODE>(v, k);
        high_move<B, CB, RB, RB, B - RB>(v, sm, vt, col);
        xf_regs<double, 1 << RB, 3 * RB - B, B - 2 * RB, MODE>(v, k);
    } else if constexpr (B > RB) {
        high_move<B, CB, RB, 0, B - RB>(v, sm, vt, col);
        xf_regs<double, 1 << RB, 2 * RB - B, B - RB, MODE>(v, k);
    }
}
template <int B, int CB, int RB, int MODE>
__device__ __forceinline__ void high_down(double (&v)[1 << RB], double *sm, int vt, int col, const Co<double> &k) {
    if constexpr (B > 2 * RB) {
        xf_regs<double, 1 << RB, 3 * RB - B, B - 2 * RB, MODE>(v, k);
        high_move<B, CB, RB, B - RB, RB>(v, sm, vt, col);
        xf_regs<double, 1 << RB, 0, RB, MODE>(v, k);
        high_move<B, CB, RB, RB, 0>(v, sm, vt, col);
    } else if constexpr (B > RB) {
        xf_regs<double, 1 << RB, 2 * RB - B, B - RB, MODE>(v, k);
        high_move<B, CB, RB, B - RB, 0>(v, sm, vt, col);
    }
    xf_regs<double, 1 << RB, 0, RB, MODE>(v, k);
}

__host__ __device__ constexpr int high_rb(int B) { return B <= 4 ? B : (B <= 8 ? 4 : 5); }
__host__ __device__ constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v / 2); }
__host__ __device__ constexpr int high_cb(int B, int NT) { return ilog2(NT) - (B - high_rb(B)); }
__host__ __device__ constexpr int high_elems(int B, int NT) {
    return ((1 << B) + (1 << (B - high_rb(B)))) << high_cb(B, NT);
}

template <int B, int S0, int NT>
__device__ __forceinline__ void high_tile(const DrArgs &P, ll x, unsigned blk, double *sm, const double *diag) {
    constexpr int RB = high_rb(B), CB = high_cb(B, NT), R = 1 << RB, TOP = B - RB;
    const int col = threadIdx.x & ((1 << CB) - 1), vt = threadIdx.x >> CB;
    const unsigned low = (blk << CB) + (unsigned)col;
    const ll p0 = x * P.Nloc + low;
    const ll lo = p0 + ((ll)high_vrow<RB, 0>(vt) << S0), up = p0 + ((ll)high_vrow<RB, TOP>(vt) << S0);
    double v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = P.e[lo + ((ll)j << S0)];
    if ((col & 15) == 0) {
#pragma unroll
        for (int j = 0; j < R; ++j) prefetch_line(P.a + lo + ((ll)j << S0));
    }
    high_up<B, CB, RB, XF_APRIME>(v, sm, vt, col, P.kAp);
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] += P.a[up + ((ll)j << (S0 + TOP))];
    high_down<B, CB, RB, XF_UNIT>(v, sm, vt, col, P.kQ);
    const double *dg = diag + __popc(low) + __popc((unsigned)vt);
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] *= dg[__popc((unsigned)j)];
    high_up<B, CB, RB, XF_UNIT>(v, sm, vt, col, P.kQ);
#pragma unroll
    for (int j = 0; j < R; ++j) P.a[up + ((ll)j << (S0 + TOP))] = v[j];
    high_down<B, CB, RB, XF_A>(v, sm, vt, col, P.kA);
#pragma unroll
    for (int j = 0; j < R; ++j) P.e[lo + ((ll)j << S0)] = v[j];
}

// Alternatives below M have BH + 1 window bits from S0 - 1, the others BH from S0 (= n - 1 - BH); the larger
// tiles come first.
template <int BH, int S0, int NT>
__global__ void __launch_bounds__(NT, 512 / NT) dr_high_kernel(DrArgs P, int M) {
    extern __shared__ __align__(16) double dr_sm[];
    __shared__ double sdiag[32];
    if (P.active && !P.active[blockIdx.y]) return;
    {
        const ll o = (ll)blockIdx.y * P.bstride;
        P.a += o; P.e += o;
    }
    if (threadIdx.x < 32) sdiag[threadIdx.x] = P.diag[threadIdx.x];
    __syncthreads();
    constexpr unsigned big = 1u << (S0 - 1 - high_cb(BH + 1, NT)), small = 1u << (S0 - high_cb(BH, NT));
    if (blockIdx.x < (unsigned)M * big) {
        const unsigned x = blockIdx.x / big;
        high_tile<BH + 1, S0 - 1, NT>(P, x, blockIdx.x - x * big, dr_sm, sdiag);
    } else {
        const unsigned r = blockIdx.x - (unsigned)M * big, x = r / small;
        high_tile<BH, S0, NT>(P, M + x, r - x * small, dr_sm, sdiag);
    }
}

// ---------------------------------------------------------------- middle passes
// Window [s0, s0 + B) of both streams in place, one column of one stream (blockIdx.z: a, e) per thread; s0 =
// s_mid - 1 for the alternatives below M. BEFORE the high window: Q^T on a and Q^T A' on e; after it: Q on a,
// A Q on e. Bound by HBM: 6.1-6.4 TB/s.
template <int B, bool BEFORE>
__global__ void __launch_bounds__(256) dr_mid_kernel(DrArgs P, int M, int s_mid) {
    if (P.active && !P.active[blockIdx.y]) return;
    constexpr int R = 1 << B;
    const ll per = P.Nloc >> B;                              // columns of one alternative
    const ll i = blockIdx.x * (ll)blockDim.x + threadIdx.x;
    const ll x = i / per;
    if (x >= P.n) return;
    const int s0 = x < M ? s_mid - 1 : s_mid;
    const ll r = i - x * per, low = r & ((1LL << s0) - 1);
    double *p = (blockIdx.z ? P.e : P.a) + (ll)blockIdx.y * P.bstride + x * P.Nloc + ((r >> s0) << (s0 + B)) + low;
    double v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = p[(ll)j << s0];
    if (blockIdx.z == 0) {
        xf_regs<double, R, 0, B, XF_UNIT>(v, P.kQ);
    } else if (BEFORE) {
        xf_regs<double, R, 0, B, XF_APRIME>(v, P.kAp);
        xf_regs<double, R, 0, B, XF_UNIT>(v, P.kQ);
    } else {
        xf_regs<double, R, 0, B, XF_GEN>(v, P.kAQ);
    }
#pragma unroll
    for (int j = 0; j < R; ++j) p[(ll)j << s0] = v[j];
}

// ---------------------------------------------------------------- into and out of the iteration
// One warp per 512 values: c, d, a = Q^T_L (x2 + z / b), e = (Q^T A')_L (s - y / b).
template <int B>
__device__ __forceinline__ void dr_begin_chunk(const DrArgs &P, ll at, double *w, int lane, const double *x2,
                                               const double *s, const double *y, const double *z) {
    constexpr int G = 1 << (B - 4);
    const int g = lane & (G - 1), run = lane / G;
    w += run * (17 << (B - 4));
    const ll p0 = at + ((ll)run << B) + g;
    const double ib = 1.0 / P.b, ra = 1.0 - P.alpha;
    double v[DR_R];
#pragma unroll
    for (int j = 0; j < DR_R; ++j) {
        const ll p = p0 + (j << (B - 4));
        const double xv = x2[p], zv = ib * z[p];
        P.c[p] = ra * xv - zv;
        v[j] = xv + zv;
    }
    run_top_stages<B, XF_UNIT>(v, lane, P.kQ);
    run_to_low<B>(v, w, g);
    run_low_stages<XF_UNIT>(v, P.kQ);
    run_to_top<B>(v, w, g);
#pragma unroll
    for (int j = 0; j < DR_R; ++j) {
        const ll p = p0 + (j << (B - 4));
        P.a[p] = v[j];
        const double sv = s[p], yv = ib * y[p];
        P.d[p] = ra * sv + yv;
        v[j] = sv - yv;
    }
    run_top_stages<B, XF_APRIME>(v, lane, P.kAp);
    run_top_stages<B, XF_UNIT>(v, lane, P.kQ);
    run_to_low<B>(v, w, g);
    run_low_stages<XF_APRIME>(v, P.kAp);
    run_low_stages<XF_UNIT>(v, P.kQ);
    run_to_top<B>(v, w, g);
#pragma unroll
    for (int j = 0; j < DR_R; ++j) P.e[p0 + (j << (B - 4))] = v[j];
}

template <int M>
__global__ void __launch_bounds__(128) dr_begin_kernel(DrArgs P, const double *x2, const double *s, const double *y,
                                                       const double *z) {
    __shared__ double sm[4 * 544];
    const ll o = (ll)blockIdx.y * P.bstride;
    P.a += o; P.e += o; P.c += o; P.d += o;
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const ll at = ((ll)blockIdx.x * 4 + wi) << 9;
    const int x = (int)(at / P.Nloc);
    if (x >= P.n) return;
    double *w = sm + wi * 544;
    if (x < M) dr_begin_chunk<M - 1>(P, at, w, lane, x2 + o, s + o, y + o, z + o);
    else dr_begin_chunk<M>(P, at, w, lane, x2 + o, s + o, y + o, z + o);
}

// The thresholds start unset (NaN: no value is above it, so the first step takes every member).
__global__ void dr_unset_kernel(double *tau, ll count, ll tstride) {
    const ll i = blockIdx.x * (ll)blockDim.x + threadIdx.x;
    if (i < count) tau[blockIdx.y * tstride + i] = __longlong_as_double(0x7ff8000000000000LL);
}

__global__ void dr_end_kernel(const double *c, double *x2, double *s, double *y, double *z, ll m, double alpha, double b) {
    const ll i = blockIdx.x * (ll)blockDim.x + threadIdx.x;
    if (i >= m) return;
    const double u = x2[i], t = s[i];
    z[i] = b * ((1.0 - alpha) * u - c[i]);
    s[i] = t > 0.0 ? t : 0.0;
    y[i] = t < 0.0 ? b * t : 0.0;
}

// ---------------------------------------------------------------- launchers
// The windows of n alternatives: tiles of 2^M menus, a high window of BH bits (BH + 1 for the
// alternatives below M) and `mid` bits left to middle passes of up to 5 bits. A low tile holds its n runs of v
// in shared memory and three CTAs share an SM, a high tile holds 2^(BH + 1) rows of at least four values: without
// middle passes up to 10 high bits, with them eight (12 high bits leave one CTA per SM). M = 8 has the faster low
// kernel (n = 18 34.5 us against 39.6 with M = 9, n = 21 274 / 328, n = 22 576 / 667), M = 7 below n = 15 (an
// iteration at n = 14 15.2 us against 16.6, at n = 16 23.5 against 20.8 with M = 8); M = 9 is taken where it
// saves a middle pass (n = 20: 249 us an iteration against 320, n = 23, 28), and at n = 19, where M = 8's high
// tiles would have 32-byte rows (116 us against 118).
struct DrShape {
    int M, BH, mid;
};
static int dr_mid_bits(int n, int M) { return n - 1 - M <= 10 ? 0 : n - 1 - M - 8; }
static DrShape dr_shape(int n) {
    auto passes = [&](int M) { return (dr_mid_bits(n, M) + 4) / 5; };
    DrShape S{};
    S.M = n < 15 ? 7 : n == 19 || passes(9) < passes(8) ? 9 : 8;
    S.mid = dr_mid_bits(n, S.M);
    S.BH = n - 1 - S.M - S.mid;
    return S;
}

// The kernels go out in plain stream order: launched ahead with programmatic dependent launch, their CTAs
// wait on the SMs beside the kernel before, and a replayed iteration takes longer (n = 15: 20.2 against
// 18.2 us, n = 16: 29.8 / 22.2, n = 20: 291 / 267).
template <class... KArgs, class... Args>
static void dr_launch(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    kern<<<grid, block, smem, st>>>(args...);
}

static void dr_prof(const char *what, const DrArgs &P, int slots, double slabs, cudaStream_t st) {
    if (!g_prof) return;
    const double S = (double)P.Nloc * P.n * slots;
    prof_begin(what, slabs * S * 8.0, st);
}

template <int M, int NT, int GL, bool OUT>
static void dr_low_go(const DrArgs &P, int slots, cudaStream_t st) {
    static std::atomic<unsigned long long> optin{0};
    const size_t smem = 8 * (size_t)std::max(dr_low_elems(M, P.n), NT / 32 * 544);
    smem_optin(dr_low_kernel<M, NT, GL, OUT>, 160 * 1024, optin);
    const ll chunks = ((ll)P.n * P.Nloc) >> 9;
    const unsigned grid = (1u << (P.n - M)) + (unsigned)((chunks + NT / 32 - 1) / (NT / 32));
    dr_prof(OUT ? "dr_low_out<f64>" : "dr_low<f64>", P, slots, OUT ? 10.0 : 8.0, st);
    dr_launch(dr_low_kernel<M, NT, GL, OUT>, dim3(grid, (unsigned)slots), dim3(NT), smem, st, P);
    RUMB_LAUNCH("dr_low_kernel");
    prof_end(st);
}
// 16 lanes per observed menu hold up to 16 alternatives, a warp more
template <bool OUT>
static void dr_low(const DrArgs &P, int M, int slots, cudaStream_t st) {
    if (M == 7) dr_low_go<7, 256, 16, OUT>(P, slots, st);
    else if (M == 8 && P.n <= 16) dr_low_go<8, 256, 16, OUT>(P, slots, st);
    else if (M == 8 && P.n <= 18) dr_low_go<8, 128, 32, OUT>(P, slots, st);   // n = 18: 34.5 us against 36
    else if (M == 8) dr_low_go<8, 256, 32, OUT>(P, slots, st);                // n = 22: 576 us against 612
    else dr_low_go<9, 256, 32, OUT>(P, slots, st);
}

template <int BH, int S0, int NT>
static void dr_high_go(const DrArgs &P, int M, int slots, cudaStream_t st) {
    static std::atomic<unsigned long long> optin{0};
    const size_t smem = 8 * (size_t)std::max(high_elems(BH, NT), high_elems(BH + 1, NT));
    smem_optin(dr_high_kernel<BH, S0, NT>, 160 * 1024, optin);
    constexpr unsigned big = 1u << (S0 - 1 - high_cb(BH + 1, NT)), small = 1u << (S0 - high_cb(BH, NT));
    dr_prof("dr_high<f64>", P, slots, 4.0, st);
    dr_launch(dr_high_kernel<BH, S0, NT>, dim3((unsigned)M * big + (unsigned)(P.n - M) * small, (unsigned)slots), dim3(NT),
               smem, st, P, M);
    RUMB_LAUNCH("dr_high_kernel");
    prof_end(st);
}
template <bool BEFORE>
static void dr_mid(const DrArgs &P, const DrShape &S, int slots, cudaStream_t st) {
    for (int s = S.M, left = S.mid; left > 0;) {
        const int passes = (left + 4) / 5, B = (left + passes - 1) / passes;
        const ll cols = ((ll)P.n * P.Nloc) >> B;
        const dim3 grid(grid_for(cols, 256), (unsigned)slots, 2);
        dr_prof(BEFORE ? "dr_mid_before<f64>" : "dr_mid_after<f64>", P, slots, 4.0, st);
        switch (B) {
            case 1: dr_launch(dr_mid_kernel<1, BEFORE>, grid, dim3(256), 0, st, P, S.M, s); break;
            case 2: dr_launch(dr_mid_kernel<2, BEFORE>, grid, dim3(256), 0, st, P, S.M, s); break;
            case 3: dr_launch(dr_mid_kernel<3, BEFORE>, grid, dim3(256), 0, st, P, S.M, s); break;
            case 4: dr_launch(dr_mid_kernel<4, BEFORE>, grid, dim3(256), 0, st, P, S.M, s); break;
            default: dr_launch(dr_mid_kernel<5, BEFORE>, grid, dim3(256), 0, st, P, S.M, s); break;
        }
        RUMB_LAUNCH("dr_mid_kernel");
        prof_end(st);
        s += B;
        left -= B;
    }
}

void dr_iteration(const DrArgs &P0, int slots, bool last, cudaStream_t st) {
    const DrShape S = dr_shape(P0.n);
    DrArgs P = P0;
    dr_mid<true>(P, S, slots, st);
    // threads per CTA: small lattices have few tiles, and more of them with fewer threads
    switch (P.n) {
        case 13: dr_high_go<5, 7, 64>(P, S.M, slots, st); break;
        case 14: dr_high_go<6, 7, 64>(P, S.M, slots, st); break;
        case 15: dr_high_go<6, 8, 128>(P, S.M, slots, st); break;
        case 16: dr_high_go<7, 8, 128>(P, S.M, slots, st); break;
        case 17: dr_high_go<8, 8, 128>(P, S.M, slots, st); break;
        case 18: dr_high_go<9, 8, 256>(P, S.M, slots, st); break;
        case 19: dr_high_go<9, 9, 256>(P, S.M, slots, st); break;
        case 20: dr_high_go<10, 9, 256>(P, S.M, slots, st); break;
#define DR_CASE(n) case n: dr_high_go<8, n - 9, 256>(P, S.M, slots, st); break;
        DR_CASE(21) DR_CASE(22) DR_CASE(23) DR_CASE(24) DR_CASE(25) DR_CASE(26) DR_CASE(27) DR_CASE(28) DR_CASE(29)
        DR_CASE(30)
#undef DR_CASE
        default: fail(RUMB_E_INTERNAL, "dr_high: no kernel for this n");
    }
    dr_mid<false>(P, S, slots, st);
    if (last) dr_low<true>(P, S.M, slots, st);
    else dr_low<false>(P, S.M, slots, st);
}

void dr_begin(const DrArgs &P, int slots, const double *x2, const double *s, const double *y, const double *z,
              cudaStream_t st) {
    const DrShape S = dr_shape(P.n);
    const ll chunks = ((ll)P.n * P.Nloc) >> 9;
    const dim3 grid((unsigned)((chunks + 3) / 4), (unsigned)slots);
    switch (S.M) {
        case 7: dr_begin_kernel<7><<<grid, 128, 0, st>>>(P, x2, s, y, z); break;
        case 8: dr_begin_kernel<8><<<grid, 128, 0, st>>>(P, x2, s, y, z); break;
        default: dr_begin_kernel<9><<<grid, 128, 0, st>>>(P, x2, s, y, z); break;
    }
    RUMB_LAUNCH("dr_begin_kernel");
    // the thresholds share a slab of the state (see the caller): set after the state has been read
    dr_unset_kernel<<<dim3(grid_for(1LL << P.n, 256), (unsigned)slots), 256, 0, st>>>(P.tau, 1LL << P.n, P.tstride);
    RUMB_LAUNCH("dr_unset_kernel");
}

void dr_end(const DrArgs &P, double *x2, double *s, double *y, double *z, cudaStream_t st) {
    const ll m = (ll)P.n * P.Nloc;
    dr_end_kernel<<<grid_for(m, 256), 256, 0, st>>>(P.c, x2, s, y, z, m, P.alpha, P.b);
    RUMB_LAUNCH("dr_end_kernel");
}

}  // namespace rumb
