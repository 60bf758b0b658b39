// The float64 BM-ADMM iteration as two kernels (csrc/dr.cu).
//
// With one penalty b for both blocks the reference's one_iter (solver/bm_admm/solver.py:240-254,
// fuse_xk, prox_all, fuse_z, fuse_sy: :37-51,66-139) carries four slabs x2, s, y, z that hold two
// slabs' worth of information. Put
//     v = xo - z / b (the point the prox reads), u = prox(v):   x2' = u,          z' = b (u - v)
//     t = y / b - a  (the point the clamp reads):               s' = max(t, 0),   y' = b min(t, 0)
// Then with c = (1 - alpha) x2 - z / b and d = (1 - alpha) s + y / b, one iteration is
//     rhs = (x2 + z / b) + A' (s - y / b)  =  (2 u - v) + A' |t|
//     q   = D Q^T rhs                         (D the eigen-space diagonal, in the rest index)
//     v'  = c + alpha Q q,   u' = prox(v'),   c' = v' - alpha u'
//     t'  = d + alpha A Q q,                  d' = min(t', 0) + (1 - alpha) max(t', 0)
// and every transform factors over the rest bits, so with a low window L and a high window H
//     kernel low    a = Q_H q, e = (A Q)_H q in;   v' = c + alpha Q_L a,  t' = d + alpha (A Q)_L e;
//                   a = Q^T_L (2 u' - v'),  e = (Q^T A')_L |t'| out
//     kernel high   a, e in;  q = D Q^T_H (a + A'_H e);  a = Q_H q, e = (A Q)_H q out
// Each reads and writes two slabs per stream: 12 n 2^(n-1) values an iteration, against 20 for the
// three transform passes and the prox over the four state slabs. The prox couples all alternatives
// of a menu, so a low CTA owns 2^M consecutive menus, whose entries are one contiguous run per
// alternative (2^(M-1) values for i < M, 2^M for i >= M and in the base mask); those runs are
// exactly the low window's transforms, M - 1 bits for i < M and M bits for the others, and the high
// window is the rest. Lattices beyond the two windows run middle passes on both streams.
// Measured on one B200, an iteration in a replayed graph: 10.3 / 14.6 / 44.0 / 249 / 1,319 us at n = 13 / 16 /
// 18 / 20 / 22, where the transform passes with the prox took 17.9 / 30.1 / 92 / 444 / 2,190 us with their
// share of the checks. What bounds it: latency of the two kernels to n = 16, the low kernel's dependent prox
// steps at n = 18 (its slabs stay in L2), the high kernel's exchanges through shared memory at n = 20, and
// memory from n = 21.
#pragma once
#include "xform.cuh"

namespace rumb {

struct DrArgs {
    int n;
    ll Nloc;
    double *c, *d;              // the state between iterations
    double *a, *e;              // the two streams
    double *tau;                // per menu: the last threshold (a starting point for the next)
    const double *xhat;
    const uint32_t *menu_obs;   // per menu: its observed members
    double *u_out, *t_out;      // the u and t slabs, written by the last iteration of a sequence
    const double *diag;         // eigen-space diagonal by popcount, with the unit forms' scales
    Co<double> kQ, kAQ, kA, kAp;   // Q (unit form), A Q / q00, A, A'
    double alpha, b, inv_c1;    // b and 1 / (b + 2)
    ll bstride, tstride;        // batched draws: elements between draws' slabs and thresholds (grid.y)
    const int *active;
};

// Smaller lattices are left to the one-pass transform and the lanes prox. Both sides with dependent launches
// and their share of the checks: n = 12 12.0 us an iteration against 13.9 here, n = 13 17.9 against 14.5; since
// then plain launches took the former to 9.6 and the latter to 11.9.
constexpr int DR_MIN_N = 13;

// One iteration's launches (n >= DR_MIN_N); last: also write u_out and t_out.
void dr_iteration(const DrArgs &P, int slots, bool last, cudaStream_t st);
// From the slabs x2, s, y, z (any state) to c, d, a, e and unset thresholds; slots as given.
void dr_begin(const DrArgs &P, int slots, const double *x2, const double *s, const double *y, const double *z,
              cudaStream_t st);
// From u (in x2), t (in s) and c back to x2, s, y, z.
void dr_end(const DrArgs &P, double *x2, double *s, double *y, double *z, cudaStream_t st);

}  // namespace rumb
