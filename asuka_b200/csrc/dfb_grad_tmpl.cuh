// Adjoint-first Rys derivative contraction over shared-exponent auxiliary groups.
//
// The gradient needs sum Gamma . d(ab|f)/dR, never the derivative integrals themselves, and the
// auxiliary shells of one atom and angular momentum usually are contractions of ONE set of
// primitives.  So the adjoint is taken to primitive auxiliary functions first (Gamma_q = sum_s c_sq
// Gamma_s), its bra indices (a, b) are folded onto the functions e on centre A alone (the transposed
// horizontal recurrence, rows D0; rows D1 = dD0/d(AB) carry the part of the B derivative that lowers
// b), and every primitive triplet is then evaluated once per group instead of once per shell, with
// scalars as its only results:
//
//   S0 = sum D0[e,f] X[ex,fx] Y[ey,fy] Z[ez,fz]        (X, Y, Z: 2D recurrence tables of one root)
//   S1 = the same with e raised by one in a direction, S2 with e lowered (times e_d),
//   T  = sum D1[e,f] X Y Z
//   dE/dA = 2a S1 - S2 + T,  dE/dB = 2b (S1 + AB S0) - T,  dE/dC = -(dE/dA + dE/dB).
//
// One lane holds one Rys root of one task (AO pair, primitive range of a group): the roots of a task
// sit in neighbouring lanes (a team), evaluate their own node and weight, and share the task's rows,
// which the warp first forms in shared memory.  Accumulators are scalars.  Per f the z column is
// contracted through its adjoint column zb (zb[ez] += D0 XY), which costs one multiply-add per element
// for all three z results.
//
// Bound by memory latency in the low classes (Rys-table rows, Gamma and pair records; FP64 pipe 10 to 22 %,
// 12 warps per SM at about 165 registers), by few tasks in the high ones.  (H2O)8/ma-TZVP, 416 AO / 1824 aux:
// 3c derivative contraction 15.7 ms with one evaluation per shell, 6.5 ms here (8.5 with the transformed
// adjoint through HBM, 9.3 with rows staged per block instead of per warp); 2c derivatives 1.30 -> 0.32 ms.
#pragma once
#include "dfb_rys_tmpl.cuh"

namespace dfb {

// One auxiliary primitive range of a group: its Gamma rows are row0 .. row0 + nq - 1 (one row = one
// primitive shell), counted from the start of the class's rows; pairs below plo are skipped.
struct GradChunk {
    int group, prim0, nq, row0, plo;
};

// Groups: 6 ints each -- representative shell, first primitive, primitives, shells, first
// coefficient (coef[s * nprim + k]), first entry of the shell list.
struct GradGroups {
    const int* info;
    const double* coef;
    const int* shells;
    const double *pexp, *rexp;  // per distinct primitive: exponent and reciprocal
    const double* cxyz;         // aux shell centres
    const int *aostart, *atom;  // per aux shell
};
constexpr int GG_REP = 0, GG_P0 = 1, GG_NK = 2, GG_NS = 3, GG_COEF = 4, GG_SH = 5, GG_N = 6;

struct GradArgs {
    const int *shA, *shB, *pstart, *npair_prim;         // per pair
    const double* rec;   // per primitive pair: p, 1/p, 2 pi^(5/2) cK / p, P (3), 2a, 2b
    const double* cxyz;
    const int* atom;
    int b_dummy;         // bra = one primitive aux function on centre A (metric): P = A, no B
    const int* pairs;    // pair indices of the class
    int npair, nchunk;   // tasks = npair x nchunk
    long nwarp;          // warps of the launch
    int tiled;           // 1: a warp takes one chunk and a tile of pairs; 0: any 32 / nr consecutive tasks
    GradGroups gg;
    const GradChunk* chunks;
    int nq, qc;          // largest primitive count of a chunk, primitives staged at a time
    int warp_sz;         // doubles of shared memory per warp
    const int* aostart;
    const double* bar;
    long sP, sM, sN;
    int lc, nr;
    double* grad;
    int natm, smem_grad;
    RysTable tab;
};

constexpr int GRAD_THREADS = 128;
constexpr int GRAD_WARPS = GRAD_THREADS / 32;

// Rows per primitive and aux component f: the NE values of D0 and, for each of the NLOW functions e
// below the top shell, the three D1 values.
template <int LA, int LB>
struct GradShape {
    static constexpr int L1 = LA + LB;
    static constexpr int NE = c_ncb(L1 + 1) - c_ncb(LA);
    static constexpr int NLOW = LB > 0 ? c_ncb(L1) - c_ncb(LA) : 0;
    static constexpr int RF = NE + 3 * NLOW;
};

// Node and weight of root u of the nr-point rule.
__device__ __forceinline__ void rys_one(const RysTable& tab, int nr, int u, double T, double& x, double& w) {
    if (T >= tab.tmax) {
        const double* h = tab.herm + tab.hoff[nr];
        const double rs = rsqrt(T);
        x = __ldg(h + u) * (rs * rs);
        w = __ldg(h + nr + u) * rs;
        return;
    }
    const double Th = T * tab.inv_h;
    int k = (int)Th;
    if (k > tab.nint - 1) k = tab.nint - 1;
    const double t = 2.0 * (Th - (double)k) - 1.0;
    const double t2 = t * t, t4 = t2 * t2, t8 = t4 * t4;
    constexpr int S = DFB_RYS_DEG + 1;
    const double2* cx = reinterpret_cast<const double2*>(tab.coef + tab.offs[nr] + ((size_t)k * (2 * nr) + u) * S);
    const double2* cw = cx + nr * (S / 2);
    double a[S], b[S];
#pragma unroll
    for (int d = 0; d < S / 2; ++d) {
        const double2 v = __ldg(cx + d), v2 = __ldg(cw + d);
        a[2 * d] = v.x;
        a[2 * d + 1] = v.y;
        b[2 * d] = v2.x;
        b[2 * d + 1] = v2.y;
    }
    x = poly9(a, t, t2, t4, t8);
    w = poly9(b, t, t2, t4, t8);
}

// First column (b = 0) of a 2D recurrence table.
template <int NM>
__device__ __forceinline__ void rys_col0(double (&c)[NM + 1], double g00, double C, double B1) {
    c[0] = g00;
    if constexpr (NM > 0) c[1] = C * g00;
#pragma unroll
    for (int a = 2; a <= NM; ++a) c[a] = fma(C, c[a - 1], (B1 * (double)(a - 1)) * c[a - 2]);
}

// Next column: c <- column b+1, p <- column b, with fb = b B1'.
template <int NM>
__device__ __forceinline__ void rys_coln(double (&c)[NM + 1], double (&p)[NM + 1], double Cp, double B0, double fb) {
#pragma unroll
    for (int a = NM; a >= 0; --a) {  // descending: c[a - 1] is still column b
        double n = fma(Cp, c[a], fb * p[a]);
        if (a > 0) n = fma((double)a * B0, c[a > 0 ? a - 1 : 0], n);
        p[a] = c[a];
        c[a] = n;
    }
}

// f(0), f(1), ..., f(N - 1) with compile-time arguments: every array index below is a constant.
template <class F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
    static_for_impl(f, std::make_integer_sequence<int, N>{});
}

// The scalars of one primitive triplet and root.
struct GradSums {
    double s0, s1[3], s2[3], t[3];
};

// One aux component f: rows D0 and D1 at w (row stride RS doubles), columns x, y, z of its 2D tables.
template <int LA, int LB, int RS>
__device__ __forceinline__ void grad_component(const double* w, const double (&x)[LA + LB + 2],
                                               const double (&y)[LA + LB + 2], const double (&z)[LA + LB + 2],
                                               double (&s)[LA + LB + 1], double (&sy1)[LA + LB + 1],
                                               double (&sy2)[LA + LB + 1], GradSums& S) {
    using G = GradShape<LA, LB>;
    constexpr int L1 = G::L1;
    double zb[L1 + 1], yw[L1 + 1];
    static_for<L1 + 1>([&](auto ii) {
        constexpr int i = decltype(ii)::value;
        zb[i] = 0.0;
        if constexpr (i > 0) yw[i] = (double)i * y[i - 1];
    });
    static_for<L1 + 1>([&](auto iex) {
        static_for<L1 + 1>([&](auto iey) {
            constexpr int ex = decltype(iex)::value, ey = decltype(iey)::value;
            if constexpr (ex + ey <= L1) {
                const double xy = x[ex] * y[ey];
                double v = 0.0;
                static_for<L1 + 1>([&](auto iez) {
                    constexpr int ez = decltype(iez)::value, l = ex + ey + ez;
                    if constexpr (l >= LA && l <= L1) {
                        constexpr int e = c_eidx(LA, ex, ey, ez);
                        const double d = w[RS * e];
                        v = fma(d, z[ez], v);
                        zb[ez] = fma(d, xy, zb[ez]);
                        if constexpr (LB > 0 && l < L1) {
                            const double q = xy * z[ez];
#pragma unroll
                            for (int k = 0; k < 3; ++k)
                                S.t[k] = fma(w[RS * (G::NE + 3 * e + k)], q, S.t[k]);
                        }
                    }
                });
                s[ex] = fma(y[ey], v, s[ex]);
                sy1[ex] = fma(y[ey + 1], v, sy1[ex]);
                if constexpr (ey > 0) sy2[ex] = fma(yw[ey], v, sy2[ex]);
            }
        });
    });
    static_for<L1 + 1>([&](auto iez) {
        constexpr int ez = decltype(iez)::value;
        S.s1[2] = fma(zb[ez], z[ez + 1], S.s1[2]);
        if constexpr (ez > 0) S.s2[2] = fma(zb[ez], (double)ez * z[ez - 1], S.s2[2]);
    });
}

// Close the x direction: the sums over y and z per ex against column x.
template <int L1>
__device__ __forceinline__ void grad_x_end(const double (&x)[L1 + 2], const double (&sx)[L1 + 1],
                                           const double (&sy1)[L1 + 1], const double (&sy2)[L1 + 1], GradSums& S) {
    static_for<L1 + 1>([&](auto iex) {
        constexpr int ex = decltype(iex)::value;
        S.s0 = fma(x[ex], sx[ex], S.s0);
        S.s1[0] = fma(x[ex + 1], sx[ex], S.s1[0]);
        if constexpr (ex > 0) S.s2[0] = fma((double)ex * x[ex - 1], sx[ex], S.s2[0]);
        S.s1[1] = fma(x[ex], sy1[ex], S.s1[1]);
        S.s2[1] = fma(x[ex], sy2[ex], S.s2[1]);
    });
}

// binomial coefficients for n <= 4 in closed form (folds in unrolled loops)
__device__ __forceinline__ constexpr int c_bin(int n, int k) {
    return k == 0 ? 1 : k == 1 ? n : k == 2 ? n * (n - 1) / 2 : k == 3 ? n * (n - 1) * (n - 2) / 6
                                                                       : n * (n - 1) * (n - 2) * (n - 3) / 24;
}

// Adjoint of one (task, primitive, f) mixed over the group's shells: elements [I0, I0 + N) of the bra
// block (a-major).
template <int LA, int LB, int N>
__device__ __forceinline__ void grad_gamma(const GradArgs& g, const GradChunk& ch, int pair, int prim, int f, int i0,
                                           double (&gam)[N]) {
    constexpr int NB = c_ncart(LB);
    const int* gi = g.gg.info + GG_N * ch.group;
    const int ns = gi[GG_NS], nk = gi[GG_NK];
    const int* sh = g.gg.shells + gi[GG_SH];
    const double* cf = g.gg.coef + gi[GG_COEF] + (prim - gi[GG_P0]);
    const int shA = g.shA[pair], shB = g.shB[pair];
#pragma unroll
    for (int i = 0; i < N; ++i) gam[i] = 0.0;
    if (LB == 0 && g.b_dummy) {
        // metric: the bra is primitive `pair` of group shB; the unordered pair counts twice
        const int* gb = g.gg.info + GG_N * shB;
        const int nst = gb[GG_NS], nkt = gb[GG_NK];
        const double* ct = g.gg.coef + gb[GG_COEF] + (pair - gb[GG_P0]);
        for (int t = 0; t < nst; ++t) {
            const double c2 = 2.0 * ct[t * nkt];
            const double* bt = g.bar + ((long)g.gg.aostart[g.gg.shells[gb[GG_SH] + t]] + i0) * g.sP + (long)f * g.sM;
            for (int s = 0; s < ns; ++s) {
                const double c = c2 * cf[s * nk];
                const double* b = bt + (long)g.gg.aostart[sh[s]] * g.sM;
#pragma unroll
                for (int i = 0; i < N; ++i) gam[i] = fma(c, __ldg(b + i * g.sP), gam[i]);
            }
        }
        return;
    }
    const double fac = shA != shB ? 2.0 : 1.0;  // both orders of an off-diagonal AO pair
    const double* base = g.bar + ((long)g.aostart[shA] + i0 / NB) * g.sM + (long)g.aostart[shB] * g.sN + (long)f * g.sP;
    for (int s = 0; s < ns; ++s) {
        const double c = fac * __ldg(cf + s * nk);
        const double* b = base + (long)g.gg.aostart[sh[s]] * g.sP;
#pragma unroll
        for (int i = 0; i < N; ++i) gam[i] = fma(c, __ldg(b + (i / NB) * g.sM + (i % NB) * g.sN), gam[i]);
    }
}

// The same for QB primitives at once with the group's row offsets and coefficients (off[s],
// cf[s * QB + k]) in shared memory: every Gamma element is read once for all QB.
template <int LA, int LB, int QB, int N>
__device__ __forceinline__ void grad_gamma_q(const double* __restrict__ base, long sM, long sN, const long* off,
                                             const double* cf, int ns, double (&gam)[QB][N]) {
    constexpr int NB = c_ncart(LB);
    constexpr int US = N <= 3 ? 4 : N <= 9 ? 2 : 1;  // shells in flight
#pragma unroll
    for (int k = 0; k < QB; ++k)
#pragma unroll
        for (int i = 0; i < N; ++i) gam[k][i] = 0.0;
#pragma unroll US
    for (int s = 0; s < ns; ++s) {
        const double* b = base + off[s];
        double c[QB];
#pragma unroll
        for (int k = 0; k < QB; ++k) c[k] = cf[s * QB + k];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const double v = __ldg(b + (i / NB) * sM + (i % NB) * sN);
#pragma unroll
            for (int k = 0; k < QB; ++k) gam[k][i] = fma(c[k], v, gam[k][i]);
        }
    }
}

// Transposed horizontal recurrence (a b| = sum_k C(b,k) AB^(b-k) (a+k| of the functions with x power ex:
// gam(i) = element i of the bra block, rows at w (row stride RS).
template <int LA, int LB, int RS, class Gam>
__device__ __forceinline__ void grad_hrr_x(int ex, const double (&ABp)[3][LB + 1], const Gam& gam, double* w) {
    using G = GradShape<LA, LB>;
    constexpr int NB = c_ncart(LB), L1 = G::L1;
#pragma unroll
    for (int ey = 0; ey <= L1; ++ey) {
#pragma unroll
        for (int ez = 0; ez <= L1; ++ez) {
            if (ex + ey + ez < LA || ex + ey + ez > L1) continue;
            const bool low = ex + ey + ez < L1;
            const int e = c_eidx(LA, ex, ey, ez);
            double v = 0.0, t[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int bx = 0; bx <= LB; ++bx) {
#pragma unroll
                for (int by = 0; by <= LB - bx; ++by) {
#pragma unroll
                    for (int kx = 0; kx <= bx; ++kx) {
#pragma unroll
                        for (int ky = 0; ky <= by; ++ky) {
                            const int bz = LB - bx - by, kz = (ex + ey + ez) - LA - kx - ky;
                            if (kz < 0 || kz > bz || kx > ex || ky > ey || kz > ez) continue;
                            const int ax = ex - kx, az = ez - kz;
                            const int ia = ((LA - ax) * (LA - ax + 1)) / 2 + az;
                            const int ib = ((LB - bx) * (LB - bx + 1)) / 2 + bz;
                            const int nx = bx - kx, ny = by - ky, nz = bz - kz;
                            const double gv = (double)(c_bin(bx, kx) * c_bin(by, ky) * c_bin(bz, kz)) * gam(ia * NB + ib);
                            const double px = ABp[0][nx], py = ABp[1][ny], pz = ABp[2][nz];
                            v = fma(gv, px * py * pz, v);
                            if (low) {
                                if (nx > 0) t[0] = fma(gv * nx, ABp[0][nx > 0 ? nx - 1 : 0] * py * pz, t[0]);
                                if (ny > 0) t[1] = fma(gv * ny, px * ABp[1][ny > 0 ? ny - 1 : 0] * pz, t[1]);
                                if (nz > 0) t[2] = fma(gv * nz, px * py * ABp[2][nz > 0 ? nz - 1 : 0], t[2]);
                            }
                        }
                    }
                }
            }
            w[RS * e] = v;
            if (low) {
#pragma unroll
                for (int d = 0; d < 3; ++d) w[RS * (G::NE + 3 * e + d)] = t[d];
            }
        }
    }
}

template <int LB>
__device__ __forceinline__ void grad_ab_powers(const GradArgs& g, int pair, double (&ABp)[3][LB + 1]) {
    const int shA = g.shA[pair], shB = g.shB[pair];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double ab = g.cxyz[3 * shA + d] - g.cxyz[3 * shB + d];
        ABp[d][0] = 1.0;
#pragma unroll
        for (int k = 1; k <= LB; ++k) ABp[d][k] = ABp[d][k - 1] * ab;
    }
}

// The same for one function e with run-time loops: the bra classes whose unrolled recurrence is too long to
// compile (l_B >= 3, which have few tasks).
template <int LA, int LB, int RS, class Gam>
__device__ __noinline__ void grad_hrr_e(int e, const double (&ABp)[3][LB + 1], const Gam& gam, double* w) {
    using G = GradShape<LA, LB>;
    int l = LA, r = e;
    while (r >= (l + 1) * (l + 2) / 2) r -= (l + 1) * (l + 2) / 2, ++l;
    int m = 0;  // m = l - ex
    while (r > m) r -= ++m;
    const int ex = l - m, ey = m - r, ez = r;
    double v = 0.0, t[3] = {0.0, 0.0, 0.0};
    int ib = 0;
    for (int bx = LB; bx >= 0; --bx) {
        for (int by = LB - bx; by >= 0; --by, ++ib) {
            const int bz = LB - bx - by;
            for (int kx = 0; kx <= bx && kx <= ex; ++kx) {
                for (int ky = 0; ky <= by && ky <= ey; ++ky) {
                    const int kz = l - LA - kx - ky;
                    if (kz < 0 || kz > bz || kz > ez) continue;
                    const int ax = ex - kx, az = ez - kz;
                    const double gv = (double)(c_bin(bx, kx) * c_bin(by, ky) * c_bin(bz, kz)) *
                                      gam((((LA - ax) * (LA - ax + 1)) / 2 + az) * c_ncart(LB) + ib);
                    const int nx = bx - kx, ny = by - ky, nz = bz - kz;
                    const double px = ABp[0][nx], py = ABp[1][ny], pz = ABp[2][nz];
                    v = fma(gv, px * py * pz, v);
                    if (nx > 0) t[0] = fma(gv * nx, ABp[0][nx - 1] * py * pz, t[0]);
                    if (ny > 0) t[1] = fma(gv * ny, px * ABp[1][ny - 1] * pz, t[1]);
                    if (nz > 0) t[2] = fma(gv * nz, px * py * ABp[2][nz - 1], t[2]);
                }
            }
        }
    }
    w[RS * e] = v;
    if (l < LA + LB)
        for (int d = 0; d < 3; ++d) w[RS * (G::NE + 3 * e + d)] = t[d];
}

// Rows of one (task, primitive, f) from its mixed adjoint.
template <int LA, int LB, int RS>
__device__ __forceinline__ void grad_rows(const double (&gam)[c_ncart(LA) * c_ncart(LB)], const double (&ABp)[3][LB + 1],
                                          double* w) {
    if constexpr (LB == 0) {
#pragma unroll
        for (int i = 0; i < c_ncart(LA); ++i) w[RS * i] = gam[i];  // e = a
    } else {
#pragma unroll
        for (int ex = 0; ex <= LA + LB; ++ex) grad_hrr_x<LA, LB, RS>(ex, ABp, [&](int i) { return gam[i]; }, w);
    }
}

// One primitive pair, and the root data of one primitive triplet: all the recurrence tables need.
struct GradPair {
    double p, rp, ckr, P[3], PA[3], a2, b2;
};
struct GradRoot {
    double B0, B1, B1p, C[3], Cp[3], w;
};

__device__ __forceinline__ GradPair grad_pair(const double* rec, int b_dummy, int iab, const double (&A)[3]) {
    GradPair r;
    const double2* q = reinterpret_cast<const double2*>(rec) + 4L * iab;
    const double2 v0 = __ldg(q), v1 = __ldg(q + 1), v2 = __ldg(q + 2), v3 = __ldg(q + 3);
    r.p = v0.x;
    r.rp = v0.y;
    r.ckr = v1.x;
    r.P[0] = b_dummy ? A[0] : v1.y;
    r.P[1] = b_dummy ? A[1] : v2.x;
    r.P[2] = b_dummy ? A[2] : v2.y;
    r.a2 = v3.x;
    r.b2 = v3.y;
#pragma unroll
    for (int d = 0; d < 3; ++d) r.PA[d] = r.P[d] - A[d];
    return r;
}

__device__ __forceinline__ GradRoot grad_root(const GradArgs& g, const GradPair& a, int nr, int u, const double (&C)[3],
                                              double q, double rq) {
    GradRoot r;
    const double s = rsqrt(a.p + q);
    const double inv = s * s;
    double cp[3], R2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        cp[d] = C[d] - a.P[d];
        R2 = fma(cp[d], cp[d], R2);
    }
    double x, w;
    rys_one(g.tab, nr, u, a.p * q * inv * R2, x, w);
    r.w = w * a.ckr * rq * s;
    r.B0 = 0.5 * x * inv;
    r.B1 = fma(0.5 * (1.0 - x), a.rp, r.B0);
    r.B1p = fma(0.5 * (1.0 - x), rq, r.B0);
    const double fc = q * inv * x, fp = -a.p * inv * x;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        r.C[d] = fma(fc, cp[d], a.PA[d]);
        r.Cp[d] = fp * cp[d];
    }
    return r;
}

// fx ranges of the component slices: slice i holds fx0(i) <= fx < fx0(i + 1).  The rows of one primitive
// take at most GRAD_ROW_BYTES of shared memory per lane (a single fx may exceed it).
constexpr int GRAD_ROW_BYTES = 640;
template <int LA, int LB, int LC>
struct GradSlices {
    static constexpr int NR = (LA + LB + LC + 1) / 2 + 1;
    __host__ __device__ static constexpr int most() { return GRAD_ROW_BYTES * NR / (8 * GradShape<LA, LB>::RF); }
    __host__ __device__ static constexpr int fx0(int i) {
        int fx = 0;
        for (int k = 0; k < i && fx <= LC; ++k) {
            int n = 0;
            do {
                n += LC - fx + 1;
                ++fx;
            } while (fx <= LC && n + LC - fx + 1 <= most());
        }
        return fx;
    }
    __host__ __device__ static constexpr int count() {
        int n = 0;
        while (fx0(n) <= LC) ++n;
        return n;
    }
    // components in [fxa, fxb)
    __host__ __device__ static constexpr int nf(int fxa, int fxb) {
        int n = 0;
        for (int fx = fxa; fx < fxb; ++fx) n += LC - fx + 1;
        return n;
    }
    __host__ __device__ static constexpr int max_nf() {
        int m = 0;
        for (int i = 0; i < count(); ++i) {
            const int n = nf(fx0(i), fx0(i + 1));
            m = n > m ? n : m;
        }
        return m;
    }
};

// Scalars of all components of a slice for one root; rows of local component lf at w + lf * RF * RS.
template <int LA, int LB, int LC, int FXA, int FXB, int RS>
__device__ __forceinline__ void grad_slice(const GradRoot& r, const double* w, GradSums& S) {
    constexpr int L1 = LA + LB, NM = L1 + 1, RF = GradShape<LA, LB>::RF;
    constexpr int MY = LC - FXA;  // largest fy of the slice
    double Yt[MY + 1][NM + 1];
    {
        double yc[NM + 1], yp[NM + 1];
        rys_col0<NM>(yc, 1.0, r.C[1], r.B1);
#pragma unroll
        for (int a = 0; a <= NM; ++a) yp[a] = 0.0;
#pragma unroll
        for (int b = 0; b <= MY; ++b) {
#pragma unroll
            for (int a = 0; a <= NM; ++a) Yt[b][a] = yc[a];
            if (b < MY) rys_coln<NM>(yc, yp, r.Cp[1], r.B0, (double)b * r.B1p);
        }
    }
    double xc[NM + 1], xp[NM + 1], z0[NM + 1];
    rys_col0<NM>(xc, r.w, r.C[0], r.B1);
    rys_col0<NM>(z0, 1.0, r.C[2], r.B1);
#pragma unroll
    for (int a = 0; a <= NM; ++a) xp[a] = 0.0;
    static_for<FXB>([&](auto ifx) {
        constexpr int fx = decltype(ifx)::value;
        if constexpr (fx >= FXA) {
            double sx[L1 + 1], sy1[L1 + 1], sy2[L1 + 1];
            double zc[NM + 1], zp[NM + 1];
#pragma unroll
            for (int i = 0; i <= L1; ++i) sx[i] = sy1[i] = sy2[i] = 0.0;
#pragma unroll
            for (int a = 0; a <= NM; ++a) {
                zc[a] = z0[a];
                zp[a] = 0.0;
            }
            constexpr int lf0 = GradSlices<LA, LB, LC>::nf(FXA, fx);
            static_for<LC - fx + 1>([&](auto ifz) {
                constexpr int fz = decltype(ifz)::value, fy = LC - fx - fz;
                grad_component<LA, LB, RS>(w + (lf0 + fz) * RF * RS, xc, Yt[fy], zc, sx, sy1, sy2, S);
                if constexpr (fy > 0) rys_coln<NM>(zc, zp, r.Cp[2], r.B0, (double)fz * r.B1p);
            });
            grad_x_end<L1>(xc, sx, sy1, sy2, S);
        }
        if constexpr (fx + 1 < FXB) rys_coln<NM>(xc, xp, r.Cp[0], r.B0, (double)fx * r.B1p);
    });
}

// One component f = (fx, fy, fz) given at run time, its columns built by their recurrences.
template <int LA, int LB, int RS>
__device__ __forceinline__ void grad_single(const GradRoot& r, const int (&fd)[3], const double* w, GradSums& S) {
    constexpr int L1 = LA + LB, NM = L1 + 1;
    double c[3][NM + 1];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double p[NM + 1];
        rys_col0<NM>(c[d], d == 0 ? r.w : 1.0, r.C[d], r.B1);
#pragma unroll
        for (int a = 0; a <= NM; ++a) p[a] = 0.0;
#pragma unroll 1
        for (int b = 0; b < fd[d]; ++b) rys_coln<NM>(c[d], p, r.Cp[d], r.B0, (double)b * r.B1p);
    }
    double sx[L1 + 1], sy1[L1 + 1], sy2[L1 + 1];
#pragma unroll
    for (int i = 0; i <= L1; ++i) sx[i] = sy1[i] = sy2[i] = 0.0;
    grad_component<LA, LB, RS>(w, c[0], c[1], c[2], sx, sy1, sy2, S);
    grad_x_end<L1>(c[0], sx, sy1, sy2, S);
}

// G[3 at + d] += v[d] over the lanes that are on: lanes with one atom are summed first (a warp's pairs share
// few atoms), so an address takes one addition per warp and atom instead of one per lane.
__device__ __forceinline__ void grad_warp_add(double* G, int at, const double (&v)[3], bool on) {
    const int lane = threadIdx.x & 31;
    unsigned left = __ballot_sync(0xffffffffu, on);
    while (left) {
        const int lead = __ffs(left) - 1;
        const int key = __shfl_sync(0xffffffffu, at, lead);
        const bool mine = on && at == key;
        double s[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            s[d] = mine ? v[d] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s[d] += __shfl_xor_sync(0xffffffffu, s[d], o);
        }
        if (lane == lead) {
#pragma unroll
            for (int d = 0; d < 3; ++d) atomicAdd(G + 3 * key + d, s[d]);
        }
        left &= ~__ballot_sync(0xffffffffu, mine);
    }
}

// The work of one warp: its tasks' rows staged for g.qc primitives at a time, then every lane's root of
// every primitive triplet.  `stage(team, pair, chunk, prim, rows)` is called by whole warps;
// `eval(root, rows, S)` adds the scalars of one root.  UNR: triplets whose roots are evaluated together
// (two table gathers in flight where the arithmetic of one triplet does not hide them).
template <int LA, int LB, int NR, int RS, int UNR, class Stage, class Eval>
__device__ __forceinline__ void grad_warp(const GradArgs& g, int prim_sz, int warp_sz, const Stage& stage,
                                          const Eval& eval) {
    extern __shared__ double sm[];
    const int ng = g.smem_grad ? 3 * g.natm : 0;
    const int tid = threadIdx.x, lane = tid & 31;
    double* sgrad = sm;
    double* rows = sm + ng + (tid >> 5) * warp_sz;  // [qc][prim_sz]
    for (int i = tid; i < ng; i += GRAD_THREADS) sgrad[i] = 0.0;
    __syncthreads();
    double* G0 = g.smem_grad ? sgrad : g.grad;
    const int nr = NR > 0 ? NR : g.nr;
    const int tw = 32 / nr;  // tasks per warp
    const int team = lane / nr, u = lane - team * nr;
    const long wid = (long)blockIdx.x * GRAD_WARPS + (tid >> 5);
    if (wid < g.nwarp) {
        // tiled: consecutive warps take the chunks of one tile of pairs (heaviest pairs first), so the
        // long tasks start early and a warp shares centre C
        int ck = 0, pi = -1;
        if (g.tiled) {
            const long tile = wid / g.nchunk;
            ck = (int)(wid - tile * g.nchunk);
            pi = (int)tile * tw + team;
            if (pi >= g.npair) pi = -1;
        } else {
            const long t = wid * tw + team;
            if (t < (long)g.npair * g.nchunk) {
                ck = (int)(t / g.npair);
                pi = (int)(t - (long)ck * g.npair);
            }
        }
        const GradChunk ch = g.chunks[ck];
        int pair = -1, atA = 0, atB = 0, p0 = 0, p1 = 0;
        const int rep = g.gg.info[GG_N * ch.group + GG_REP];
        const int atC = g.gg.atom[rep];
        double A[3] = {0, 0, 0}, AB[3] = {0, 0, 0};
        const double C[3] = {g.gg.cxyz[3 * rep], g.gg.cxyz[3 * rep + 1], g.gg.cxyz[3 * rep + 2]};
        if (team < tw && pi >= ch.plo) {
            pair = g.pairs[pi];
            const int shA = g.shA[pair];
            atA = g.atom[shA];
            atB = g.b_dummy ? atC : g.atom[g.shB[pair]];
            // three centres on one atom: the derivatives cancel on it
            if (atA == atC && atB == atC) pair = -1;
        }
        if (pair >= 0) {
            const int shA = g.shA[pair];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                A[d] = g.cxyz[3 * shA + d];
                if (!g.b_dummy) AB[d] = A[d] - g.cxyz[3 * g.shB[pair] + d];
            }
            p0 = g.pstart[pair];
            p1 = p0 + g.npair_prim[pair];
        }
        double gA[3] = {0, 0, 0}, gB[3] = {0, 0, 0};
        if (__any_sync(0xffffffffu, pair >= 0)) {
            for (int k0 = 0; k0 < g.nq; k0 += g.qc) {
                __syncwarp();  // the previous primitives' rows are consumed
                stage(tw, pair, ck, k0, rows);
                __syncwarp();
                if (pair < 0) continue;
                const int kn = ch.nq - k0 < g.qc ? ch.nq - k0 : g.qc;
                const double* qx = g.gg.pexp + ch.prim0 + k0;
                const double* rqx = g.gg.rexp + ch.prim0 + k0;
                for (int iab = p0; iab < p1; ++iab) {
                    const GradPair pr = grad_pair(g.rec, g.b_dummy, iab, A);
                    GradSums S;
                    S.s0 = 0.0;
#pragma unroll
                    for (int d = 0; d < 3; ++d) S.s1[d] = S.s2[d] = S.t[d] = 0.0;
                    int k = 0;
                    if constexpr (UNR == 2) {
                        for (; k + 1 < kn; k += 2) {
                            const GradRoot r0 = grad_root(g, pr, nr, u, C, __ldg(qx + k), __ldg(rqx + k));
                            const GradRoot r1 = grad_root(g, pr, nr, u, C, __ldg(qx + k + 1), __ldg(rqx + k + 1));
                            eval(r0, rows + k * prim_sz + team, S);
                            eval(r1, rows + (k + 1) * prim_sz + team, S);
                        }
                    }
                    for (; k < kn; ++k)
                        eval(grad_root(g, pr, nr, u, C, __ldg(qx + k), __ldg(rqx + k)), rows + k * prim_sz + team, S);
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        gA[d] += fma(pr.a2, S.s1[d], S.t[d] - S.s2[d]);
                        gB[d] += fma(pr.b2, fma(AB[d], S.s0, S.s1[d]), -S.t[d]);
                    }
                }
            }
            double gC[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) gC[d] = -(gA[d] + gB[d]);
            const bool on = pair >= 0;
            grad_warp_add(G0, atA, gA, on);
            if (!g.b_dummy) grad_warp_add(G0, atB, gB, on);
            grad_warp_add(G0, atC, gC, on);
        }
    }
    if (g.smem_grad) {
        __syncthreads();
        for (int i = tid; i < ng; i += GRAD_THREADS)
            if (sgrad[i] != 0.0) atomicAdd(g.grad + i, sgrad[i]);
    }
}

// Primitives staged at a time: as many as fit GRAD_STAGE_BYTES per warp (what shared memory leaves of L1
// serves the Rys table's gathers) and a lane's registers.
constexpr int GRAD_STAGE_BYTES = 6 * 1024;
constexpr int GRAD_MAXS = 16;  // shells of a group whose offsets and coefficients a warp keeps
template <int LA, int LB, int LC>
__host__ __device__ constexpr int grad_qb() {
    using SL = GradSlices<LA, LB, LC>;
    const int prim = 8 * SL::max_nf() * GradShape<LA, LB>::RF * (32 / SL::NR);
    const int q = GRAD_STAGE_BYTES / prim, r = 40 / (c_ncart(LA) * c_ncart(LB));
    const int m = q < r ? q : r;
    return m >= 4 ? 4 : m >= 2 ? 2 : 1;
}

// Compile-time lc: the y table of a root lives in registers, every loop over components unrolls;
// blockIdx.y = component slice.
template <int LA, int LB, int LC>
__global__ void __launch_bounds__(GRAD_THREADS) k_rys_grad(GradArgs g) {
    using SL = GradSlices<LA, LB, LC>;
    constexpr int RS = 32 / SL::NR, RF = GradShape<LA, LB>::RF, UNR = LA + LB + LC <= 3 ? 2 : 1;
    constexpr int QB = grad_qb<LA, LB, LC>();
    static_for<SL::count()>([&](auto is) {
        constexpr int I = decltype(is)::value, FXA = SL::fx0(I), FXB = SL::fx0(I + 1), NFL = SL::nf(FXA, FXB);
        if (blockIdx.y == I) {
            const int lane = threadIdx.x & 31;
            grad_warp<LA, LB, SL::NR, RS, UNR>(
                g, NFL * RF * RS, g.warp_sz,
                [&](int tw, int pair, int ck, int k0, double* rows) {
                    constexpr int NAB = c_ncart(LA) * c_ncart(LB), PS = NFL * RF * RS;
                    const GradChunk c0 = g.chunks[ck];
                    const int* gi = g.gg.info + GG_N * c0.group;
                    const int ns = gi[GG_NS], nk = gi[GG_NK];
                    // shared group: its row offsets and coefficients once per warp, then item = (team, component)
                    const bool shared = g.tiled && !g.b_dummy && ns <= GRAD_MAXS;
                    long* off = reinterpret_cast<long*>(rows + g.qc * PS);
                    double* cf = reinterpret_cast<double*>(off + GRAD_MAXS);
                    if (shared) {
                        if (k0 == 0 && lane < ns)
                            off[lane] = (long)g.gg.aostart[g.gg.shells[gi[GG_SH] + lane]] * g.sP;
                        for (int i = lane; i < ns * QB; i += 32) {
                            const int k = k0 + i % QB;
                            cf[i] = k < c0.nq ? g.gg.coef[gi[GG_COEF] + (i / QB) * nk + c0.prim0 - gi[GG_P0] + k] : 0.0;
                        }
                        __syncwarp();
                    }
                    const int nit = tw * NFL;
                    for (int i0 = 0; i0 < nit; i0 += 32) {
                        const int it = i0 + lane, sl = it % tw;
                        int lf = it / tw;
                        const int pr = __shfl_sync(0xffffffffu, pair, sl * SL::NR);
                        const int c2 = __shfl_sync(0xffffffffu, ck, sl * SL::NR);
                        if (it >= nit || pr < 0) continue;
                        double* w = rows + lf * RF * RS + sl;
                        int fx = FXA;
                        while (lf > LC - fx) lf -= LC - fx++ + 1;
                        const int f = ((LC - fx) * (LC - fx + 1)) / 2 + lf;
                        double ABp[3][LB + 1];
                        if constexpr (LB > 0) grad_ab_powers<LB>(g, pr, ABp);
                        if (shared) {
                            const int shA = g.shA[pr], shB = g.shB[pr];
                            const double fac = shA != shB ? 2.0 : 1.0;  // both orders of an off-diagonal AO pair
                            double gam[QB][NAB];
                            grad_gamma_q<LA, LB, QB>(g.bar + (long)g.aostart[shA] * g.sM + (long)g.aostart[shB] * g.sN +
                                                         (long)f * g.sP,
                                                     g.sM, g.sN, off, cf, ns, gam);
#pragma unroll
                            for (int k = 0; k < QB; ++k) {
                                if (k0 + k >= c0.nq) break;
#pragma unroll
                                for (int i = 0; i < NAB; ++i) gam[k][i] *= fac;
                                grad_rows<LA, LB, RS>(gam[k], ABp, w + k * PS);
                            }
                        } else {
                            const GradChunk ch = g.chunks[c2];
#pragma unroll 1
                            for (int k = 0; k < QB && k0 + k < ch.nq; ++k) {
                                double gam[NAB];
                                grad_gamma<LA, LB>(g, ch, pr, ch.prim0 + k0 + k, f, 0, gam);
                                grad_rows<LA, LB, RS>(gam, ABp, w + k * PS);
                            }
                        }
                    }
                },
                [](const GradRoot& r, const double* w, GradSums& S) { grad_slice<LA, LB, LC, FXA, FXB, RS>(r, w, S); });
        }
    });
}

// Any lc, one component f per block (blockIdx.y): classes whose rows or unrolled code are too large,
// which have few tasks.  RS = the tasks per warp at the class family's smallest root count.  Two steps
// form the rows: the mixed adjoint by (team, a), then the recurrence by (team, ex), so that the lanes
// share what would be thousands of operations per team.
template <int LA, int LB, int RS>
__global__ void __launch_bounds__(GRAD_THREADS) k_rys_grad_f(GradArgs g) {
    constexpr int NA = c_ncart(LA), NB = c_ncart(LB), RF = GradShape<LA, LB>::RF, L1 = LA + LB;
    const int f = blockIdx.y, lane = threadIdx.x & 31;
    int s = 0, fz = f;  // s = lc - fx
    while (fz > s) fz -= ++s;
    const int fd[3] = {g.lc - s, s - fz, fz};
    grad_warp<LA, LB, 0, RS, 1>(
        g, RF * RS, g.warp_sz,
        [&](int tw, int pair, int ck, int k0, double* rows) {
            double* gam = LB == 0 ? rows : rows + RF * RS;  // [NA * NB][RS]
            for (int i0 = 0; i0 < tw * NA; i0 += 32) {
                const int it = i0 + lane, sl = it % tw, ia = it / tw;
                const int pr = __shfl_sync(0xffffffffu, pair, sl * g.nr);
                const int c2 = __shfl_sync(0xffffffffu, ck, sl * g.nr);
                if (ia >= NA || pr < 0) continue;
                const GradChunk ch = g.chunks[c2];
                if (k0 >= ch.nq) continue;
                double v[NB];
                grad_gamma<LA, LB>(g, ch, pr, ch.prim0 + k0, f, ia * NB, v);
#pragma unroll
                for (int i = 0; i < NB; ++i) gam[(ia * NB + i) * RS + sl] = v[i];
            }
            if constexpr (LB > 0) {
                constexpr bool UNROLL = LB < 3;
                constexpr int NIT = UNROLL ? L1 + 1 : GradShape<LA, LB>::NE;  // items per team: ex, or e
                __syncwarp();
                for (int i0 = 0; i0 < tw * NIT; i0 += 32) {
                    const int it = i0 + lane, sl = it % tw, j = it / tw;
                    const int pr = __shfl_sync(0xffffffffu, pair, sl * g.nr);
                    if (j >= NIT || pr < 0) continue;
                    double ABp[3][LB + 1];
                    grad_ab_powers<LB>(g, pr, ABp);
                    const auto gm = [&](int i) { return gam[i * RS + sl]; };
                    if constexpr (UNROLL) {
                        static_for<L1 + 1>([&](auto ix) {
                            constexpr int EX = decltype(ix)::value;
                            if (j == EX) grad_hrr_x<LA, LB, RS>(EX, ABp, gm, rows + sl);
                        });
                    } else {
                        grad_hrr_e<LA, LB, RS>(j, ABp, gm, rows + sl);
                    }
                }
            }
        },
        [&](const GradRoot& r, const double* w, GradSums& S) { grad_single<LA, LB, RS>(r, fd, w, S); });
}

// One launch of an angular class (dispatchers defined per (LA, LB) in dfb_grad_*.cu).
struct GradLaunch {
    GradArgs g;
    cudaStream_t st;
};

// Shared memory: gradient, then per warp the rows of qc primitives (prim doubles each) and extra doubles.
template <class K>
inline cudaError_t grad_launch(K kern, const GradLaunch& L, int qc, int prim, int extra, int ny) {
    GradArgs g = L.g;
    const int tw = 32 / g.nr;
    g.qc = qc;
    g.warp_sz = prim * g.qc + extra;
    const size_t sm = sizeof(double) * ((g.smem_grad ? 3 * g.natm : 0) + (size_t)GRAD_WARPS * g.warp_sz);
    if (sm > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    // tiles of pairs waste the end of the last tile: worth it from two tiles on
    g.tiled = g.npair >= 2 * tw;
    g.nwarp = g.tiled ? ((long)g.npair + tw - 1) / tw * g.nchunk : ((long)g.npair * g.nchunk + tw - 1) / tw;
    const long nblk = (g.nwarp + GRAD_WARPS - 1) / GRAD_WARPS;
    if (nblk > 2147483647L) return cudaErrorInvalidValue;
    kern<<<dim3((unsigned)nblk, ny), GRAD_THREADS, sm, L.st>>>(g);
    return cudaGetLastError();
}

// The register kernel takes a class up to (d d|, (f p| and (g s| when its y table is at most GRAD_TABLE
// doubles, its unrolled code at most GRAD_CODE multiply-adds, and one fx keeps to twice GRAD_ROW_BYTES.
constexpr int GRAD_TABLE = 36, GRAD_CODE = 3600;
template <int LA, int LB, int LC>
constexpr bool grad_fixed() {
    using G = GradShape<LA, LB>;
    constexpr int nf = c_ncart(LC), groups = (LA + LB + 1) * (LA + LB + 2) / 2;
    return LA + LB <= 4 && LC <= 6 && (LA + LB + 2) * (LC + 1) <= GRAD_TABLE &&
           nf * (2 * G::NE + 4 * groups + 4 * G::NLOW) <= GRAD_CODE &&
           (LC + 1) * G::RF * 8 <= 2 * GRAD_ROW_BYTES * GradSlices<LA, LB, LC>::NR;
}

template <int LA, int LB, int LC>  // lc >= LC
inline cudaError_t grad_launch_f(const GradLaunch& L) {
    constexpr int RS = 32 / ((LA + LB + LC + 1) / 2 + 1);
    return grad_launch(k_rys_grad_f<LA, LB, RS>, L, 1, GradShape<LA, LB>::RF * RS,
                       LB > 0 ? c_ncart(LA) * c_ncart(LB) * RS : 0, (L.g.lc + 1) * (L.g.lc + 2) / 2);
}

template <int LA, int LB, int LC = 0>
inline cudaError_t grad_launch_lc(const GradLaunch& L) {
    if constexpr (grad_fixed<LA, LB, LC>()) {
        using SL = GradSlices<LA, LB, LC>;
        if (L.g.lc == LC)
            return grad_launch(k_rys_grad<LA, LB, LC>, L, grad_qb<LA, LB, LC>(),
                               SL::max_nf() * GradShape<LA, LB>::RF * (32 / SL::NR),
                               GRAD_MAXS * (1 + grad_qb<LA, LB, LC>()), SL::count());
        return grad_launch_lc<LA, LB, LC + 1>(L);
    } else {
        return grad_launch_f<LA, LB, LC>(L);
    }
}

}  // namespace dfb
