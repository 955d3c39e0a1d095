// Integrals over primitive auxiliary functions, contracted per shared-exponent group.
//
// The auxiliary shells of a group are contractions of one primitive set, so (e 0|f) is evaluated
// once per (AO pair, primitive) into the rows of W (tiles of 32 pairs, 256-byte segments), and
// k_prim_out contracts a group's rows to its shells, applies the horizontal recurrence and writes
// the 3c tensor (k_prim_out2: both sides of the metric).  A wave takes whole groups over a range of pair tiles,
// so that its rows stay within the scratch given per stream (8 to 32 MB, or one group over one tile).
//
// (H2O)8/ma-TZVP, 416 AO / 1824 aux: 3c integrals 5.5 ms with one evaluation per shell, 4.75 ms here, of which
// the contraction k_prim_out takes most (its blocks wait on dependent loads); metric 0.80 -> 0.33 ms.
// (H2O)3/ma-QZVP, whole FP64 step: 52.7 -> 31.8 ms.
#pragma once
#include "dfb_grad_tmpl.cuh"

namespace dfb {

struct PrimArgs {
    const int *shA, *shB, *pstart, *npair_prim;
    const double* rec;   // as in GradArgs
    const double* cxyz;
    int b_dummy;
    const int* pairs;
    int npair, ntile;
    GradGroups gg;
    const GradChunk* chunks;
    int nchunk, row_base;
    double* W;  // [(row - row_base) * ntile + tile][nf * NE][32]
    int lc, nr;
    RysTable tab;
};

// Geometry of one primitive triplet.
struct PrimTriplet {
    double PA[3], CP[3], p, q, rp, rq, inv, T, pref;
};

__device__ __forceinline__ PrimTriplet prim_triplet(const PrimArgs& g, int iab, const double (&A)[3], const double (&C)[3],
                                                    double q, double rq) {
    PrimTriplet t;
    const GradPair pr = grad_pair(g.rec, g.b_dummy, iab, A);
    t.p = pr.p;
    t.q = q;
    t.rp = pr.rp;
    t.rq = rq;
    const double P0 = pr.P[0], P1 = pr.P[1], P2 = pr.P[2];
    t.PA[0] = pr.PA[0];
    t.PA[1] = pr.PA[1];
    t.PA[2] = pr.PA[2];
    t.CP[0] = C[0] - P0;
    t.CP[1] = C[1] - P1;
    t.CP[2] = C[2] - P2;
    const double s = rsqrt(t.p + q);
    t.inv = s * s;
    t.T = t.p * q * t.inv * (t.CP[0] * t.CP[0] + t.CP[1] * t.CP[1] + t.CP[2] * t.CP[2]);
    t.pref = pr.ckr * rq * s;
    return t;
}

// One component subset of one class: thread = AO pair, the primitives of the chunk one after the
// other, accumulators (e 0|f) in registers (CL: Cls<LA, LB, LC, FS, FSI, 0> of dfb_rys_tmpl.cuh).
template <class CL>
__device__ __forceinline__ void prim_body(const PrimArgs& g, const GradChunk& ch, int pi, double* sroot) {
    using R = typename CL::R;
    constexpr int NR = CL::NR, NM = CL::NM, NE = CL::ne(0), NF = CL::NF, RS = GRAD_THREADS;
    const int pair = g.pairs[pi];
    const int shA = g.shA[pair];
    const int rep = g.gg.info[GG_N * ch.group + GG_REP];
    const double A[3] = {g.cxyz[3 * shA], g.cxyz[3 * shA + 1], g.cxyz[3 * shA + 2]};
    const double C[3] = {g.gg.cxyz[3 * rep], g.gg.cxyz[3 * rep + 1], g.gg.cxyz[3 * rep + 2]};
    const int p0 = g.pstart[pair], p1 = p0 + g.npair_prim[pair];
    const double* cnr = g.tab.coef + g.tab.offs[NR];
    for (int k = 0; k < ch.nq; ++k) {
        const double q = g.gg.pexp[ch.prim0 + k], rq = g.gg.rexp[ch.prim0 + k];
        typename CL::Acc acc;
        CL::zero(acc);
        for (int iab = p0; iab < p1; ++iab) {
            const PrimTriplet t = prim_triplet(g, iab, A, C, q, rq);
            constexpr int NRR = NR <= 2 ? NR : 1;
            double xr[NRR], wr[NRR];
            if constexpr (NR <= 2)
                rys_eval_t<NR>(g.tab, cnr, t.T, xr, wr);
            else
                rys_eval_smem<NR, RS>(g.tab, cnr, t.T, sroot);
            const double qi = q * t.inv, pii = t.p * t.inv, h_p = 0.5 * t.rp, h_q = 0.5 * rq;
#pragma unroll
            for (int u = 0; u < NR; ++u) {
                double x, w;
                if constexpr (NR <= 2) {
                    x = xr[u < NRR ? u : 0];
                    w = wr[u < NRR ? u : 0];
                } else {
                    x = sroot[u * RS];
                    w = sroot[(NR + u) * RS];
                }
                const double B0 = x * 0.5 * t.inv;
                const double B1 = fma(1.0 - x, h_p, B0), B1p = fma(1.0 - x, h_q, B0);
                typename CL::GtX Gx;
                typename CL::GtY Gy;
                typename CL::GtZ Gz;
                const double fc = qi * x, fp = -pii * x;
                const R b0 = (R)B0, b1 = (R)B1, b1p = (R)B1p;
                build_G_t<NM, CL::MDX, R>(Gx, (R)(t.pref * w), (R)fma(fc, t.CP[0], t.PA[0]), (R)(fp * t.CP[0]), b0, b1, b1p);
                build_G_t<NM, CL::MDY, R>(Gy, R(1), (R)fma(fc, t.CP[1], t.PA[1]), (R)(fp * t.CP[1]), b0, b1, b1p);
                build_G_t<NM, CL::MDZ, R>(Gz, R(1), (R)fma(fc, t.CP[2], t.PA[2]), (R)(fp * t.CP[2]), b0, b1, b1p);
                CL::acc_all(acc, Gx, Gy, Gz, R(0), R(0));
            }
        }
        double* w = g.W + ((long)(ch.row0 + k - g.row_base) * g.ntile + (pi >> 5)) * (NF * NE * 32) + (pi & 31);
#pragma unroll
        for (int f = 0; f < CL::NL; ++f)
#pragma unroll
            for (int e = 0; e < NE; ++e) w[32 * ((CL::F0 + f) * NE + e)] = (double)acc.a0[e][f];
    }
}

// R = float: the recurrence tables and the accumulators of each primitive in FP32 (mixed mode).
template <int LA, int LB, int LC, int FS, typename R>
__global__ void __launch_bounds__(GRAD_THREADS) k_prim_int(PrimArgs g) {
    __shared__ double sroots[((LA + LB + LC) / 2 + 1 > 2) ? 2 * ((LA + LB + LC) / 2 + 1) * GRAD_THREADS : 1];
    const int pi = blockIdx.z * GRAD_THREADS + threadIdx.x;  // heaviest pairs first, for every chunk
    if (pi >= g.npair) return;
    const GradChunk ch = g.chunks[blockIdx.x];
    if (pi < ch.plo) return;
    static_for<FS>([&](auto i) {
        constexpr int I = decltype(i)::value;
        if (blockIdx.y == I) prim_body<Cls<LA, LB, LC, FS, I, 0, R>>(g, ch, pi, sroots + threadIdx.x);
    });
}

// Any lc, one aux component f per thread (blockIdx.y): columns fx, fy and fz of the recurrence tables
// are built by their recurrences for each root; the accumulators are the NE functions e.
template <int LA, int LB>
__global__ void __launch_bounds__(GRAD_THREADS) k_prim_int_f(PrimArgs g) {
    constexpr int L1 = LA + LB, NE = GradShape<LA, LB>::NE;
    const int pi = blockIdx.z * GRAD_THREADS + threadIdx.x;  // heaviest pairs first, for every chunk
    if (pi >= g.npair) return;
    const GradChunk ch = g.chunks[blockIdx.x];
    if (pi < ch.plo) return;
    const int lc = g.lc, nr = g.nr, f = blockIdx.y, nf = (lc + 1) * (lc + 2) / 2;
    int s = 0, fz = f;  // s = lc - fx
    while (fz > s) fz -= ++s;
    const int fx = lc - s, fy = s - fz;
    const int pair = g.pairs[pi];
    const int shA = g.shA[pair];
    const int rep = g.gg.info[GG_N * ch.group + GG_REP];
    const double A[3] = {g.cxyz[3 * shA], g.cxyz[3 * shA + 1], g.cxyz[3 * shA + 2]};
    const double C[3] = {g.gg.cxyz[3 * rep], g.gg.cxyz[3 * rep + 1], g.gg.cxyz[3 * rep + 2]};
    const int p0 = g.pstart[pair], p1 = p0 + g.npair_prim[pair];
    for (int k = 0; k < ch.nq; ++k) {
        const double q = g.gg.pexp[ch.prim0 + k], rq = g.gg.rexp[ch.prim0 + k];
        double acc[NE];
#pragma unroll
        for (int e = 0; e < NE; ++e) acc[e] = 0.0;
        for (int iab = p0; iab < p1; ++iab) {
            const PrimTriplet t = prim_triplet(g, iab, A, C, q, rq);
#pragma unroll 1
            for (int u = 0; u < nr; ++u) {
                double x, w;
                rys_one(g.tab, nr, u, t.T, x, w);
                const double B0 = 0.5 * x * t.inv;
                const double B1 = fma(0.5 * (1.0 - x), t.rp, B0), B1p = fma(0.5 * (1.0 - x), rq, B0);
                const double fc = q * t.inv * x, fp = -t.p * t.inv * x;
                double X[L1 + 1], Y[L1 + 1], Z[L1 + 1];
                auto column = [&](double(&c)[L1 + 1], double g00, int d, int n) {
                    double prev[L1 + 1];
                    rys_col0<L1>(c, g00, fma(fc, d == 0 ? t.CP[0] : d == 1 ? t.CP[1] : t.CP[2],
                                             d == 0 ? t.PA[0] : d == 1 ? t.PA[1] : t.PA[2]), B1);
#pragma unroll
                    for (int a = 0; a <= L1; ++a) prev[a] = 0.0;
                    const double Cp = fp * (d == 0 ? t.CP[0] : d == 1 ? t.CP[1] : t.CP[2]);
#pragma unroll 1
                    for (int b = 0; b < n; ++b) rys_coln<L1>(c, prev, Cp, B0, (double)b * B1p);
                };
                column(X, t.pref * w, 0, fx);
                column(Y, 1.0, 1, fy);
                column(Z, 1.0, 2, fz);
                static_for<L1 + 1>([&](auto iex) {
                    static_for<L1 + 1>([&](auto iey) {
                        constexpr int ex = decltype(iex)::value, ey = decltype(iey)::value;
                        if constexpr (ex + ey <= L1) {
                            const double xy = X[ex] * Y[ey];
                            static_for<L1 + 1>([&](auto iez) {
                                constexpr int ez = decltype(iez)::value, l = ex + ey + ez;
                                if constexpr (l >= LA && l <= L1) {
                                    constexpr int e = c_eidx(LA, ex, ey, ez);
                                    acc[e] = fma(xy, Z[ez], acc[e]);
                                }
                            });
                        }
                    });
                });
            }
        }
        double* w = g.W + ((long)(ch.row0 + k - g.row_base) * g.ntile + (pi >> 5)) * ((long)nf * NE * 32) +
                    (long)f * NE * 32 + (pi & 31);
#pragma unroll
        for (int e = 0; e < NE; ++e) w[32 * e] = acc[e];
    }
}

struct PrimOutArgs {
    const int *shA, *shB;
    const double* cxyz;
    const int* aostart;
    const int* pairs;
    int npair, ntile;
    GradGroups gg;
    const int2* groups;  // (group, first row) of the wave
    int row_base;
    const double* W;
    double* out;
    long sP, sM, sN;
    int lc;
    int nbatch;          // blocks over the shells of a group
};

// Shells per block of the contraction: as many as registers allow, since every batch reads the group's rows
// again (the blocks of the other batches are neighbours).
template <int LA, int LB>
__host__ __device__ constexpr int prim_batch() {
    constexpr int ne = GradShape<LA, LB>::NE;
    return ne <= 6 ? 6 : ne <= 10 ? 5 : ne <= 16 ? 3 : ne <= 31 ? 2 : 1;
}
constexpr int PRIM_COEF = 32;  // primitives whose coefficients a block keeps in shared memory

// Warps per block: the staged values of a block stay near 50 KB.
template <int LA, int LB>
__host__ __device__ constexpr int prim_warps() {
    return c_ncart(LA) * c_ncart(LB) <= 36 ? 4 : c_ncart(LA) * c_ncart(LB) <= 100 ? 2 : 1;
}

template <int LA, int LB>
__global__ void __launch_bounds__(32 * prim_warps<LA, LB>()) k_prim_out(PrimOutArgs m) {
    using G = GradShape<LA, LB>;
    constexpr int NE = G::NE, BS = prim_batch<LA, LB>(), NA = c_ncart(LA), NB = c_ncart(LB), NAB = NA * NB;
    extern __shared__ double stage_all[];  // [warp][NAB][33]
    __shared__ int s_ao[32 * prim_warps<LA, LB>()][2];
    __shared__ double s_cf[BS * PRIM_COEF];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile = blockIdx.x / m.nbatch, s0 = (blockIdx.x - tile * m.nbatch) * BS;
    double* stage = stage_all + warp * NAB * 33;
    const int pi0 = (tile * prim_warps<LA, LB>() + warp) * 32, pi = pi0 + lane;
    const int np = m.npair - pi0 < 32 ? m.npair - pi0 : 32;  // pairs of this warp
    const int2 gr = m.groups[blockIdx.z];
    const int* gi = m.gg.info + GG_N * gr.x;
    const int ns = gi[GG_NS], nk = gi[GG_NK];
    if (s0 >= ns) return;
    const double* cf = m.gg.coef + gi[GG_COEF];
    const bool keep = nk <= PRIM_COEF;
    if (keep)
        for (int i = threadIdx.x; i < BS * nk; i += blockDim.x)
            s_cf[i] = s0 + i % BS < ns ? cf[(s0 + i % BS) * nk + i / BS] : 0.0;
    __syncthreads();
    if (np <= 0) return;
    const bool on = lane < np;
    const int f = blockIdx.y, nf = (m.lc + 1) * (m.lc + 2) / 2;
    const int pair = m.pairs[on ? pi : pi0];
    const int shA = m.shA[pair], shB = m.shB[pair];
    double ABp[3][LB + 1];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double ab = m.cxyz[3 * shA + d] - m.cxyz[3 * shB + d];
        ABp[d][0] = 1.0;
#pragma unroll
        for (int k = 1; k <= LB; ++k) ABp[d][k] = ABp[d][k - 1] * ab;
    }
    s_ao[threadIdx.x][0] = m.aostart[shA];
    s_ao[threadIdx.x][1] = m.aostart[shB];
    const int* sh = m.gg.shells + gi[GG_SH];
    const long row_sz = (long)m.ntile * nf * NE * 32;
    const double* w0 = m.W + (long)(gr.y - m.row_base) * row_sz + ((long)(pi0 >> 5) * nf + f) * (NE * 32) + (on ? lane : 0);
    {
        double E[BS][NE];
#pragma unroll
        for (int s = 0; s < BS; ++s)
#pragma unroll
            for (int e = 0; e < NE; ++e) E[s][e] = 0.0;
        const double* w = w0;
        constexpr int UK = NE <= 3 ? 8 : NE <= 10 ? 4 : NE <= 16 ? 2 : 1;  // rows in flight
#pragma unroll UK
        for (int k = 0; k < nk; ++k) {
            double c[BS];
#pragma unroll
            for (int s = 0; s < BS; ++s)
                c[s] = keep ? s_cf[k * BS + s] : s0 + s < ns ? __ldg(cf + (s0 + s) * nk + k) : 0.0;
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const double v = __ldg(w + k * row_sz + 32 * e);
#pragma unroll
                for (int s = 0; s < BS; ++s) E[s][e] = fma(c[s], v, E[s][e]);
            }
        }
#pragma unroll
        for (int s = 0; s < BS; ++s) {
            if (s0 + s >= ns) break;
            double* o = m.out + (long)(m.gg.aostart[sh[s0 + s]] + f) * m.sP;
            __syncwarp();  // the previous shell's values are written (and s_ao is set)
            // (a b| = sum_k C(b,k) AB^(b-k) (a+k|
#pragma unroll
            for (int ax = 0; ax <= LA; ++ax) {
#pragma unroll
                for (int ay = 0; ay <= LA; ++ay) {
#pragma unroll
                    for (int bx = 0; bx <= LB; ++bx) {
#pragma unroll
                        for (int by = 0; by <= LB; ++by) {
                            const int az = LA - ax - ay, bz = LB - bx - by;
                            if (az < 0 || bz < 0) continue;
                            double v = 0.0;
#pragma unroll
                            for (int kx = 0; kx <= LB; ++kx) {
#pragma unroll
                                for (int ky = 0; ky <= LB; ++ky) {
#pragma unroll
                                    for (int kz = 0; kz <= LB; ++kz) {
                                        if (kx > bx || ky > by || kz > bz) continue;
                                        const double c = (double)(c_bin(bx, kx) * c_bin(by, ky) * c_bin(bz, kz)) *
                                                         ABp[0][bx - kx] * ABp[1][by - ky] * ABp[2][bz - kz];
                                        v = fma(c, E[s][c_eidx(LA, ax + kx, ay + ky, az + kz)], v);
                                    }
                                }
                            }
                            const int ia = ((LA - ax) * (LA - ax + 1)) / 2 + az, ib = ((LB - bx) * (LB - bx + 1)) / 2 + bz;
                            stage[(ia * NB + ib) * 33 + lane] = v;
                        }
                    }
                }
            }
            __syncwarp();
            const int rowlen = np * NB;
            for (int ia = 0; ia < NA; ++ia) {
                for (int j = lane; j < rowlen; j += 32) {
                    const int pr = j / NB, ib = j - pr * NB;
                    const long mu = s_ao[warp * 32 + pr][0] + ia, nu = s_ao[warp * 32 + pr][1] + ib;
                    o[mu * m.sM + nu * m.sN] = stage[(ia * NB + ib) * 33 + pr];
                }
            }
            for (int j = lane; j < np * NAB; j += 32) {
                const int ia = j % NA, rest = j / NA;
                const int ib = rest % NB, pr = rest / NB;
                const long mu = s_ao[warp * 32 + pr][0] + ia, nu = s_ao[warp * 32 + pr][1] + ib;
                o[nu * m.sM + mu * m.sN] = stage[(ia * NB + ib) * 33 + pr];
            }
        }
    }
}

// Launches of one angular class (defined per (LA, LB) in dfb_prim_*.cu).
struct PrimLaunch {
    PrimArgs g;
    PrimOutArgs m;
    int ngroup, f32, max_ns;
    cudaStream_t st;
};

template <int LA, int LB>
inline cudaError_t prim_launch_out(const PrimLaunch& L) {
    const int nf = (L.g.lc + 1) * (L.g.lc + 2) / 2;
    constexpr int nt = 32 * prim_warps<LA, LB>();
    constexpr size_t sm = sizeof(double) * prim_warps<LA, LB>() * c_ncart(LA) * c_ncart(LB) * 33;
    if (sm > 40 * 1024) {  // static shared memory beside it
        cudaError_t e = cudaFuncSetAttribute(k_prim_out<LA, LB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    PrimOutArgs m = L.m;
    m.nbatch = (L.max_ns + prim_batch<LA, LB>() - 1) / prim_batch<LA, LB>();
    const long nx = ((long)L.g.npair + nt - 1) / nt * m.nbatch;
    if (nx > 2147483647L) return cudaErrorInvalidValue;
    k_prim_out<LA, LB><<<dim3((unsigned)nx, nf, L.ngroup), nt, sm, L.st>>>(m);
    return cudaGetLastError();
}

template <int LA, int LB>
inline cudaError_t prim_launch_f(const PrimLaunch& L) {
    const int nf = (L.g.lc + 1) * (L.g.lc + 2) / 2;
    k_prim_int_f<LA, LB><<<dim3(L.g.nchunk, nf, (L.g.npair + GRAD_THREADS - 1) / GRAD_THREADS), GRAD_THREADS, 0, L.st>>>(L.g);
    return cudaGetLastError();
}

// Subsets of the aux components for classes on the register kernel: the fewest for which a subset's
// accumulators stay within BUD doubles; 0 = more than 8 subsets would be needed.
constexpr int PRIM_ACC = 48;
template <int LA, int LB, int LC>
constexpr int prim_fs() {
    const int nf = c_ncart(LC), ne = GradShape<LA, LB>::NE;
    for (int fs = 1; fs <= nf && fs <= 8; ++fs) {
        const int nfs = (nf + fs - 1) / fs;
        if ((nf + nfs - 1) / nfs == fs && nfs * ne <= PRIM_ACC) return fs;
    }
    return 0;
}

template <int LA, int LB, int LC = 0>
inline cudaError_t prim_launch_int(const PrimLaunch& L) {
    if constexpr (LC <= 6) {
        constexpr int FS = prim_fs<LA, LB, LC>();
        if constexpr (FS > 0) {
            if (L.g.lc == LC) {
                const dim3 grid(L.g.nchunk, FS, (L.g.npair + GRAD_THREADS - 1) / GRAD_THREADS);
                if (L.f32)
                    k_prim_int<LA, LB, LC, FS, float><<<grid, GRAD_THREADS, 0, L.st>>>(L.g);
                else
                    k_prim_int<LA, LB, LC, FS, double><<<grid, GRAD_THREADS, 0, L.st>>>(L.g);
                return cudaGetLastError();
            }
            return prim_launch_int<LA, LB, LC + 1>(L);
        }
    }
    return prim_launch_f<LA, LB>(L);
}

}  // namespace dfb
