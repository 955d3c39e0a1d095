// Host side of the primitive-group integrals (kernels: dfb_prim_tmpl.cuh) and the two-sided
// contraction of the metric.

#include "../../include/dfb.h"
#include "dfb_internal.h"
#include "dfb_prim_tmpl.cuh"

namespace dfb {

#define DFB_PRIM_DECL(A, B)                        \
    cudaError_t prim_int_##A##B(const PrimLaunch&); \
    cudaError_t prim_out_##A##B(const PrimLaunch&);
DFB_PRIM_DECL(0, 0)
DFB_PRIM_DECL(1, 0)
DFB_PRIM_DECL(1, 1)
DFB_PRIM_DECL(2, 0)
DFB_PRIM_DECL(2, 1)
DFB_PRIM_DECL(2, 2)
DFB_PRIM_DECL(3, 0)
DFB_PRIM_DECL(3, 1)
DFB_PRIM_DECL(3, 2)
DFB_PRIM_DECL(3, 3)
DFB_PRIM_DECL(4, 0)
DFB_PRIM_DECL(4, 1)
DFB_PRIM_DECL(4, 2)
DFB_PRIM_DECL(4, 3)
DFB_PRIM_DECL(4, 4)
#undef DFB_PRIM_DECL
cudaError_t prim_int_50(const PrimLaunch&);
cudaError_t prim_int_60(const PrimLaunch&);
cudaError_t prim_int_70(const PrimLaunch&);
cudaError_t prim_int_80(const PrimLaunch&);

typedef cudaError_t (*prim_fn)(const PrimLaunch&);
static const prim_fn kOut[5][5] = {
    {prim_out_00, nullptr, nullptr, nullptr, nullptr},
    {prim_out_10, prim_out_11, nullptr, nullptr, nullptr},
    {prim_out_20, prim_out_21, prim_out_22, nullptr, nullptr},
    {prim_out_30, prim_out_31, prim_out_32, prim_out_33, nullptr},
    {prim_out_40, prim_out_41, prim_out_42, prim_out_43, prim_out_44}};
static const prim_fn kInt[9][5] = {
    {prim_int_00, nullptr, nullptr, nullptr, nullptr},
    {prim_int_10, prim_int_11, nullptr, nullptr, nullptr},
    {prim_int_20, prim_int_21, prim_int_22, nullptr, nullptr},
    {prim_int_30, prim_int_31, prim_int_32, prim_int_33, nullptr},
    {prim_int_40, prim_int_41, prim_int_42, prim_int_43, prim_int_44},
    {prim_int_50}, {prim_int_60}, {prim_int_70}, {prim_int_80}};

const RysTable* rys_table_of_current_device();  // dfb_rys.cu; nullptr before the upload

// Metric: V[(t, a), (s, f)] = sum_pq c_tp c_sq E_q[f][a][p] for one (bra group, ket group); thread =
// element (f, a), up to PRIM_MB x PRIM_MB shell pairs per pass.  blockIdx.x = bra group, blockIdx.y =
// ket group of the wave.  With equal l the bra groups before the ket group are left to the mirrored
// pair; a group with itself writes each element once.
constexpr int PRIM_MB = 6;
__global__ void __launch_bounds__(128) k_prim_out2(PrimOutArgs m, const int* __restrict__ bgroups, int bra_p0, int la,
                                                   int same_l) {
    const int gb = bgroups[blockIdx.x];
    const int2 gr = m.groups[blockIdx.y];
    if (same_l && gb < gr.x) return;
    const int na = ncart(la), nf = ncart(m.lc);
    const int* bi = m.gg.info + GG_N * gb;
    const int* ki = m.gg.info + GG_N * gr.x;
    const int nst = bi[GG_NS], nkt = bi[GG_NK], nss = ki[GG_NS], nks = ki[GG_NK];
    const double* ct = m.gg.coef + bi[GG_COEF];
    const double* cs = m.gg.coef + ki[GG_COEF];
    const int pl0 = bi[GG_P0] - bra_p0;
    const long tile_sz = (long)nf * na * 32, row_sz = (long)m.ntile * tile_sz;
    const double* w0 = m.W + (long)(gr.y - m.row_base) * row_sz;
    for (int el = threadIdx.x; el < na * nf; el += blockDim.x) {
        const int f = el / na, a = el - f * na;
        for (int t0 = 0; t0 < nst; t0 += PRIM_MB) {
            for (int s0 = 0; s0 < nss; s0 += PRIM_MB) {
                double acc[PRIM_MB][PRIM_MB];
#pragma unroll
                for (int t = 0; t < PRIM_MB; ++t)
#pragma unroll
                    for (int s = 0; s < PRIM_MB; ++s) acc[t][s] = 0.0;
                for (int q = 0; q < nks; ++q) {
                    double u[PRIM_MB];
#pragma unroll
                    for (int t = 0; t < PRIM_MB; ++t) u[t] = 0.0;
                    const double* w = w0 + q * row_sz + (long)el * 32;
                    for (int p = 0; p < nkt; ++p) {
                        const int pl = pl0 + p;
                        const double v = __ldg(w + (pl >> 5) * tile_sz + (pl & 31));
#pragma unroll
                        for (int t = 0; t < PRIM_MB; ++t)
                            if (t0 + t < nst) u[t] = fma(__ldg(ct + (t0 + t) * nkt + p), v, u[t]);
                    }
#pragma unroll
                    for (int s = 0; s < PRIM_MB; ++s) {
                        if (s0 + s >= nss) break;
                        const double c = __ldg(cs + (s0 + s) * nks + q);
#pragma unroll
                        for (int t = 0; t < PRIM_MB; ++t) acc[t][s] = fma(c, u[t], acc[t][s]);
                    }
                }
#pragma unroll
                for (int t = 0; t < PRIM_MB; ++t) {
                    if (t0 + t >= nst) break;
                    const long P = m.gg.aostart[m.gg.shells[bi[GG_SH] + t0 + t]] + a;
#pragma unroll
                    for (int s = 0; s < PRIM_MB; ++s) {
                        if (s0 + s >= nss) break;
                        const long Q = m.gg.aostart[m.gg.shells[ki[GG_SH] + s0 + s]] + f;
                        m.out[P * m.sP + Q * m.sM] = acc[t][s];
                        if (gb != gr.x) m.out[Q * m.sP + P * m.sM] = acc[t][s];
                    }
                }
            }
        }
    }
}

// Zeros for AO pairs without primitive pairs: thread = element of the pair's block, blockIdx.x = pair,
// blockIdx.y strides over the aux functions.  The index of the smaller stride runs fastest.
__global__ void __launch_bounds__(128) k_zero_pairs(const int* __restrict__ list, const int* __restrict__ shA,
                                                    const int* __restrict__ shB, const int* __restrict__ aostart,
                                                    const int* __restrict__ nao_sh, long naux, double* __restrict__ out,
                                                    long sP, long sM, long sN) {
    const int pair = list[blockIdx.x];
    const int A = shA[pair], B = shB[pair];
    const int na = nao_sh[A], nb = nao_sh[B];
    const bool p_first = sP < sN;
    for (long i = (long)blockIdx.y * blockDim.x + threadIdx.x; i < naux * na * nb; i += (long)gridDim.y * blockDim.x) {
        const long P = p_first ? i % naux : i / (na * nb);
        const int ab = (int)(p_first ? i / naux : i % (na * nb)), ia = ab / nb, ib = ab - ia * nb;
        const long mu = aostart[A] + ia, nu = aostart[B] + ib;
        out[P * sP + mu * sM + nu * sN] = 0.0;
        out[P * sP + nu * sM + mu * sN] = 0.0;
    }
}

static long prim_row(int la, int lb, int lc) {
    return (long)(ncart_below(la + lb + 1) - ncart_below(la)) * ncart(lc);
}

}  // namespace dfb

using namespace dfb;

// Doubles of one row over a tile of 32 pairs; the most rows of one group.
static long tile_row(const dfb_prim_class_t& c) { return prim_row(c.la, c.lb, c.lc) * 32; }
static long group_rows(const dfb_prim_class_t& c) {
    long most = 0;
    for (int k = 0; k < c.ngroup; ++k) most = c.rows[k + 1] - c.rows[k] > most ? c.rows[k + 1] - c.rows[k] : most;
    return most;
}

// A wave holds whole groups.  `target` doubles bound it unless one group takes more: then one group over all pairs up
// to PRIM_OVER times the target, and over a range of pair tiles beyond (at least one tile).  Cutting the pairs costs
// launches and short waves: integrals of 12 waters TZVP in blocks, where one group over all pairs is 1.0 to 1.7 of
// 8 MB, 17.0 ms cut and 15.5 uncut.  The metric contracts pairs of groups: its waves hold all pairs, whose
// count grows with the primitives of one l only.
constexpr long PRIM_OVER = 4;
extern "C" long dfb_prim_scratch(const dfb_prim_class_t* cls, int ncls, long target) {
    long need = 1;
    for (int i = 0; i < ncls; ++i) {
        const dfb_prim_class_t& c = cls[i];
        if (c.ngroup <= 0 || c.npair <= 0) continue;
        const long tiles = ((long)c.npair + 31) / 32, one = group_rows(c) * tile_row(c);
        long n = one * tiles;
        if (!c.bra_groups && n > PRIM_OVER * target) n = one > PRIM_OVER * target ? one : PRIM_OVER * target;
        if (n < target) n = target;
        const long all = c.rows[c.ngroup] * tile_row(c) * tiles;
        if (n > all) n = all;
        if (n > need) need = n;
    }
    return need;
}

extern "C" int dfb_prim_integrals(const dfb_bra_t* bra, const dfb_groups_t* gr, const dfb_prim_class_t* cls, int ncls,
                                  double* out, long sP, long sM, long sN, double* scratch, long scratch_doubles,
                                  void* const* streams, int nstreams) {
    clear_error();
    if (!bra || !gr || (ncls > 0 && !cls) || !out || nstreams < 1 || !streams || !scratch)
        return set_error(DFB_ERR_INVALID, "invalid arguments to dfb_prim_integrals");
    const RysTable* tab = rys_table_of_current_device();
    if (!tab) return set_error(DFB_ERR_NOT_INITIALISED, "Rys table not uploaded on this device");
    const long slice = (scratch_doubles / nstreams) & ~31L;
    for (int i = 0; i < ncls; ++i) {
        const dfb_prim_class_t& c = cls[i];
        if (!dfb_grad_supported(c.la, c.lb, c.lc, bra->b_dummy))
            return set_error(DFB_ERR_UNSUPPORTED, "integral class (%d,%d,%d) is not supported", c.la, c.lb, c.lc);
        if (c.npair <= 0 || c.ngroup <= 0) continue;
        if (!c.pairs || !c.chunks || !c.groups || !c.rows || !c.first_chunk || c.max_shells < 1 || (bra->b_dummy && !c.bra_groups))
            return set_error(DFB_ERR_INVALID, "integral class without lists");
        cudaStream_t st = (cudaStream_t)streams[i % nstreams];
        double* W = scratch + (i % nstreams) * slice;
        PrimLaunch L;
        L.st = st;
        L.f32 = c.f32;
        L.max_ns = c.max_shells;
        PrimArgs& g = L.g;
        g.shA = bra->shA;
        g.shB = bra->shB;
        g.pstart = bra->pstart;
        g.npair_prim = bra->npair;
        g.rec = bra->rec;
        g.cxyz = bra->cxyz;
        g.b_dummy = bra->b_dummy;
        g.gg = {gr->info, gr->coef, gr->shells, gr->pexp, gr->rexp, gr->cxyz, gr->aostart, gr->atom};
        g.W = W;
        g.lc = c.lc;
        g.nr = (c.la + c.lb + c.lc) / 2 + 1;
        g.tab = *tab;
        PrimOutArgs& m = L.m;
        m.shA = bra->shA;
        m.shB = bra->shB;
        m.cxyz = bra->cxyz;
        m.aostart = bra->aostart;
        m.gg = g.gg;
        m.W = W;
        m.out = out;
        m.sP = sP;
        m.sM = sM;
        m.sN = sN;
        m.lc = c.lc;
        // tiles of a wave: all of them where one group over all fits, else what does (blockIdx.z covers 65535 x 128
        // pairs)
        const long tiles = ((long)c.npair + 31) / 32, big = group_rows(c);
        long step = tiles;
        if (!bra->b_dummy) {
            const long fit = big > 0 ? slice / (big * tile_row(c)) : tiles, grid = 65535L * (GRAD_THREADS / 32);
            step = tiles < fit ? tiles : fit;
            step = step < grid ? step : grid;
            if (step > 0) step = (tiles + (tiles + step - 1) / step - 1) / ((tiles + step - 1) / step);  // equal ranges
        }
        if (step < 1)
            return set_error(DFB_ERR_INVALID, "class (%d,%d,%d) needs %ld scratch doubles per stream, %ld given", c.la, c.lb,
                             c.lc, big * tile_row(c), slice);
        for (long t0 = 0; t0 < tiles; t0 += step) {
            const long p0 = 32 * t0, np = c.npair - p0 < 32 * step ? c.npair - p0 : 32 * step;
            g.pairs = m.pairs = c.pairs + p0;
            g.npair = m.npair = (int)np;
            g.ntile = m.ntile = (int)((np + 31) / 32);
            const long row = tile_row(c) * g.ntile;
            for (int k0 = 0; k0 < c.ngroup;) {
                // one wave: as many whole groups as the stream's slice of W holds
                int k1 = k0;
                while (k1 < c.ngroup && c.first_chunk[k1 + 1] - c.first_chunk[k0] <= 65535 &&
                       (c.rows[k1 + 1] - c.rows[k0]) * row <= slice)
                    ++k1;
                if (k1 == k0)
                    return set_error(DFB_ERR_INVALID, "class (%d,%d,%d) needs %ld scratch doubles per stream, %ld given",
                                     c.la, c.lb, c.lc, (c.rows[k0 + 1] - c.rows[k0]) * row, slice);
                g.chunks = reinterpret_cast<const GradChunk*>(c.chunks) + c.first_chunk[k0];
                g.nchunk = (int)(c.first_chunk[k1] - c.first_chunk[k0]);
                g.row_base = m.row_base = (int)c.rows[k0];
                m.groups = reinterpret_cast<const int2*>(c.groups) + k0;
                L.ngroup = k1 - k0;
                cudaError_t e = kInt[c.la][c.lb](L);
                if (e != cudaSuccess) return set_cuda_error("primitive integral launch", e);
                if (bra->b_dummy) {
                    k_prim_out2<<<dim3(c.nbra_groups, L.ngroup), 128, 0, st>>>(m, c.bra_groups, c.bra_prim0, c.la,
                                                                              c.la == c.lc);
                    e = cudaGetLastError();
                } else {
                    e = kOut[c.la][c.lb](L);
                }
                if (e != cudaSuccess) return set_cuda_error("group contraction launch", e);
                count_launches(2);
                k0 = k1;
            }
        }
    }
    return DFB_OK;
}

extern "C" int dfb_zero_pairs(const dfb_bra_t* bra, const int* list, int npairs, const int* shell_size, long naux,
                              double* out, long sP, long sM, long sN, void* stream) {
    clear_error();
    if (!bra || npairs < 0 || naux < 0 || (npairs > 0 && (!list || !shell_size || !out)))
        return set_error(DFB_ERR_INVALID, "invalid arguments to dfb_zero_pairs");
    if (npairs == 0 || naux == 0) return DFB_OK;
    long ny = (naux + 127) / 128;
    if (ny > 64) ny = 64;
    k_zero_pairs<<<dim3((unsigned)npairs, (unsigned)ny), 128, 0, (cudaStream_t)stream>>>(
        list, bra->shA, bra->shB, bra->aostart, shell_size, naux, out, sP, sM, sN);
    count_launches(1);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DFB_OK : set_cuda_error("k_zero_pairs launch", e);
}
