// Host side of the adjoint-first derivative contraction (kernels: dfb_grad_tmpl.cuh).

#include <stdint.h>

#include "../../include/dfb.h"
#include "dfb_grad_tmpl.cuh"
#include "dfb_internal.h"

namespace dfb {

#define DFB_GRAD_DECL(A, B) cudaError_t grad_run_##A##B(const GradLaunch&);
DFB_GRAD_DECL(0, 0)
DFB_GRAD_DECL(1, 0)
DFB_GRAD_DECL(1, 1)
DFB_GRAD_DECL(2, 0)
DFB_GRAD_DECL(2, 1)
DFB_GRAD_DECL(2, 2)
DFB_GRAD_DECL(3, 0)
DFB_GRAD_DECL(3, 1)
DFB_GRAD_DECL(3, 2)
DFB_GRAD_DECL(3, 3)
DFB_GRAD_DECL(4, 0)
DFB_GRAD_DECL(4, 1)
DFB_GRAD_DECL(4, 2)
DFB_GRAD_DECL(4, 3)
DFB_GRAD_DECL(4, 4)
#undef DFB_GRAD_DECL
cudaError_t grad_run_50(const GradLaunch&);
cudaError_t grad_run_60(const GradLaunch&);
cudaError_t grad_run_70(const GradLaunch&);
cudaError_t grad_run_80(const GradLaunch&);

typedef cudaError_t (*grad_fn)(const GradLaunch&);
static const grad_fn kRun[9][5] = {
    {grad_run_00, nullptr, nullptr, nullptr, nullptr},
    {grad_run_10, grad_run_11, nullptr, nullptr, nullptr},
    {grad_run_20, grad_run_21, grad_run_22, nullptr, nullptr},
    {grad_run_30, grad_run_31, grad_run_32, grad_run_33, nullptr},
    {grad_run_40, grad_run_41, grad_run_42, grad_run_43, grad_run_44},
    {grad_run_50}, {grad_run_60}, {grad_run_70}, {grad_run_80}};

static bool grad_has(int la, int lb, int lc, bool dummy) {
    if (la < 0 || lb < 0 || lc < 0 || lb > la || lc > DFB_LMAX) return false;
    if (dummy) return lb == 0 && la <= 8;
    return la <= 4;
}

// Records of the primitive pairs, 64 bytes each (a kernel's lanes gather them with four 16-byte loads):
// p, 1/p, the prefactor 2 pi^(5/2) cK / p, P, 2a, 2b.
__global__ void k_pair_ext(long n, const double* __restrict__ eta, const double* __restrict__ Px,
                           const double* __restrict__ Py, const double* __restrict__ Pz, const double* __restrict__ cK,
                           const double* __restrict__ ea, const double* __restrict__ eb, double* __restrict__ rec) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double p = eta[i], r = 1.0 / p;
    double2* q = reinterpret_cast<double2*>(rec) + 4 * i;
    q[0] = make_double2(p, r);
    q[1] = make_double2(kTwoPi52_t * cK[i] * r, Px[i]);
    q[2] = make_double2(Py[i], Pz[i]);
    q[3] = make_double2(2.0 * ea[i], 2.0 * eb[i]);
}

const RysTable* rys_table_of_current_device();  // dfb_rys.cu; nullptr before the upload

}  // namespace dfb

using namespace dfb;

extern "C" int dfb_pair_ext(const double* eta, const double* Px, const double* Py, const double* Pz, const double* cK,
                            const double* ea, const double* eb, long npp, double* rec, void* stream) {
    clear_error();
    if (npp < 0 || (npp > 0 && (!eta || !Px || !Py || !Pz || !cK || !ea || !eb || !rec || ((uintptr_t)rec & 15))))
        return set_error(DFB_ERR_INVALID, "invalid arguments to dfb_pair_ext");
    if (npp == 0) return DFB_OK;
    k_pair_ext<<<(unsigned)((npp + 255) / 256), 256, 0, (cudaStream_t)stream>>>(npp, eta, Px, Py, Pz, cK, ea, eb, rec);
    count_launches(1);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DFB_OK : set_cuda_error("k_pair_ext launch", e);
}

extern "C" int dfb_grad_supported(int la, int lb, int lc, int b_dummy) { return grad_has(la, lb, lc, b_dummy != 0); }

extern "C" int dfb_grad_contract(const dfb_bra_t* bra, const dfb_groups_t* gr, const dfb_grad_class_t* cls, int ncls,
                                 const double* bar, long sP, long sM, long sN, double* grad, int natm,
                                 void* const* streams, int nstreams) {
    clear_error();
    if (!bra || !gr || (ncls > 0 && !cls) || !bar || !grad || natm < 1 || nstreams < 1 || !streams)
        return set_error(DFB_ERR_INVALID, "invalid arguments to dfb_grad_contract");
    const RysTable* tab = rys_table_of_current_device();
    if (!tab) return set_error(DFB_ERR_NOT_INITIALISED, "Rys table not uploaded on this device");
    GradLaunch L;
    GradArgs& g = L.g;
    g.shA = bra->shA;
    g.shB = bra->shB;
    g.pstart = bra->pstart;
    g.npair_prim = bra->npair;
    g.rec = bra->rec;
    g.cxyz = bra->cxyz;
    g.atom = bra->atom;
    g.aostart = bra->aostart;
    g.b_dummy = bra->b_dummy;
    g.gg = {gr->info, gr->coef, gr->shells, gr->pexp, gr->rexp, gr->cxyz, gr->aostart, gr->atom};
    g.bar = bar;
    g.sP = sP;
    g.sM = sM;
    g.sN = sN;
    g.grad = grad;
    g.natm = natm;
    g.smem_grad = 3L * natm <= 2048;
    g.tab = *tab;
    for (int i = 0; i < ncls; ++i) {
        const dfb_grad_class_t& c = cls[i];
        if (!grad_has(c.la, c.lb, c.lc, bra->b_dummy != 0))
            return set_error(DFB_ERR_UNSUPPORTED, "derivative class (%d,%d,%d) is not supported", c.la, c.lb, c.lc);
        if (c.npair <= 0 || c.nchunk <= 0) continue;
        if (!c.pairs || !c.chunks || c.nq < 1) return set_error(DFB_ERR_INVALID, "derivative class without lists");
        g.pairs = c.pairs;
        g.npair = c.npair;
        g.nchunk = c.nchunk;
        g.chunks = reinterpret_cast<const GradChunk*>(c.chunks);
        g.nq = c.nq;
        g.lc = c.lc;
        g.nr = (c.la + c.lb + c.lc + 1) / 2 + 1;
        L.st = (cudaStream_t)streams[i % nstreams];
        cudaError_t e = kRun[c.la][c.lb](L);
        if (e != cudaSuccess) return set_cuda_error("k_rys_grad launch", e);
        count_launches(1);
    }
    return DFB_OK;
}
