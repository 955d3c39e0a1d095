// FP64 dense kernels: the 3c adjoint of the DF gradient, and the exchange update (k_dsyrk).
//
// The 3c adjoint
//
//   Gamma[P] = Cw A_P Cw^T = U_P Cw^T,    U_P = Cw A_P,   A_P = d_P I - Z_P / 2 (symmetric)
//
// written as (nP, nao, nao).  The inner dimension is only nocc (tens), so the product is
// bound by writing Gamma (8 nP nao^2 bytes) and by the FP64 FMA pipe, not by reading U and Cw.
// Gamma_P is symmetric: one CTA computes one 64 x 64 tile (mt <= nt) of one P, 16 x 16 threads
// with 4 x 4 outputs each, operands staged in shared memory in k chunks of 32; the tile is
// staged in shared memory and written, and for an off-diagonal tile also its transpose, both
// row-contiguous.  In a diagonal tile the upper entries are mirrored onto the
// lower ones, so every Gamma_P is exactly symmetric.  About 0.57 of the full product's FMAs
// for nao = 416 (28 of 49 tiles).
//
// The reference forms this adjoint through its whitened-factor route (df_whiten_adjoint_Qmn,
// asuka/integrals/df_adjoint.py:172-235) with cuBLAS GEMMs; this build's adjoint formulation
// needs Gamma = Cw A_P Cw^T instead.

#include "../../include/dfb.h"
#include "dfb_internal.h"

namespace dfb {
namespace dense {

constexpr int GT = 64;       // tile edge
constexpr int KC = 64;       // k per shared-memory chunk
constexpr int NT = 256;      // threads per CTA (16 x 16)
constexpr int SK = GT + 2;   // row stride of the operand chunks (16-byte aligned rows)
constexpr int SC = GT + 1;   // row stride of the tile stage

// Position of tile column r (= 4 tx + 2 h + q: thread tx's pair h, element q) inside a row of
// the B chunk: the pairs of the 16 column threads are contiguous per h, so the 16-byte loads
// of a warp read 256 contiguous bytes (two wavefronts, no bank conflict).
__device__ __forceinline__ int bpos(int r) { return 32 * ((r >> 1) & 1) + 2 * (r >> 2) + (r & 1); }

__global__ void __launch_bounds__(NT, 3) k_gamma_sym(long nP, int nao, int nocc, const double* __restrict__ U,
                                                  long sUm, long sUp, const double* __restrict__ Cw,
                                                  double* __restrict__ out, int T) {
    extern __shared__ __align__(16) double smem[];  // sA (later the tile stage) | sB
    double* sA = smem;             // sA[c * SK + r] = U[P][mu0 + r][k0 + c]
    double* sB = smem + KC * SK;   // sB[c * SK + bpos(r)] = Cw[nu0 + r][k0 + c]
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    // upper-triangle tile (mt, nt), mt <= nt, of a T x T tile grid
    int idx = blockIdx.x, mt = 0;
    while (idx >= T - mt) {
        idx -= T - mt;
        ++mt;
    }
    const int nt = mt + idx;
    const int mu0 = mt * GT, nu0 = nt * GT;
    // staging: thread covers k column lc = tid % 64 of tile rows lr0 + 4 i (i < 16)
    const int lc = tid & (KC - 1), lr0 = tid / KC;
    // with nocc <= KC the Cw tile is the same for every P of this CTA: staged once
    const bool one_chunk = nocc <= KC;
    if (one_chunk) {
        const bool kin = lc < nocc;
#pragma unroll 4
        for (int i = 0; i < GT / (NT / KC); ++i) {
            const int r = lr0 + (NT / KC) * i;
            sB[lc * SK + bpos(r)] = (kin && nu0 + r < nao) ? Cw[(long)(nu0 + r) * nocc + lc] : 0.0;
        }
    }
    for (long P = blockIdx.y; P < nP; P += gridDim.y) {
        double acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
        const double* Up = U + P * sUp;
        for (int k0 = 0; k0 < nocc; k0 += KC) {
            __syncthreads();  // the previous chunk (or the previous P's tile stage) is consumed
            const bool kin = k0 + lc < nocc;
#pragma unroll 4
            for (int i = 0; i < GT / (NT / KC); ++i) {
                const int r = lr0 + (NT / KC) * i;
                sA[lc * SK + r] = (kin && mu0 + r < nao) ? Up[(long)(mu0 + r) * sUm + k0 + lc] : 0.0;
                if (!one_chunk)
                    sB[lc * SK + bpos(r)] = (kin && nu0 + r < nao) ? Cw[(long)(nu0 + r) * nocc + k0 + lc] : 0.0;
            }
            __syncthreads();
            const double* pa = sA + 4 * ty;
            const double* pb = sB + 2 * tx;
            auto step = [&](int c) {
                const double2 a01 = *reinterpret_cast<const double2*>(pa + c * SK);
                const double2 a23 = *reinterpret_cast<const double2*>(pa + c * SK + 2);
                const double2 b01 = *reinterpret_cast<const double2*>(pb + c * SK);
                const double2 b23 = *reinterpret_cast<const double2*>(pb + c * SK + 32);
                const double a[4] = {a01.x, a01.y, a23.x, a23.y};
                const double b[4] = {b01.x, b01.y, b23.x, b23.y};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
            };
            const int kc = (nocc - k0) < KC ? (nocc - k0) : KC;
#pragma unroll 8
            for (int c = 0; c < kc; ++c) step(c);
        }
        double* outP = out + P * (long)nao * nao;
        // stage the tile in shared memory, then write it and (off the diagonal) its transpose with
        // consecutive threads on consecutive columns: every store instruction fills whole sectors.
        // A diagonal tile writes its upper part (m <= n) and mirrors the strict upper part.
        __syncthreads();  // every thread is done reading sA
        double* sC = smem;  // sC[m * SC + n], over sA (sB stays)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) sC[(4 * ty + i) * SC + 4 * tx + j] = acc[i][j];
        __syncthreads();
        const int wc = tid & (GT - 1), wr0 = tid >> 6;  // column of this thread, first row
        const bool diag = mt == nt;
        if (nu0 + wc < nao) {
#pragma unroll 4
            for (int r = wr0; r < GT; r += NT / GT) {  // tile row r, column wc
                if (mu0 + r < nao && (!diag || r <= wc)) outP[(long)(mu0 + r) * nao + nu0 + wc] = sC[r * SC + wc];
            }
        }
        if (mu0 + wc < nao) {
#pragma unroll 4
            for (int r = wr0; r < GT; r += NT / GT) {  // transposed: output row nu0 + r, column mu0 + wc
                if (nu0 + r < nao && (!diag || wc < r)) outP[(long)(nu0 + r) * nao + mu0 + wc] = sC[wc * SC + r];
            }
        }
    }
}

// Exchange update K += sum_k A(m, k) A(n, k) of the FP64 path, A(m, k) = W[kq * skq + m * sm + k1] with
// k = kq * nk1 + k1 (W[Q, mu, i]: skq = nao nocc, sm = nocc, nk1 = nocc), so W is read in place.
// Only the 64 x 64 tiles on and above the diagonal are formed (0.57 of a full product at nao 416) and k is
// cut into spans over blockIdx.y, so that a few hundred columns still fill the chip.  A launch takes one full
// wave of spans of at most SFL terms (short chains of roundings: relative error 2.3e-16 at k 72960, 8.1e-16 with
// spans of 3300); each block adds its sums to its own tile of `part`, and k_dsyrk_sum adds the spans in their
// order, so K repeats itself bit for bit.  128 threads, 8 x 4 outputs each, k chunks of 16 double-buffered
// through registers, 12 eight-byte shared-memory reads per 32 multiply-adds.  Neither unit is full: FP64 pipe
// 52 %, shared-memory wavefronts 54 %, 0.49 instructions per cycle and scheduler from 12 warps per SM (128
// registers leave four blocks).  nao 416, k 72960: 8.4 G multiply-adds with the padding and
// the whole diagonal tiles in 0.98 ms, 17 of 34 TFLOP/s (spans over all k and atomic sums 1.04; a transposed
// copy and the library's full product 1.4 to 1.5); nao 624, k 164160: 4.46 (4.71); nao 208, k 18240: 0.099 (0.116).
// part = nullptr: the sums go to C by atomic additions (several spans: in any order).
constexpr int ST = 64;        // tile edge
constexpr int SKC = 16;       // k per chunk
constexpr int SNT = 128;      // threads
constexpr int SFL = 512;      // most terms of a span
constexpr int SMIN = 128;     // least terms of a span, which ends in 64 x 64 sums (nao 58, k 2300: 512 50 us, 256 32, 128 24)
constexpr int SP = ST + 1;    // row stride of a chunk: the transposing stores of a half warp hit 16 banks

__global__ void __launch_bounds__(SNT, 4) k_dsyrk(int n, long k_lo, long k_hi, long nk1, const double* __restrict__ W,
                                                  long skq, long sm, double* __restrict__ C, long ldc, long kspan, int T,
                                                  double* __restrict__ part) {
    __shared__ double sA[2][SKC * SP], sB[2][SKC * SP];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    int idx = blockIdx.x, mt = 0;
    while (idx >= T - mt) {
        idx -= T - mt;
        ++mt;
    }
    const int nt = mt + idx, m0 = mt * ST, n0 = nt * ST;
    const bool diag = mt == nt;
    const long kbeg = k_lo + (long)blockIdx.y * kspan, kend = kbeg + kspan < k_hi ? kbeg + kspan : k_hi;
    const int lk = tid & (SKC - 1), lr = tid >> 4;  // this thread loads column lk of rows lr + 8 i
    double va[8], vb[8];
    auto load = [&](long k0) {
        const long k = k0 + lk;
        const bool in = k < kend;
        const long kq = in ? k / nk1 : 0;
        const double* p = W + kq * skq + (in ? k - kq * nk1 : 0);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = lr + 8 * i;
            va[i] = (in && m0 + r < n) ? __ldg(p + (long)(m0 + r) * sm) : 0.0;
            if (!diag) vb[i] = (in && n0 + r < n) ? __ldg(p + (long)(n0 + r) * sm) : 0.0;
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            sA[buf][lk * SP + lr + 8 * i] = va[i];
            if (!diag) sB[buf][lk * SP + lr + 8 * i] = vb[i];
        }
    };
    double acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    load(kbeg);
    store(0);
    __syncthreads();
    int buf = 0;
    for (long k0 = kbeg; k0 < kend; k0 += SKC) {
        const bool more = k0 + SKC < kend;
        if (more) load(k0 + SKC);
        const double* pa = sA[buf] + 8 * ty;
        const double* pb = (diag ? sA[buf] : sB[buf]) + tx;
#pragma unroll
        for (int c = 0; c < SKC; ++c) {
            double a[8], b[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = pa[c * SP + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = pb[c * SP + 16 * j];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        if (more) store(buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
    if (part) {
        double* own = part + ((long)blockIdx.y * gridDim.x + blockIdx.x) * (ST * ST) + tid;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                double* q = own + (i * 4 + j) * SNT;
                *q = k_lo == 0 ? acc[i][j] : *q + acc[i][j];
            }
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + 8 * ty + i;
        if (m >= n) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = n0 + tx + 16 * j;
            if (c >= n || (diag && c < m)) continue;  // a diagonal tile mirrors its upper part
            atomicAdd(C + (long)m * ldc + c, acc[i][j]);
            if (c != m) atomicAdd(C + (long)c * ldc + m, acc[i][j]);
        }
    }
}

// C += the spans of one tile, in their order: thread = element, both orders of an off-diagonal pair.
__global__ void __launch_bounds__(256) k_dsyrk_sum(int n, int ns, const double* __restrict__ part, double* __restrict__ C,
                                                   long ldc, int T) {
    int idx = blockIdx.x, mt = 0;
    while (idx >= T - mt) {
        idx -= T - mt;
        ++mt;
    }
    const int e = blockIdx.y * 256 + threadIdx.x, r = e / SNT, tid = e % SNT;
    const int m = mt * ST + 8 * (tid >> 4) + r / 4, c = (mt + idx) * ST + (tid & 15) + 16 * (r % 4);
    if (m >= n || c >= n || (idx == 0 && c < m)) return;
    const double* p = part + (long)blockIdx.x * (ST * ST) + e;
    double v = 0.0;
#pragma unroll 8
    for (int s = 0; s < ns; ++s) v += p[(long)s * gridDim.x * (ST * ST)];
    C[(long)m * ldc + c] += v;
    if (c != m) C[(long)c * ldc + m] += v;
}

// The launches of an exchange update of n rows: `nslab` slabs of k, each `ns` spans.
struct SyrkPlan {
    int T;
    long ntiles, ns, span, nslab;
};
static SyrkPlan syrk_plan(int n, long K, bool one_launch) {
    SyrkPlan p;
    p.T = (n + ST - 1) / ST;
    p.ntiles = (long)p.T * (p.T + 1) / 2;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long slots = 4L * sms;  // blocks resident at a time
    // full waves: the span count rounded down, over as few waves (up to three) as leave less than a tenth idle
    p.ns = 1;
    double best = 0.0;
    for (int w = 1; w <= 3 && best < 0.9; ++w) {
        const long ns = w * slots / p.ntiles;
        const double use = (double)ns * p.ntiles / ((double)w * slots);
        if (ns >= 1 && use > best + 0.02) {
            best = use;
            p.ns = ns;
        }
    }
    const long most = (K + SMIN - 1) / SMIN;
    if (p.ns > most) p.ns = most;
    p.nslab = one_launch ? 1 : (K + p.ns * SFL - 1) / (p.ns * SFL);
    p.span = (K + p.nslab * p.ns - 1) / (p.nslab * p.ns);
    p.span = (p.span + SKC - 1) / SKC * SKC;
    if (p.nslab == 1) p.ns = (K + p.span - 1) / p.span;
    return p;
}

// Inverses of the nb x nb diagonal blocks of a lower-triangular L by forward substitution.  A CTA takes 32
// columns of one block (lane = column) and walks its rows in panels of 16, the next panel of L read ahead
// through registers: each warp forms the dot products of two rows with the solved ones, then one warp solves
// the panel's triangle.  Bound by the chain of panels, not by the number of blocks, and one launch where
// batched library solves and products of growing blocks took twenty (eight 256-row blocks: 0.125 against
// 0.27 ms; row by row, with a global load in every row's chain, 0.27 ms).
constexpr int IC = 32, IW = 8, INB = 256, IP = 16;

__global__ void __launch_bounds__(32 * IW) k_tri_inv(int n, int nb, const double* __restrict__ L, long ldl,
                                                     double* __restrict__ out) {
    extern __shared__ double sm[];
    double* x = sm;                       // [nb][32] solved rows
    double* S = x + (long)nb * IC;        // [IP][32]
    double* pan = S + IP * IC;            // [2][IP][nb]: rows of the panel, columns from j0
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int r0 = blockIdx.y * nb, m = n - r0 < nb ? n - r0 : nb;  // rows of this block
    const int j0 = blockIdx.x * IC, col = j0 + lane;
    const double* Lb = L + (long)r0 * ldl + r0;
    double* O = out + (long)blockIdx.y * nb * nb;
    if (j0 >= m) return;
    for (int i = w; i < j0; i += IW) O[(long)i * nb + col] = 0.0;  // above the diagonal (col < nb)
    double pre[IP];  // this thread's column j0 + tid of the next panel's rows
    auto fetch = [&](int p0) {
#pragma unroll
        for (int r = 0; r < IP; ++r) {
            const int i = p0 + r, k = j0 + tid;
            pre[r] = (i < m && k <= i) ? __ldg(Lb + (long)i * ldl + k) : 0.0;
        }
    };
    auto put = [&](int buf) {
        if (tid < nb - j0) {
#pragma unroll
            for (int r = 0; r < IP; ++r) pan[(buf * IP + r) * nb + tid] = pre[r];
        }
    };
    fetch(j0);
    put(0);
    __syncthreads();
    int buf = 0;
    for (int p0 = j0; p0 < m; p0 += IP, buf ^= 1) {
        const bool more = p0 + IP < m;
        if (more) fetch(p0 + IP);
        const double* P = pan + buf * IP * nb;
#pragma unroll
        for (int h = 0; h < IP / IW; ++h) {
            const double* row = P + (w + h * IW) * nb;
            double s[4] = {0.0, 0.0, 0.0, 0.0};
            for (int k = 0; k < p0 - j0; k += 4) {  // p0 - j0 is a multiple of IP
#pragma unroll
                for (int q = 0; q < 4; ++q) s[q] = fma(row[k + q], x[(j0 + k + q) * IC + lane], s[q]);
            }
            S[(w + h * IW) * IC + lane] = (s[0] + s[1]) + (s[2] + s[3]);
        }
        __syncthreads();
        if (w == 0) {
            double xr[IP];
#pragma unroll
            for (int r = 0; r < IP; ++r) {
                const int i = p0 + r;
                double t = (col == i ? 1.0 : 0.0) - S[r * IC + lane];
#pragma unroll
                for (int q = 0; q < IP; ++q)
                    if (q < r) t = fma(-P[r * nb + p0 - j0 + q], xr[q], t);
                const double d = P[r * nb + p0 - j0 + r];
                xr[r] = (i < m && col <= i) ? t / d : 0.0;
                if (i < m) {
                    x[i * IC + lane] = xr[r];
                    if (col < m) O[(long)i * nb + col] = xr[r];
                }
            }
        }
        if (more) put(buf ^ 1);
        __syncthreads();
    }
}

}  // namespace dense
}  // namespace dfb

using namespace dfb;

extern "C" int dfb_gamma_sym(long nP, int nao, int nocc, const double* U, long sU_mu, long sU_P, const double* Cw,
                             double* out, void* stream) {
    clear_error();
    if (nP < 0 || nao < 0 || nocc < 0)
        return set_error(DFB_ERR_INVALID, "invalid sizes to dfb_gamma_sym (nP %ld, nao %d, nocc %d)", nP, nao, nocc);
    if (nP == 0 || nao == 0) return DFB_OK;
    if (nocc == 0) return set_error(DFB_ERR_INVALID, "nocc == 0: Gamma is zero (clear it instead)");
    if (!U || !Cw || !out || sU_mu < nocc || sU_P < 0)
        return set_error(DFB_ERR_INVALID, "invalid pointers or strides to dfb_gamma_sym");
    const int T = (nao + dense::GT - 1) / dense::GT;
    const long ntiles = (long)T * (T + 1) / 2;
    if (ntiles > 0x7fffffffL) return set_error(DFB_ERR_UNSUPPORTED, "nao %d too large", nao);
    // four P per CTA: the Cw tile is staged once per CTA, and many short CTAs keep the last wave small
    long gy = (nP + 3) / 4;
    if (gy > 65535) gy = 65535;
    if (gy < 1) gy = 1;
    const size_t smem = sizeof(double) * 2 * dense::KC * dense::SK;
    cudaError_t e = cudaFuncSetAttribute(dense::k_gamma_sym, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return set_cuda_error("cudaFuncSetAttribute(k_gamma_sym)", e);
    dense::k_gamma_sym<<<dim3((unsigned)ntiles, (unsigned)gy), dense::NT, smem, (cudaStream_t)stream>>>(
        nP, nao, nocc, U, sU_mu, sU_P, Cw, out, T);
    count_launches(1);
    e = cudaGetLastError();
    if (e != cudaSuccess) return set_cuda_error("k_gamma_sym launch", e);
    return DFB_OK;
}

extern "C" long dfb_dsyrk_scratch(int n, long nkq, long nk1) {
    if (n <= 0 || nkq <= 0 || nk1 <= 0) return 0;
    const dense::SyrkPlan p = dense::syrk_plan(n, nkq * nk1, false);
    return p.ns * p.nslab > 1 ? p.ns * p.ntiles * dense::ST * dense::ST : 0;
}

extern "C" int dfb_dsyrk_ws(int n, long nkq, long nk1, const double* W, long skq, long sm, double* C, long ldc,
                            double* ws, long ws_doubles, void* stream) {
    clear_error();
    if (n < 0 || nkq < 0 || nk1 < 0 || ldc < n)
        return set_error(DFB_ERR_INVALID, "invalid sizes to dfb_dsyrk (n %d, k %ld x %ld)", n, nkq, nk1);
    const long K = nkq * nk1;
    if (n == 0 || K == 0) return DFB_OK;
    if (!W || !C) return set_error(DFB_ERR_INVALID, "invalid pointers to dfb_dsyrk");
    const dense::SyrkPlan p = dense::syrk_plan(n, K, !ws);
    if (p.ntiles > 0x7fffffffL) return set_error(DFB_ERR_UNSUPPORTED, "n %d too large", n);
    if (p.ns * p.nslab == 1) ws = nullptr;  // one span: no sums to add
    if (ws && ws_doubles < p.ns * p.ntiles * dense::ST * dense::ST)
        return set_error(DFB_ERR_INVALID, "dfb_dsyrk needs %ld scratch doubles, %ld given",
                         p.ns * p.ntiles * dense::ST * dense::ST, ws_doubles);
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaSuccess;
    const long slab = p.ns * p.span;
    for (long k0 = 0; k0 < K && e == cudaSuccess; k0 += slab) {
        // the last slab may leave spans without terms: they keep what their tiles of ws hold
        const long k1 = k0 + slab < K ? k0 + slab : K, ny = (k1 - k0 + p.span - 1) / p.span;
        dense::k_dsyrk<<<dim3((unsigned)p.ntiles, (unsigned)ny), dense::SNT, 0, st>>>(n, k0, k1, nk1, W, skq, sm, C, ldc,
                                                                                      p.span, p.T, ws);
        count_launches(1);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return set_cuda_error("k_dsyrk launch", e);
    if (ws) {
        dense::k_dsyrk_sum<<<dim3((unsigned)p.ntiles, dense::ST * dense::ST / 256), 256, 0, st>>>(n, (int)p.ns, ws, C, ldc,
                                                                                                 p.T);
        count_launches(1);
        e = cudaGetLastError();
        if (e != cudaSuccess) return set_cuda_error("k_dsyrk_sum launch", e);
    }
    return DFB_OK;
}

extern "C" int dfb_dsyrk(int n, long nkq, long nk1, const double* W, long skq, long sm, double* C, long ldc, void* stream) {
    return dfb_dsyrk_ws(n, nkq, nk1, W, skq, sm, C, ldc, nullptr, 0, stream);
}

extern "C" int dfb_tri_inv(int n, int nb, const double* L, long ldl, double* out, void* stream) {
    clear_error();
    if (n < 0 || nb < 32 || nb > dense::INB || nb % 32 || ldl < n)
        return set_error(DFB_ERR_INVALID, "invalid sizes to dfb_tri_inv (n %d, nb %d)", n, nb);
    if (n == 0) return DFB_OK;
    if (!L || !out) return set_error(DFB_ERR_INVALID, "invalid pointers to dfb_tri_inv");
    const int nblk = (n + nb - 1) / nb;
    const size_t sm = sizeof(double) * ((size_t)nb * dense::IC + dense::IP * dense::IC + 2 * dense::IP * nb);
    cudaError_t e = cudaFuncSetAttribute(dense::k_tri_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return set_cuda_error("cudaFuncSetAttribute(k_tri_inv)", e);
    dense::k_tri_inv<<<dim3(nb / dense::IC, nblk), 32 * dense::IW, sm, (cudaStream_t)stream>>>(n, nb, L, ldl, out);
    count_launches(1);
    e = cudaGetLastError();
    return e == cudaSuccess ? DFB_OK : set_cuda_error("k_tri_inv launch", e);
}
