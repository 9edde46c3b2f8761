// fdtd_kernels.cu -- the small sm_100a kernels of one GSvit FDTD time step: the
// 1D TSF grid (aux_step, 1 CTA), the TSF face corrections, the NFFF running DFT
// and the far-field integration.  The field updates are in fdtd_bulk.cu (TMA
// tiles) and fdtd_flat.cu.  The *_batch forms take device tables of per-plan
// parameters and serve many plans in one launch.
#include <cuda_runtime.h>

#include "../../include/gsvit_b200.h"
#include "fdtd_device.cuh"
#include "fdtd_kernels.cuh"

namespace {

// ------------------------------------------------------------ TSF face tables

// This step's TSF corrections for every face cell (source.c:547-771 and
// 1476-1672): the 1D grid value at corr*dcomp(cell) by the cubic
// interpolation of dline.c:89-111 (FP64), projected by gex..ghz, scaled by
// dt/(dx mu0) for H or (dt/dx)/epsilon(cell) for E, gated by TSF_SKIP, the
// source-skip map and (k0 face) the PEC test.  Runs after aux_step.
template <class R>
__device__ __forceinline__ void tsf_face_cell(const DevPlan &P, int t)
{
    using V2 = typename Tab<R>::V2;
    const int i0 = P.t0[0], j0 = P.t0[1], k0 = P.t0[2], in = P.t1[0], jn = P.t1[1], kn = P.t1[2];
    const int ni = in - i0 + 1, nj = jn - j0 + 1, nk = kn - k0 + 1;
    const int sz[3] = {nj * nk, ni * nk, ni * nj};
    if (!P.tsf_on || t >= 2 * (sz[0] + sz[1] + sz[2])) return;
    int f = 0, off = t;
    while (f < 6 && off >= sz[f / 2]) { off -= sz[f / 2]; f++; }
    if (f >= 6) return;
    const int a = off / P.tnb[f], b = off % P.tnb[f];
    const uint8_t fl = P.tmap[f][off];
    const double hc = P.hcor;
    V2 dh{0, 0}, de{0, 0};
    const float4 *cls4 = reinterpret_cast<const float4 *>(P.classes);
    if (fl & 1) {
        int ei, ej, ek;   // E cell; dH / dE are the dcomp positions of the H and E corrections
        double dH, dE;
        if (f < 2) {
            const int j = j0 + a, k = k0 + b;
            if (f == 0) { ei = i0; dH = tsf_dcomp(P, i0, j, k); dE = tsf_dcomp(P, i0 - 1, j, k); }
            else { ei = in; dH = tsf_dcomp(P, in, j, k); dE = dH; }
            ej = j; ek = k;
        } else if (f < 4) {
            const int i = i0 + a, k = k0 + b;
            if (f == 2) { ej = j0; dH = tsf_dcomp(P, i, j0, k); dE = tsf_dcomp(P, i, j0 - 1, k); }
            else { ej = jn; dH = tsf_dcomp(P, i, jn, k); dE = dH; }
            ei = i; ek = k;
        } else {
            const int i = i0 + a, j = j0 + b;
            if (f == 4) { ek = k0; dH = tsf_dcomp(P, i, j, k0); dE = tsf_dcomp(P, i, j, k0 - 1); }
            else { ek = kn; dH = tsf_dcomp(P, i, j, kn); dE = dH; }
            ei = i; ej = j;
        }
        const double ve = tsf_dval(P.aux_e, P.jres, dH);
        const double vh = tsf_dval(P.aux_h, P.jres, dE);
        const double ce = (double)Tab<R>::tsfe(P, cls4, cls_at(P, ei, ej, ek));
        const bool pec = (fl & 2) != 0;
        switch (f) {
        case 0:
            if (ek < kn) dh.x = -(R)(hc * (ve * P.gez));
            if (ej < jn) dh.y = (R)(hc * (ve * P.gey));
            if (ej < jn) de.x = (R)(ce * (vh * P.ghz));
            if (ek < kn) de.y = -(R)(ce * (vh * P.ghy));
            break;
        case 1:
            if (ek < kn) dh.x = (R)(hc * (ve * P.gez));
            if (ej < jn) dh.y = -(R)(hc * (ve * P.gey));
            if (ej < jn) de.x = -(R)(ce * (vh * P.ghz));
            if (ek < kn) de.y = (R)(ce * (vh * P.ghy));
            break;
        case 2:
            if (ek < kn) dh.x = (R)(hc * (ve * P.gez));
            if (ei < in) dh.y = -(R)(hc * (ve * P.gex));
            if (ei < in) de.x = -(R)(ce * (vh * P.ghz));
            if (ek < kn) de.y = (R)(ce * (vh * P.ghx));
            break;
        case 3:
            if (ek < kn) dh.x = -(R)(hc * (ve * P.gez));
            if (ei < in) dh.y = (R)(hc * (ve * P.gex));
            if (ei < in) de.x = (R)(ce * (vh * P.ghz));
            if (ek < kn) de.y = -(R)(ce * (vh * P.ghx));
            break;
        case 4:
            if (ej < jn && !pec) dh.x = -(R)(hc * (ve * P.gey));
            if (ei < in && !pec) dh.y = (R)(hc * (ve * P.gex));
            if (ei < in && !pec) de.x = (R)(ce * (vh * P.ghy));
            if (ej < jn && !pec) de.y = -(R)(ce * (vh * P.ghx));
            break;
        default:
            if (ej < jn) dh.x = (R)(hc * (ve * P.gey));
            if (ei < in) dh.y = -(R)(hc * (ve * P.gex));
            if (ei < in) de.x = -(R)(ce * (vh * P.ghy));
            if (ej < jn) de.y = (R)(ce * (vh * P.ghx));
            break;
        }
    }
    reinterpret_cast<V2 *>(P.tcor_h[f])[off] = dh;
    reinterpret_cast<V2 *>(P.tcor_e[f])[off] = de;
    (void)a; (void)b;
}

__global__ void tsf_face_kernel(const __grid_constant__ DevPlan P, int total)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < total) {
        if (P.real64) tsf_face_cell<double>(P, t);
        else tsf_face_cell<float>(P, t);
    }
}

__global__ void tsf_face_batch(const DevPlan *plans)
{
    tsf_face_cell<float>(plans[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x);
}

// ------------------------------------------------------------ 1D aux grid

// 1D TSF grid step of source.c:1469-1473 over 1dpool.c:84-162, in FP64 with
// the reference's operation order (no contraction); also records the probes
// of the previous step (output.c:341-352).
__device__ __forceinline__ void aux_line(const DevAux &A, int s)
{
    if (A.res <= 0) return;
    const int tid = threadIdx.x, nt = blockDim.x;
    double *e = A.e, *h = A.h;
    const int r = A.res;
    for (int i = 1 + tid; i < r; i += nt)               // sv_1dpool_ystep_e
        e[i] = __dadd_rn(e[i], __dmul_rn(A.ce, __dadd_rn(h[i - 1], -h[i])));
    __syncthreads();
    if (tid == 0) {
        double *b = A.bnd;
        e[0] = __dadd_rn(b[1], __dmul_rn(A.lc, __dadd_rn(e[1], -b[0])));          // sv_1dpool_boundary
        h[0] = __dadd_rn(b[3], __dmul_rn(A.lc, __dadd_rn(h[1], -b[2])));
        e[r - 1] = __dadd_rn(b[5], __dmul_rn(A.lc, __dadd_rn(e[r - 2], -b[4])));
        h[r - 1] = __dadd_rn(b[7], __dmul_rn(A.lc, __dadd_rn(h[r - 2], -b[6])));
        b[0] = e[0]; b[1] = e[1]; b[2] = h[0]; b[3] = h[1];                          // _boundary_copy
        b[4] = e[r - 1]; b[5] = e[r - 2]; b[6] = h[r - 1]; b[7] = h[r - 2];
        e[0] = (s < A.nwave) ? A.wave[s] : 0.0;                                        // _apply_source
    }
    __syncthreads();
    for (int i = tid; i < r - 1; i += nt)               // sv_1dpool_ystep_h
        h[i] = __dadd_rn(h[i], __dmul_rn(A.chh, __dadd_rn(e[i], -e[i + 1])));
}

// the probes of step s, whose fields are behind `fields`
__device__ __forceinline__ void probe_row(const DevAux &A, const float *const *fields, int s)
{
    if (s < 0 || s >= A.nsteps_planned) return;
    for (int q = threadIdx.x; q < A.nprobes * 6; q += blockDim.x) {
        const int p = q / 6, comp = q % 6;
        A.probe_out[((size_t)p * A.nsteps_planned + s) * 6 + comp] = ld_any(fields[comp], A.probe_cells[p], A.storage) * (comp >= 3 ? (double)A.ihs : 1.0);
    }
}

// does an array of FP32 (FP64) values hold one that is neither +0 nor -0?
__global__ void any_nonzero_kernel(const uint32_t *p, int64_t words, int real64, int *flag)
{
    bool any = false;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < words; q += (int64_t)gridDim.x * blockDim.x)
        any = any || (p[q] & (real64 && !(q & 1) ? 0xffffffffu : 0x7fffffffu));
    if (any) *flag = 1;
}

__global__ void aux_line_kernel(const DevAux A)
{
    const int s = *A.step + A.off;
    if (A.off != 1) probe_row(A, A.fields, s - (A.off ? 2 : 1));
    aux_line(A, s);
}

__global__ void close_steps_kernel(const DevAux A, const float *const *before)
{
    const int s = *A.step + A.off;   // steps done after this call
    if (before && A.off >= 2) probe_row(A, before, s - 2);
    probe_row(A, A.fields, s - 1);
    __syncthreads();
    if (threadIdx.x == 0) *A.step = s;
}

// batches: the probes of the previous step, the 1D grid, the step counter
__global__ void aux_step_batch(const DevAux *Aux)
{
    const DevAux &A = Aux[blockIdx.x];
    const int s = *A.step;
    probe_row(A, A.fields, s - 1);
    aux_line(A, s);
    __syncthreads();
    if (threadIdx.x == 0) *A.step = s + 1;
}

// the probes of the last completed step
__global__ void probe_capture_kernel(const DevAux A) { probe_row(A, A.fields, *A.step - 1); }

// ------------------------------------------------------------ NFFF running DFT

// Per surface cell s and frequency f:  Ehat += E(step) w,  Dhat += dE/dn(step) w,
// w = exp(-i omega step dt).  FP64 accumulators.  Each step stores the nine
// raw E samples of the cell (E, E(c+st), E(c-st) per component) in ring slot
// step % NFFF_RING; the step that fills the last slot folds the block into the
// accumulators in step order, with the arithmetic of a per-step update, so the
// sums are those of accumulating every step (the accumulators are read and
// written once per NFFF_RING steps instead of every step).
constexpr int NFFF_TW_MAXF = 16;   // frequencies whose twiddles a CTA tabulates in shared memory

// exp(-i omega_f (first_step + j) dt) of the block's steps, computed once per
// CTA: tw[f * nslots + j] = (cos, sin).  All threads of the CTA take part.
__device__ __forceinline__ void nfff_twiddles(const DevNfff &N, int first_step, int nslots, double2 *tw)
{
    for (int t = threadIdx.x; t < nslots * N.nfreq; t += blockDim.x) {
        double sn, cs;
        sincos(N.omega_dt[t / nslots] * (double)(first_step + t % nslots), &sn, &cs);
        tw[t] = make_double2(cs, sn);
    }
    __syncthreads();
}

// tw: the CTA's twiddle table, or nullptr to evaluate them per cell.  S: the
// element type of the sample ring (FP32; FP64 for FP64-storage plans)
// STAGE (FP32 samples only): the cell's ring (8 x 9 values) is read once into
// registers instead of once per frequency (the ring is far larger than L2),
// at 144 registers a thread; the same arithmetic in the same order.
template <class S, bool STAGE = false>
__device__ __forceinline__ void nfff_fold(const DevNfff &N, int s, int first_step, int nslots, bool clear, const double2 *tw)
{
    const size_t ns = (size_t)N.ns;
    S *ring = reinterpret_cast<S *>(N.ring);
    if constexpr (STAGE && sizeof(S) == 4) {
        float rv[NFFF_RING][9];
#pragma unroll
        for (int j = 0; j < NFFF_RING; j++)
#pragma unroll
            for (int q = 0; q < 9; q++) rv[j][q] = j < nslots ? ring[((size_t)j * 9 + q) * ns + s] : 0.f;
        for (int f = 0; f < N.nfreq; f++) {
            double2 A[6];
            for (int q = 0; q < 6; q++) A[q] = N.acc[((size_t)f * 6 + q) * ns + s];
#pragma unroll
            for (int j = 0; j < NFFF_RING; j++) {
                if (j >= nslots) break;
                double v[6];
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    v[a] = (double)rv[j][3 * a];
                    v[3 + a] = ((double)rv[j][3 * a + 1] - (double)rv[j][3 * a + 2]) * N.inv2dx;
                }
                double sn, cs;
                if (tw) { cs = tw[f * nslots + j].x; sn = tw[f * nslots + j].y; }
                else sincos(N.omega_dt[f] * (double)(first_step + j), &sn, &cs);
#pragma unroll
                for (int q = 0; q < 6; q++) {
                    A[q].x += v[q] * cs;
                    A[q].y -= v[q] * sn;
                }
            }
            for (int q = 0; q < 6; q++) N.acc[((size_t)f * 6 + q) * ns + s] = A[q];
        }
        if (clear)
            for (int j = 0; j < nslots; j++)
                for (int q = 0; q < 9; q++) ring[((size_t)j * 9 + q) * ns + s] = 0;
        return;
    }
    for (int f = 0; f < N.nfreq; f++) {
        double2 A[6];
        for (int q = 0; q < 6; q++) A[q] = N.acc[((size_t)f * 6 + q) * ns + s];
        for (int j = 0; j < nslots; j++) {
            const S *r = ring + (size_t)j * 9 * ns + s;
            double v[6];
            for (int a = 0; a < 3; a++) {
                v[a] = (double)r[(3 * a) * ns];
                v[3 + a] = ((double)r[(3 * a + 1) * ns] - (double)r[(3 * a + 2) * ns]) * N.inv2dx;
            }
            double sn, cs;
            if (tw) { cs = tw[f * nslots + j].x; sn = tw[f * nslots + j].y; }
            else sincos(N.omega_dt[f] * (double)(first_step + j), &sn, &cs);
            for (int q = 0; q < 6; q++) {
                A[q].x += v[q] * cs;
                A[q].y -= v[q] * sn;
            }
        }
        for (int q = 0; q < 6; q++) N.acc[((size_t)f * 6 + q) * ns + s] = A[q];
    }
    if (clear)
        for (int j = 0; j < nslots; j++)
            for (int q = 0; q < 9; q++) ring[((size_t)j * 9 + q) * ns + s] = 0;
}

// the steps since the last full block (device step counter % NFFF_RING); their
// slots are cleared, so the fold at the end of the block adds zeros for them
__global__ void nfff_fold_pending_kernel(const DevNfff N)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (N.ns <= 0 || N.nfreq <= 0) return;
    const int done = *N.step;
    const int pending = done % NFFF_RING;
    if (pending == 0) return;
    __shared__ double2 tw[NFFF_RING * NFFF_TW_MAXF];
    const bool table = N.nfreq <= NFFF_TW_MAXF;
    if (table) nfff_twiddles(N, done - pending, pending, tw);
    if (s < N.ns) {
        if (N.storage == FDTD_STORE_F64) nfff_fold<double>(N, s, done - pending, pending, true, table ? tw : nullptr);
        else nfff_fold<float>(N, s, done - pending, pending, true, table ? tw : nullptr);
    }
}

// The NFFF step in two launches (single plans and batches): the sampling, which every step
// does, in a light kernel (few registers, full occupancy: its nine gathered
// loads a cell want many in flight), and the fold, which only the step that
// fills the ring does, in a kernel that every other step leaves at once.
// Both launch every step, so a captured graph is right at any step offset.
template <class S>
__device__ __forceinline__ void nfff_sample_cell(const DevNfff &N, int s)
{
    if (N.ns <= 0 || N.nfreq <= 0 || s >= N.ns) return;
    const int step = *N.step + N.off;
    if (step < 0) return;
    const size_t ns = (size_t)N.ns;
    const int64_t c = N.cell[s];
    const int64_t st = N.nstride[s];
    S *r = reinterpret_cast<S *>(N.ring) + (size_t)(step % NFFF_RING) * 9 * ns + s;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float *E = N.e[a];
        r[(3 * a) * ns] = (S)ld_any(E, c, N.storage);
        r[(3 * a + 1) * ns] = (S)ld_any(E, c + st, N.storage);
        r[(3 * a + 2) * ns] = (S)ld_any(E, c - st, N.storage);
    }
}

__global__ void nfff_sample_kernel(const DevNfff N)
{
    if (N.storage == FDTD_STORE_F64) nfff_sample_cell<double>(N, blockIdx.x * blockDim.x + threadIdx.x);
    else nfff_sample_cell<float>(N, blockIdx.x * blockDim.x + threadIdx.x);
}

// the step counter is the same for every thread of the launch: a CTA either
// leaves at once or reaches the twiddle table's barrier with all its threads
template <class S>
__device__ __forceinline__ void nfff_fold_full_ring(const DevNfff &N, int s)
{
    if (N.ns <= 0 || N.nfreq <= 0) return;
    const int step = *N.step + N.off;
    if (step < 0 || step % NFFF_RING != NFFF_RING - 1) return;
    __shared__ double2 tw[NFFF_RING * NFFF_TW_MAXF];
    const bool table = N.nfreq <= NFFF_TW_MAXF;
    if (table) nfff_twiddles(N, step - (NFFF_RING - 1), NFFF_RING, tw);
    if (s < N.ns) nfff_fold<S, true>(N, s, step - (NFFF_RING - 1), NFFF_RING, false, table ? tw : nullptr);
}

__global__ void __launch_bounds__(128, 3) nfff_fold_kernel(const DevNfff N)
{
    if (N.storage == FDTD_STORE_F64) nfff_fold_full_ring<double>(N, blockIdx.x * blockDim.x + threadIdx.x);
    else nfff_fold_full_ring<float>(N, blockIdx.x * blockDim.x + threadIdx.x);
}

// batches: one plan per CTA row (blockIdx.y), so the step counter and the fold
// decision are the same for every thread of a CTA
__global__ void nfff_sample_batch(const DevNfff *N)
{
    nfff_sample_cell<float>(N[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x);
}

__global__ void __launch_bounds__(128, 3) nfff_fold_batch(const DevNfff *N)
{
    nfff_fold_full_ring<float>(N[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x);
}

// ------------------------------------------------------------ far-field integration

// F_hat_n(omega) = sum_s A_s exp(-i omega (R_ns - istart_n) dt) *
//   [(-c' + b e^{i omega dt} + c' e^{2 i omega dt}) Ehat_s + sgn_f a e^{i omega dt} Dhat_s]
// with r, cos(theta), a, b, c and the retarded index R = (int)(1 + r/(c dt)) of
// farfield.c:175-405: the DFT of the reference time-domain series.
//
// Tiled over (far points x surface-cell groups): a CTA owns 128 * FF_PTS far
// points and one group of surface cells, staged 32 at a time in shared memory
// with their accumulators for NF frequencies.  exp(-i omega R dt) = w comes from
// a table over R; exp(+i omega istart dt), the face area and the sum over groups
// are applied by farfield_reduce_kernel.  FP64 throughout.
//
// With z = exp(i omega dt), z^2 - 1 = 2 i sin(omega dt) z and q = 1/r a pair adds
//   w q cos(theta) (q + i kappa) * (-z Ehat / 4 pi)  +  w q * (sgn z Dhat / 4 pi),
// kappa = sin(omega dt) / (c dt): the factors of a cell alone are formed when it
// is staged, and the reference's square root and division run only for pairs
// whose retarded index they could decide.  What bounds it is FP64 arithmetic (its
// pipe 67 % busy, at 11 warps an SM that wait for its latency); each read of a
// staged cell serves the thread's FF_PTS points (192^3, 4186 points, 3 frequencies: 13.9 ms with the factors formed
// pair by pair, 11.7 with three staged terms and a point a thread, 7.0 now).
constexpr int FF_PTS = FF_TILE / 128;

template <int NF>
__global__ void __launch_bounds__(128) farfield_partial_kernel(const DevFarfield F, int f0)
{
    constexpr int CH = 32;
    __shared__ double2 sacc[CH][NF][6];   // per staged cell, frequency and component: -z Ehat / 4 pi, sgn z Dhat / 4 pi
    __shared__ double sgeo[CH][6];        // cell, outward normal
    const int per = (F.ns + F.groups - 1) / F.groups;
    const int s0 = blockIdx.y * per, s1 = min(F.ns, s0 + per);
    const double C0 = 299792458.0, PI = 3.14159265358979323846;
    const double dt = F.dt, dx = F.dx, c0dt = C0 * dt, cells = dx / c0dt;
    const double idx = 1.0 / dx, k4 = 1.0 / (4.0 * PI);
    int pt[FF_PTS];
    double x[FF_PTS], y[FF_PTS], z[FF_PTS], acc[FF_PTS][NF][3][2], kappa[NF];
#pragma unroll
    for (int u = 0; u < FF_PTS; u++) {
        pt[u] = (blockIdx.x * FF_PTS + u) * blockDim.x + threadIdx.x;
        const int p = min(pt[u], F.npoints - 1);   // past the end: the last point again, not stored
        x[u] = F.points[3 * p]; y[u] = F.points[3 * p + 1]; z[u] = F.points[3 * p + 2];
#pragma unroll
        for (int f = 0; f < NF; f++)
#pragma unroll
            for (int q = 0; q < 3; q++) acc[u][f][q][0] = acc[u][f][q][1] = 0.0;
    }
#pragma unroll
    for (int f = 0; f < NF; f++) kappa[f] = sin(F.omega[f0 + f] * dt) / c0dt;
    for (int base = s0; base < s1; base += CH) {
        const int n = min(CH, s1 - base);
        __syncthreads();
        for (int q = threadIdx.x; q < n; q += blockDim.x) {
            const int fc = F.face[base + q];
            for (int a = 0; a < 3; a++) {
                sgeo[q][a] = F.cell_ijk[3 * (base + q) + a];
                sgeo[q][3 + a] = fc / 2 == a ? ((fc & 1) ? 1.0 : -1.0) : 0.0;   // angle(): normal of the face (farfield.c:44-54)
            }
        }
        for (int t = threadIdx.x; t < n * NF * 3; t += blockDim.x) {
            const int q = t % n, fc = t / n, f = fc / 3, c = fc % 3;
            const double2 *A = F.acc + ((size_t)(f0 + f) * 6 + c) * F.ns + base + q;
            const double2 E = A[0], D = A[(size_t)3 * F.ns];
            double zs, zc;
            sincos(F.omega[f0 + f] * dt, &zs, &zc);
            const double kd = (F.face[base + q] & 1) ? k4 : -k4;
            sacc[q][f][c] = make_double2(-k4 * (zc * E.x - zs * E.y), -k4 * (zc * E.y + zs * E.x));
            sacc[q][f][3 + c] = make_double2(kd * (zc * D.x - zs * D.y), kd * (zc * D.y + zs * D.x));
        }
        __syncthreads();
        for (int q = 0; q < n; q++) {
            double ir[FF_PTS], ct[FF_PTS];
            int R[FF_PTS];
#pragma unroll
            for (int u = 0; u < FF_PTS; u++) {
                const double rx = x[u] - sgeo[q][0], ry = y[u] - sgeo[q][1], rz = z[u] - sgeo[q][2];
                const double d2 = rx * rx + ry * ry + rz * rz;
                const double dot = sgeo[q][3] * rx + sgeo[q][4] * ry + sgeo[q][5] * rz;
                // The retarded index needs the reference's square root and division
                // only where they could round across an integer (and in the
                // surface cell itself, where rt is no number).
                const double irc = rsqrt(d2);
                const double rt = 1.0 + d2 * irc * cells;
                R[u] = (int)rt;
                const double fr = rt - R[u], tol = rt * 8e-15;
                if (!(fr >= tol && fr <= 1.0 - tol)) R[u] = (int)(1.0 + sqrt(d2) * dx / c0dt);
                R[u] = min(R[u], F.ntw - 1);
                ct[u] = dot * irc;
                ir[u] = irc * idx;
            }
#pragma unroll
            for (int f = 0; f < NF; f++) {
                double wr[FF_PTS], wi[FF_PTS], gr[FF_PTS], gi[FF_PTS];
#pragma unroll
                for (int u = 0; u < FF_PTS; u++) {
                    const double2 w = __ldg(&F.tw[(size_t)(f0 + f) * F.ntw + R[u]]);
                    wr[u] = w.x * ir[u];
                    wi[u] = w.y * ir[u];
                    const double br = ct[u] * ir[u], bi = ct[u] * kappa[f];
                    gr[u] = wr[u] * br - wi[u] * bi;
                    gi[u] = wr[u] * bi + wi[u] * br;
                }
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const double2 e = sacc[q][f][c], d = sacc[q][f][3 + c];
#pragma unroll
                    for (int u = 0; u < FF_PTS; u++) {
                        acc[u][f][c][0] += gr[u] * e.x - gi[u] * e.y + wr[u] * d.x - wi[u] * d.y;
                        acc[u][f][c][1] += gr[u] * e.y + gi[u] * e.x + wr[u] * d.y + wi[u] * d.x;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int u = 0; u < FF_PTS; u++) {
        if (pt[u] >= F.npoints) continue;
        for (int f = 0; f < NF; f++)
            for (int c = 0; c < 3; c++)
                F.part[(((size_t)blockIdx.y * F.npoints + pt[u]) * F.nfreq + f0 + f) * 3 + c] = make_double2(acc[u][f][c][0], acc[u][f][c][1]);
    }
}

// out = area * exp(+i omega istart dt) * sum over groups (fixed order)
__global__ void farfield_reduce_kernel(const DevFarfield F)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= F.npoints * F.nfreq * 3) return;
    const int p = t / (F.nfreq * 3), f = (t / 3) % F.nfreq;
    double re = 0, im = 0;
    for (int g = 0; g < F.groups; g++) {
        const double2 v = F.part[(size_t)g * F.npoints * F.nfreq * 3 + t];
        re += v.x;
        im += v.y;
    }
    double sn, cs;
    sincos(F.omega[f] * (double)F.istart[p] * F.dt, &sn, &cs);
    const double area = F.dx * F.dx;
    F.out[t] = make_double2(area * (cs * re - sn * im), area * (cs * im + sn * re));
}

// The reference's far-field series, farfield.c:207-404, for every (surface
// cell, far point): r and cos(theta) as dist()/angle() (farfield.c:33-56),
// nn = (int)(step + 1 + r/(c dt)) - istart with the reference's operation
// order (the sum can round across an integer, so nn is formed exactly as
// there), three taps per component when 3 <= nn < ndata.  Neighbouring cells
// reach a point at about the same time, so a CTA sums its SERIES_CELLS cells
// in a window of the series in shared memory and adds that to the series once
// (200^3 deck, one point: 1.5 M global FP64 atomics on a few hundred addresses
// took 72 us a step, 34 now).
constexpr int SERIES_PER = 4, SERIES_CELLS = 256 * SERIES_PER, SERIES_WIN = 512;

__global__ void __launch_bounds__(256) nfff_series_kernel(const DevNfffSeries S)
{
    __shared__ double win[3][SERIES_WIN];
    __shared__ int first;
    const int step = *S.step + S.off;
    const double C0 = 299792458.0, PI = 3.14159265358979323846;
    const double dx = S.dx, dt = S.dt;
    const double size = __dmul_rn(dx, dx);
    for (int p = blockIdx.y; p < S.npoints; p += gridDim.y) {
        const double x = S.points[3 * p], y = S.points[3 * p + 1], z = S.points[3 * p + 2];
        int nn[SERIES_PER];
        double ka[SERIES_PER], kb[SERIES_PER], kc[SERIES_PER];
        if (threadIdx.x == 0) first = 0x7fffffff;
        for (int q = threadIdx.x; q < 3 * SERIES_WIN; q += blockDim.x) (&win[0][0])[q] = 0.0;
        __syncthreads();
        int lo = 0x7fffffff;
#pragma unroll
        for (int c = 0; c < SERIES_PER; c++) {
            const int s = blockIdx.x * SERIES_CELLS + c * 256 + threadIdx.x;
            nn[c] = -1;
            if (s >= S.ns) continue;
            const int fc = S.face[s];
            const double ux = x - S.cell_ijk[3 * s], uy = y - S.cell_ijk[3 * s + 1], uz = z - S.cell_ijk[3 * s + 2];
            const double rc = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(ux, ux), __dmul_rn(uy, uy)), __dmul_rn(uz, uz)));
            const double pos = (fc & 1) ? 1.0 : -1.0;
            const double dot = pos * (fc < 2 ? ux : fc < 4 ? uy : uz);
            const double ct = dot / rc;
            const double r = __dmul_rn(rc, dx);
            const int m = (int)__dadd_rn((double)(step + 1), __ddiv_rn(r, __dmul_rn(C0, dt))) - S.istart[p];
            if (m < 3 || m >= S.ndata) continue;
            nn[c] = m;
            lo = min(lo, m);
            ka[c] = pos / (4.0 * PI * r) / 2.0 / dx * size;
            kb[c] = -1.0 / (4.0 * PI) * ct / (r * r) * size;
            kc[c] = 1.0 / (4.0 * PI) * ct / (C0 * r) / 2.0 / dt * size;
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        if ((threadIdx.x & 31) == 0) atomicMin(&first, lo);
        __syncthreads();
        const int base = first - 2;   // the window holds the series from here on
#pragma unroll
        for (int c = 0; c < SERIES_PER; c++) {
            if (nn[c] < 0) continue;
            const int s = blockIdx.x * SERIES_CELLS + c * 256 + threadIdx.x;
            const int64_t cc = S.cell[s], st = S.nstride[s];
            const int w = nn[c] - base;
            for (int a = 0; a < 3; a++) {
                const float *E = S.e[a];
                const double ev = (double)ld_any(E, cc, S.storage);
                const double dv = (double)ld_any(E, cc + st, S.storage) - (double)ld_any(E, cc - st, S.storage);
                const double t0 = kc[c] * ev, t1 = ka[c] * dv + kb[c] * ev;
                if (w < SERIES_WIN) {
                    atomicAdd(&win[a][w], t0);
                    atomicAdd(&win[a][w - 1], t1);
                    atomicAdd(&win[a][w - 2], -t0);
                } else {   // a cell far from the CTA's first
                    double *F = S.series + ((size_t)p * 3 + a) * S.ndata + nn[c];
                    atomicAdd(F, t0);
                    atomicAdd(F - 1, t1);
                    atomicAdd(F - 2, -t0);
                }
            }
        }
        __syncthreads();
        for (int q = threadIdx.x; q < 3 * SERIES_WIN; q += blockDim.x) {
            const double v = (&win[0][0])[q];
            if (v != 0.0) atomicAdd(S.series + ((size_t)p * 3 + q / SERIES_WIN) * S.ndata + base + q % SERIES_WIN, v);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ host copies

// Host values to and from the storage type: double to float first (FP64 storage
// keeps the double), then to nearest; H components carry the 16-bit scale.  PCIe
// bounds the copies around these by 100 times.
template <class T, class H>
__global__ void pack_kernel(const H *src, T *dst, size_t n, float scale)
{
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
        if constexpr (sizeof(T) == 8) dst[q] = (T)src[q];
        else Stor<T>::st(reinterpret_cast<float *>(dst), (int64_t)q, (float)src[q] * scale);
    }
}

template <class T, class H>
__global__ void unpack_kernel(const T *src, H *dst, size_t n, float scale)
{
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
        if constexpr (sizeof(T) == 8) dst[q] = (H)src[q];
        else dst[q] = (H)(Stor<T>::ld(reinterpret_cast<const float *>(src), (int64_t)q) * scale);
    }
}

unsigned copy_grid(size_t n) { return (unsigned)((n + 1023) / 1024 < 148 * 8 ? (n + 1023) / 1024 : 148 * 8); }

template <class T>
void pack_t(int hsz, const void *host, float *field, size_t off, size_t n, float scale, cudaStream_t st)
{
    T *f = reinterpret_cast<T *>(field) + off;
    if (hsz == 4) pack_kernel<<<copy_grid(n), 256, 0, st>>>(static_cast<const float *>(host), f, n, scale);
    else pack_kernel<<<copy_grid(n), 256, 0, st>>>(static_cast<const double *>(host), f, n, scale);
}

template <class T>
void unpack_t(int hsz, const float *field, size_t off, void *host, size_t n, float scale, cudaStream_t st)
{
    const T *f = reinterpret_cast<const T *>(field) + off;
    if (hsz == 4) unpack_kernel<<<copy_grid(n), 256, 0, st>>>(f, static_cast<float *>(host), n, scale);
    else unpack_kernel<<<copy_grid(n), 256, 0, st>>>(f, static_cast<double *>(host), n, scale);
}

}  // namespace

void launch_pack(int storage, int hsz, const void *host, float *field, size_t off, size_t n, float scale, cudaStream_t st)
{
    if (n == 0) return;
    if (storage == FDTD_STORE_F64) pack_t<double>(hsz, host, field, off, n, scale, st);
    else if (storage == FDTD_STORE_F16) pack_t<__half>(hsz, host, field, off, n, scale, st);
    else if (storage == FDTD_STORE_BF16) pack_t<__nv_bfloat16>(hsz, host, field, off, n, scale, st);
    else pack_t<float>(hsz, host, field, off, n, scale, st);
}

void launch_unpack(int storage, int hsz, const float *field, size_t off, void *host, size_t n, float scale, cudaStream_t st)
{
    if (n == 0) return;
    if (storage == FDTD_STORE_F64) unpack_t<double>(hsz, field, off, host, n, scale, st);
    else if (storage == FDTD_STORE_F16) unpack_t<__half>(hsz, field, off, host, n, scale, st);
    else if (storage == FDTD_STORE_BF16) unpack_t<__nv_bfloat16>(hsz, field, off, host, n, scale, st);
    else unpack_t<float>(hsz, field, off, host, n, scale, st);
}

void launch_any_nonzero(const float *p, int64_t n, int real64, int *flag, cudaStream_t st)
{
    any_nonzero_kernel<<<1184, 256, 0, st>>>(reinterpret_cast<const uint32_t *>(p), real64 ? 2 * n : n, real64, flag);
}

void launch_aux_line(const DevAux &a, cudaStream_t st) { aux_line_kernel<<<1, 1024, 0, st>>>(a); }

void launch_close_steps(const DevAux &a, const float *const *before, cudaStream_t st)
{
    close_steps_kernel<<<1, 256, 0, st>>>(a, before);
}

void launch_probe_capture(const DevAux &a, cudaStream_t st) { probe_capture_kernel<<<1, 256, 0, st>>>(a); }

void launch_tsf_faces(const DevPlan &p, int total, cudaStream_t st)
{
    if (total > 0) tsf_face_kernel<<<(total + 255) / 256, 256, 0, st>>>(p, total);
}

void launch_aux_step_batch(const DevAux *a, int nplans, cudaStream_t st)
{
    if (nplans > 0) aux_step_batch<<<nplans, 1024, 0, st>>>(a);
}

void launch_tsf_faces_batch(const DevPlan *p, int nplans, int max_cells, cudaStream_t st)
{
    if (nplans > 0 && max_cells > 0) tsf_face_batch<<<dim3((max_cells + 255) / 256, nplans), 256, 0, st>>>(p);
}

void launch_nfff_accumulate_batch(const DevNfff *n, int nplans, int max_cells, cudaStream_t st)
{
    if (nplans <= 0 || max_cells <= 0) return;
    nfff_sample_batch<<<dim3((max_cells + 255) / 256, nplans), 256, 0, st>>>(n);
    nfff_fold_batch<<<dim3((max_cells + 127) / 128, nplans), 128, 0, st>>>(n);
}

void launch_nfff_accumulate(const DevNfff &n, cudaStream_t st)
{
    if (n.ns <= 0) return;
    nfff_sample_kernel<<<(n.ns + 255) / 256, 256, 0, st>>>(n);
    nfff_fold_kernel<<<(n.ns + 127) / 128, 128, 0, st>>>(n);
}

void launch_nfff_fold_pending(const DevNfff &n, cudaStream_t st)
{
    if (n.ns <= 0 || n.nfreq <= 0) return;
    nfff_fold_pending_kernel<<<(n.ns + 255) / 256, 256, 0, st>>>(n);
}

void launch_farfield_finalize(const DevFarfield &f, cudaStream_t st)
{
    if (f.npoints <= 0 || f.nfreq <= 0) return;
    const dim3 grid((f.npoints + FF_TILE - 1) / FF_TILE, f.groups);
    for (int f0 = 0; f0 < f.nfreq; f0 += 4) {
        switch (f.nfreq - f0) {
        case 1: farfield_partial_kernel<1><<<grid, 128, 0, st>>>(f, f0); break;
        case 2: farfield_partial_kernel<2><<<grid, 128, 0, st>>>(f, f0); break;
        case 3: farfield_partial_kernel<3><<<grid, 128, 0, st>>>(f, f0); break;
        default: farfield_partial_kernel<4><<<grid, 128, 0, st>>>(f, f0); break;
        }
    }
    const int nt = f.npoints * f.nfreq * 3;
    farfield_reduce_kernel<<<(nt + 255) / 256, 256, 0, st>>>(f);
}

void launch_nfff_series(const DevNfffSeries &s, cudaStream_t st)
{
    if (s.ns <= 0 || s.npoints <= 0) return;
    const dim3 grid((s.ns + SERIES_CELLS - 1) / SERIES_CELLS, (unsigned)min(s.npoints, 65535));
    nfff_series_kernel<<<grid, 256, 0, st>>>(s);
}
