// fdtd_kernels.cuh -- launch interface of the device kernels (fdtd_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fdtd_internal.h"


struct DevAux {                 // 1D auxiliary grid of the TSF source (1dpool.c)
    double *e, *h;              // res values each
    double *bnd;                // 8 saved boundary values (Sv1DPool fbnx*)
    const double *wave;
    int nwave;
    int res;
    double ce, chh;             // (1/eps)*dt/(EPS0*dx1) and (1/mu)*dt/(MU0*dx1)
    double lc;                  // Liao factor (dt*c - dx1)/(dt*c + dx1)
    int *step;                  // device step counter
    int off;                    // steps since the counter was last advanced (aux_line, close_steps)
    // probes of the previous step
    int nprobes;
    const int64_t *probe_cells;
    const float *const *fields; // 6 pointers to the field set that holds the previous step
    double *probe_out;          // [p][nsteps][6]
    int nsteps_planned;
    int storage;                // FDTD_STORE_* of the fields
    float ihs;                  // 1 / H storage scale
};

// steps of E samples buffered per surface cell before they are folded into
// the FP64 accumulators (one accumulator read/write per NFFF_RING steps)
constexpr int NFFF_RING = 8;

struct DevNfff {
    int ns;                     // surface cells
    int nfreq;
    const int32_t *cell;        // linear index of the surface cell
    const int32_t *nstride;     // +/- stride along the face normal
    const float *const *e;      // 3 E field pointers (the set written by this step)
    double2 *acc;               // [(f*6 + q)*ns + s], q = Ex,Ey,Ez, dEx,dEy,dEz
    float *ring;                // NFFF_RING steps of raw samples [(slot*9 + 3a + r)*ns + s], r: E(c), E(c+st), E(c-st);
                                // FP32 elements (FP64 for FDTD_STORE_F64 plans)
    const double *omega_dt;     // nfreq
    const int *step;            // device step counter; the step sampled is *step + off
    int off;
    double inv2dx;
    int storage;                // FDTD_STORE_* of the fields
};

// *flag = 1 if any of n FP32 (FP64) values is not zero
void launch_any_nonzero(const float *p, int64_t n, int real64, int *flag, cudaStream_t st);
// the 1D grid step of step *a.step + a.off; also, from a.fields, the probes of two steps before (a.off >= 2) or
// of the step before (a.off == 0)
void launch_aux_line(const DevAux &a, cudaStream_t st);
// the end of a call of a.off steps: probes of its last step (a.fields) and of the one before (`before`, if set), step counter
void launch_close_steps(const DevAux &a, const float *const *before, cudaStream_t st);

// Batched forms: one launch covers many plans whose per-plan parameters are
// device tables (of this step's parity), indexed by the plan number.
void launch_aux_step_batch(const DevAux *a, int nplans, cudaStream_t st);
void launch_tsf_faces_batch(const DevPlan *p, int nplans, int max_cells, cudaStream_t st);
void launch_nfff_accumulate_batch(const DevNfff *n, int nplans, int max_cells, cudaStream_t st);
void launch_probe_capture(const DevAux &a, cudaStream_t st);
// n host values (hsz bytes each: 4 float, 8 double) at `host`, device memory, to
// and from elements off .. off+n-1 of a field stored as FDTD_STORE_*; the field
// holds `scale` times the value (pack), or `scale` undoes that (unpack)
void launch_pack(int storage, int hsz, const void *host, float *field, size_t off, size_t n, float scale, cudaStream_t st);
void launch_unpack(int storage, int hsz, const float *field, size_t off, void *host, size_t n, float scale, cudaStream_t st);
void launch_tsf_faces(const DevPlan &p, int total, cudaStream_t st);
void launch_nfff_accumulate(const DevNfff &n, cudaStream_t st);
// folds the samples of the steps since the last multiple of NFFF_RING into the
// accumulators and clears their ring slots; due before the accumulators are read
void launch_nfff_fold_pending(const DevNfff &n, cudaStream_t st);

struct DevFarfield {
    int npoints, nfreq, ns;
    const int32_t *points;      // 3*npoints
    const int32_t *istart;
    const int32_t *cell_ijk;    // 3*ns  (i,j,k of each surface cell)
    const int8_t *face;         // ns, 0..5 = x0 xn y0 yn z0 zn
    const double2 *acc;
    const double *omega;        // nfreq
    double dt, dx;
    double2 *out;               // [(p*nfreq + f)*3 + c]
    // tiled finalize
    int ntw;                    // twiddle entries per frequency
    const double2 *tw;          // [f*ntw + R] = exp(-i omega R dt)
    int groups;                 // surface-cell groups of the partial sums
    double2 *part;              // [((g*npoints + p)*nfreq + f)*3 + c] (scratch)
};

// The reference's own time-domain far-field series (farfield.c:175-405),
// accumulated exactly: three taps per (surface cell, far point) and step.
struct DevNfffSeries {
    int ns, npoints, ndata;
    const int32_t *cell;        // linear index of the surface cell
    const int32_t *nstride;     // +/- stride along the face normal
    const int32_t *cell_ijk;    // 3*ns
    const int8_t *face;         // ns
    const int32_t *points;      // 3*npoints
    const int32_t *istart;      // npoints
    const float *const *e;      // 3 E field pointers (the set written by this step)
    double *series;             // [(p*3 + c)*ndata + m]
    const int *step;            // device step counter; the step added is *step + off
    int off;
    double dx, dt;
    int storage;                // FDTD_STORE_* of the fields
};
void launch_nfff_series(const DevNfffSeries &s, cudaStream_t st);

constexpr int FF_TILE = 256;   // far points of a block of the far-field sum
void launch_farfield_finalize(const DevFarfield &f, cudaStream_t st);
