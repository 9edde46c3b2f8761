// fdtd_flat.cuh -- flat step kernels (fdtd_flat.cu): one thread per group of
// V consecutive k cells, one launch for the H half step and one for the E half
// step, over a list of boxes.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fdtd_internal.h"

// what the cells of a box can meet
enum {
    FB_X = 1, FB_Y = 2, FB_Z = 4,   // a CPML slab of that axis
    FB_EDGE = 8,                    // anything but the plain update: CPML, kappa, a grid edge
    FB_TSF = 16,                    // the TSF correction region [t0 - 1, t1]
    FB_ADE = 32,                    // a cell of the dispersive branch
    FB_ONE = 64,                    // one class for all cells, without PEC rule or design coefficients, and with
                                    // all components dispersive or none
    FB_INNER = 256,                 // the plain interior box (profiles)
    FB_SPEC = 128                   // FB_ONE, exactly one slab axis, and no grid edge but that slab's own
};

// One block of a flat kernel: FLAT_NT groups of a box from group t0 on, k
// fastest.  nk groups a row, nj rows a plane; (mk, sk) and (mj, sj) divide by
// them (flat_div).  Every block carries its box whole, so that a thread is one
// load away from its cell.
struct alignas(16) FlatBlock {
    int i0, j0, k0;
    unsigned t0;
    int nk, nj;
    unsigned total;                 // groups of the box, < 2^31
    int flags;                      // FB_*
    unsigned mk, mj;
    int8_t sk, sj;
    int16_t cls;                    // the class of a FB_ONE box
    int inst;                       // plan of the box in a batched launch
};
static_assert(sizeof(FlatBlock) == 48, "three 16-byte loads");

// threads of a block
constexpr int FLAT_NT = 128;

// n / d for n < 2^31: (umulhi(n, m) + n) >> s with s = ceil(log2 d) and
// m = floor(2^32 (2^s - d) / d) + 1 (Granlund and Montgomery, PLDI 1994)
inline void flat_magic(unsigned d, unsigned *m, int *s)
{
    int l = 0;
    while ((1ull << l) < d) l++;
    *s = l;
    *m = (unsigned)((((1ull << l) - d) << 32) / d + 1);
}

struct FlatList {
    const FlatBlock *blocks = nullptr;
    unsigned n = 0;
};

// cells per thread of a plan: 4 (FP32 and 16-bit storage) or 2 (FP64) when the
// k rows are whole vectors, else 1
int flat_width(int storage, int zr);

cudaError_t launch_flat_h(const DevPlan &p, const FlatList &l, int width, int storage, cudaStream_t st);
// beside_h: the launch before it in `st` is the step's H kernel, beside whose last blocks E may start
cudaError_t launch_flat_e(const DevPlan &p, const FlatList &l, int width, bool ade, int npoles, int storage, bool beside_h,
                          cudaStream_t st);
// many plans in one launch: plans is the device table of this step's parity
cudaError_t launch_flat_h_batch(const DevPlan *plans, const FlatList &l, int width, int storage, cudaStream_t st);
cudaError_t launch_flat_e_batch(const DevPlan *plans, const FlatList &l, int width, bool ade, int npoles, int storage,
                                cudaStream_t st);
