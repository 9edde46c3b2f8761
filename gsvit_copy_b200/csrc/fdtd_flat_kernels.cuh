// fdtd_flat_kernels.cuh -- flat step kernels: the H half step and the E half step
// of the boxes of a plan, one thread per group of V consecutive k cells.  Each
// storage type is a translation unit of its own (fdtd_flat_*.cu).
//
// H: ystep_h (yee.c:146-265), the CPML psi_H recursions and corrections with
// the zeroed outer planes (boundary.c:347-519) and the TSF H corrections
// (source.c:1464-1672).  E: ystep_e with the ADE branch, its embedded CPML, the
// ordinary update and the PEC rule (yee.c:530-1247), the CPML psi_E recursions
// and corrections (boundary.c:691-884) and the TSF E corrections
// (source.c:547-771).  H reads the input field set only and E the H it wrote,
// so no two threads of a launch share a cell.  Templated on the storage type T,
// whose arithmetic type R is FP32, or FP64 for FP64 storage, and on V.
//
// A box carries flags of what its cells can meet (FB_*), so that the branches
// on faces, TSF and dispersion are uniform over a block; the rules of the
// reference are then tested per thread (x and y faces) or per cell (z faces).
// The bodies are instantiated for what most cells are: plain cells (FACE 0), a
// slab of one axis (FACE 1, 2, 4), each with one known class (ONE: no class
// map, coefficients from one table entry, the dispersive state and psi
// requested with the fields), and for anything (FACE 7).
// Faces go in the reference's order x0 y0 z0 xn yn zn, or, when the plan asks
// for it (DevPlan::axis_order), axis by axis; the two differ by rounding in
// cells of several slabs.  Expressions keep one form in every body, so that a
// cell gets the same bits from each: BF16 storage rounds by a hash, where one
// other last bit would end in other fields.
//
// Memory bounds both kernels.  Boxes cut the k rows (at the slabs, at the metal
// surface), so the blocks are ordered by plane: the pieces of a row run at
// about the same time, and a line two of them share comes from DRAM once.
// 256^3 rough surface, H / E: 866 / 1243 MB of DRAM traffic and 162 / 280 us with
// the boxes one after the other, 702 / 1012 MB and 126 / 235 us by plane (5.6 /
// 4.3 TB/s; the kernels of one cell a thread and of the CPML tiles they
// replace took 552 us a step here, 393 now).  Tried: pairs of cells a thread
// (24 warps an SM: E 10 % slower), whole rows through bodies that can do
// everything (same traffic, E 357 us), streaming cache hints and staggered
// array offsets (no change), a persistent grid (20 % slower).
#pragma once
#include <cuda_runtime.h>

#include "fdtd_device.cuh"
#include "fdtd_flat.cuh"

namespace {

// a b + c d, the first (fma1) or the second product (fma2) unrounded, and
// a b + c with one rounding.  Written out, so that a cell gets the same bits
// from every body (and from the kernels this one replaces, whose forms these
// are) whatever the compiler would contract in each.
__device__ __forceinline__ float mad(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double mad(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma1(float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ double fma1(double a, double b, double c, double d) { return __fma_rn(a, b, __dmul_rn(c, d)); }
__device__ __forceinline__ float fma2(float a, float b, float c, float d) { return __fmaf_rn(c, d, __fmul_rn(a, b)); }
__device__ __forceinline__ double fma2(double a, double b, double c, double d) { return __fma_rn(c, d, __dmul_rn(a, b)); }

// ---- V consecutive elements

template <class T, int V>
__device__ __forceinline__ void ldv(real_t<T> (&d)[V], const float *base, int64_t c)
{
    if constexpr (V == 4) {
        const float4 v = ldg4<T>(base, c);
        d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    } else if constexpr (V == 2) {
        static_assert(sizeof(T) == 8, "pairs are for FP64");
        const double2 v = *reinterpret_cast<const double2 *>(reinterpret_cast<const double *>(base) + c);
        d[0] = v.x; d[1] = v.y;
    } else {
        d[0] = Stor<T>::ld(base, c);
    }
}

// `scale` applies to 16-bit storage only
template <class T, int V>
__device__ __forceinline__ void stv(float *base, int64_t c, const real_t<T> (&v)[V], float scale, uint32_t stp, uint32_t array)
{
    if constexpr (V == 4) {
        stg4<T>(base, c, make_float4(v[0], v[1], v[2], v[3]), scale, stp, array);
    } else if constexpr (V == 2) {
        *reinterpret_cast<double2 *>(reinterpret_cast<double *>(base) + c) = make_double2(v[0], v[1]);
    } else {
        st_any<T>(base, c, Stor<T>::scaled ? v[0] * scale : v[0], stp, array);
    }
}

// the dispersive state: elements of the arithmetic type
template <class R, int V>
__device__ __forceinline__ void ldstate(R (&d)[V], float *p, int64_t c)
{
    if constexpr (V == 4) ldq4a(d, p + c);
    else if constexpr (V == 2) ldv<R, V>(d, p, c);
    else d[0] = Tab<R>::state(p)[c];
}
template <class R, int V>
__device__ __forceinline__ void ststate(float *p, int64_t c, const R (&v)[V])
{
    if constexpr (V == 4) stq4a(p + c, v);
    else if constexpr (V == 2) stv<R, V>(p, c, v, 1.f, 0, 0);
    else Tab<R>::state(p)[c] = v[0];
}

// psi of the cells with m[c], as a vector when `vec` (every element of it is
// then inside the array)
template <class T, int V>
__device__ __forceinline__ void ldpsi(real_t<T> (&v)[V], const float *p, int64_t q, bool vec, const bool (&m)[V], float scale)
{
    if (V == 1 || vec) {
        ldv<T, V>(v, p, q);
    } else {
#pragma unroll
        for (int c = 0; c < V; c++) {
            v[c] = 0;
            if (m[c]) v[c] = Stor<T>::ld(p, q + c);
        }
    }
    if constexpr (Stor<T>::scaled) {
#pragma unroll
        for (int c = 0; c < V; c++) v[c] *= scale;
    }
}

// A vector store writes back, for the cells without m[c], the value it loaded:
// psi the rules never update, zero from the start on.
template <class T, int V>
__device__ __forceinline__ void stpsi(float *p, int64_t q, bool vec, const bool (&m)[V], float scale, const real_t<T> (&v)[V],
                                      uint32_t stp, uint32_t array)
{
    if (V > 1 && vec) {
        stv<T, V>(p, q, v, scale, stp, array);
    } else {
#pragma unroll
        for (int c = 0; c < V; c++)
            if (m[c]) st_any<T>(p, q + c, Stor<T>::scaled ? v[c] * scale : v[c], stp, array);
    }
}

// table values q .. q+V-1 of the cells with m[c]
template <class R, int V>
__device__ __forceinline__ void ldtab(R (&d)[V], const float *p, int q, bool vec, const bool (&m)[V])
{
    if constexpr (V == 4) {
        if (vec) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(p + q));
            d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
            return;
        }
    }
#pragma unroll
    for (int c = 0; c < V; c++) {
        d[c] = 0;
        if (m[c]) d[c] = Tab<R>::ld(p, q + c);
    }
}

// V values of a per-axis table from k (a multiple of V)
template <class R, int V>
__device__ __forceinline__ void ldaxis(R (&d)[V], const float *p, int k)
{
    if constexpr (V == 4) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(p + k));
        d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    } else {
#pragma unroll
        for (int c = 0; c < V; c++) d[c] = Tab<R>::ld(p, k + c);
    }
}

template <int V>
__device__ __forceinline__ uint32_t class_word(const DevPlan &P, int i, int j, int k)
{
    const uint8_t *p = P.cls + ((int64_t)i * P.yr + j) * P.cpitch + k;
    if constexpr (V == 4) return __ldg(reinterpret_cast<const uint32_t *>(p));
    else if constexpr (V == 2) return __ldg(reinterpret_cast<const uint16_t *>(p));
    else return __ldg(p);
}

template <int V>
__device__ __forceinline__ bool one_class(uint32_t cw)
{
    if constexpr (V == 4) return cw == (cw & 0xffu) * 0x01010101u;
    else if constexpr (V == 2) return (cw & 0xffu) == (cw >> 8);
    else return true;
}

// does the group of V cells from (i, j, k) touch a face of the TSF box?
// (the per-cell tests are those of tsf_add_h / tsf_add_e)
template <int V>
__device__ __forceinline__ bool tsf_hit(const DevPlan &P, int i, int j, int k)
{
    const int i0 = P.t0[0], in = P.t1[0], j0 = P.t0[1], jn = P.t1[1], k0 = P.t0[2], kn = P.t1[2], kh = k + V - 1;
    if (i < i0 - 1 || i > in || j < j0 - 1 || j > jn || kh < k0 - 1 || k > kn) return false;
    const bool fi = i <= i0 || i == in, fj = j <= j0 || j == jn;
    const bool fk = (k <= k0 && kh >= k0 - 1) || kh >= kn;
    return fi || fj || fk;
}

// ------------------------------------------------------------ the group of a thread

__device__ __forceinline__ unsigned flat_div(unsigned n, unsigned m, int s) { return (__umulhi(n, m) + n) >> s; }

struct FlatCell {
    int i, j, k, flags, inst;
    int cls;      // the class of a FB_ONE box
};

// the group of this thread; false past the end of the box
template <int V>
__device__ __forceinline__ bool flat_cell(const FlatBlock *blocks, unsigned bid, int ahead, FlatCell &c)
{
    if (threadIdx.x == 0) {
        const int64_t b = (int64_t)bid + ahead;
        if (b >= 0 && b < gridDim.x) prefetch_l2(blocks + b);
    }
    FlatBlock B;
    const int4 *src = reinterpret_cast<const int4 *>(blocks + bid);
    int4 *dst = reinterpret_cast<int4 *>(&B);
#pragma unroll
    for (int w = 0; w < (int)(sizeof(FlatBlock) / 16); w++) dst[w] = __ldg(src + w);
    const unsigned t = B.t0 + threadIdx.x;
    if (t >= B.total) return false;
    const unsigned r = flat_div(t, B.mk, B.sk), q = flat_div(r, B.mj, B.sj);
    c.k = B.k0 + V * (int)(t - r * B.nk);
    c.j = B.j0 + (int)(r - q * B.nj);
    c.i = B.i0 + (int)q;
    c.flags = B.flags;
    c.inst = B.inst;
    c.cls = B.cls;
    return true;
}

// E blocks are launched beside the last H blocks (programmatic dependent
// launch): H allows it when all its blocks have started, E waits here for H to
// end before it reads what H wrote (us a step: 64^3 launched one by one 27.4 -> 24.2,
// 200^3 replayed 160 -> 153, 256^3 381 -> 374).
__device__ __forceinline__ void e_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void after_h() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ------------------------------------------------------------ H half step

// the slab of axis AX (0 x, 1 y) that holds index q, its position there, and
// whether the H / E rules update psi at it
struct Slab {
    int f, pos, d;
};
__device__ __forceinline__ Slab slab_of(const DevPlan &P, int ax, int q, int res)
{
    const int lo = P.cp_d[2 * ax], hi = P.cp_d[2 * ax + 1];
    const bool low = q < lo;
    return Slab{low ? 2 * ax : 2 * ax + 1, low ? q : q - (res - hi), low ? lo : hi};
}

template <class T, int V, int FACE, bool ONE>
__device__ __forceinline__ void flat_h_group(const DevPlan &P, const FlatCell &g)
{
    using R = real_t<T>;
    constexpr bool ANY = FACE == 7, EDGE = FACE != 0;
    const int i = g.i, j = g.j, k = g.k, flags = g.flags;
    const int xr = P.xr, yr = P.yr, zr = P.zr;
    const int64_t c0 = (int64_t)i * P.si + (int64_t)j * P.sj + k;
    const bool il = ANY && i == xr - 1, jl = ANY && j == yr - 1, kl = (FACE & 4) && k + V == zr;
    const float *EX = P.fin[0], *EY = P.fin[1], *EZ = P.fin[2];
    R ex[V], ey[V], ez[V], exj[V], ezj[V], eyi[V], ezi[V], hx[V], hy[V], hz[V];
    ldv<T, V>(ex, EX, c0);
    ldv<T, V>(ey, EY, c0);
    ldv<T, V>(ez, EZ, c0);
    if (jl) {
#pragma unroll
        for (int c = 0; c < V; c++) exj[c] = ezj[c] = 0;
    } else {
        ldv<T, V>(exj, EX, c0 + P.sj);
        ldv<T, V>(ezj, EZ, c0 + P.sj);
    }
    if (il) {
#pragma unroll
        for (int c = 0; c < V; c++) eyi[c] = ezi[c] = 0;
    } else {
        ldv<T, V>(eyi, EY, c0 + P.si);
        ldv<T, V>(ezi, EZ, c0 + P.si);
    }
    const R exk1 = kl ? R(0) : Stor<T>::ld(EX, c0 + V), eyk1 = kl ? R(0) : Stor<T>::ld(EY, c0 + V);
    ldv<T, V>(hx, P.fin[3], c0);
    ldv<T, V>(hy, P.fin[4], c0);
    ldv<T, V>(hz, P.fin[5], c0);
    const float ips = P.ips, ps = P.ps;
    const bool iin = !ANY || (i >= 1 && !il), jin = !ANY || (j >= 1 && !jl);
    bool kin[V], kall = true;
#pragma unroll
    for (int c = 0; c < V; c++) {
        kin[c] = !(FACE & 4) || (k + c >= 1 && !(kl && c == V - 1));
        kall = kall && kin[c];
    }
    // x and y slabs: psi of the group, requested here when the box has no other
    R p0[V], p1[V];
    Slab S{0, 0, 0};
    bool on = false;
    int64_t q = 0;
    auto x_slab = [&]() {
        S = slab_of(P, 0, i, xr);
        on = P.cp_on[S.f] && jin && (S.f == X0 ? i < S.d - 1 : S.pos >= 1 && i < xr - 1);
        q = ((int64_t)S.pos * yr + j) * zr + k;
    };
    auto y_slab = [&]() {
        S = slab_of(P, 1, j, yr);
        on = P.cp_on[S.f] && iin && (S.f == Y0 ? j < S.d - 1 : S.pos >= 1 && j < yr - 1);
        q = ((int64_t)i * S.d + S.pos) * zr + k;
    };
    bool m[V], mall = true;
    auto z_slab = [&](int f) {
        S.f = f;
        S.d = P.cp_d[f];
        const int base = f == Z0 ? 0 : zr - S.d;
        S.pos = k - base;
        on = false;
        mall = true;
#pragma unroll
        for (int c = 0; c < V; c++) {
            m[c] = P.cp_on[f] && iin && jin && (f == Z0 ? k + c < S.d - 1 : S.pos + c >= 1 && k + c < zr - 1);
            on = on || m[c];
            mall = mall && m[c];
        }
        q = ((int64_t)i * yr + j) * S.d + S.pos;
    };
    auto load_psi = [&](bool vec, const bool (&mask)[V]) {
        if (!on) return;
        ldpsi<T, V>(p1, P.psih_in[S.f][1], q, vec, mask, ips);
        ldpsi<T, V>(p0, P.psih_in[S.f][0], q, vec, mask, ips);
    };
    if constexpr (FACE == 1) { x_slab(); load_psi(true, kin); }
    if constexpr (FACE == 2) { y_slab(); load_psi(true, kin); }
    if constexpr (FACE == 4) { z_slab(k < P.cp_d[Z0] ? Z0 : ZN); load_psi(V == 1 || S.d % V == 0, m); }
    const uint32_t stp = sr_step<T>(P);
    const float4 *cl = reinterpret_cast<const float4 *>(P.classes);
    const uint32_t cw = ONE ? (uint32_t)g.cls : class_word<V>(P, i, j, k);
    const bool uni = ONE || one_class<V>(cw);
    if constexpr (Stor<T>::scaled) {
#pragma unroll
        for (int c = 0; c < V; c++) { hx[c] *= P.ihs; hy[c] *= P.ihs; hz[c] *= P.ihs; }
    }
    R da = 0, db = 0;
    Tab<R>::hcoef(P, cl, cw & 0xff, da, db);
    // the forward differences take the neighbours' places: dzi, dyi, dxj, dzj
    R dxk[V], dyk[V];
#pragma unroll
    for (int c = 0; c < V; c++) {
        dyk[c] = (c + 1 < V ? ey[c + 1 < V ? c + 1 : 0] : eyk1) - ey[c];
        dxk[c] = (c + 1 < V ? ex[c + 1 < V ? c + 1 : 0] : exk1) - ex[c];
    }
#pragma unroll
    for (int c = 0; c < V; c++) {
        ezj[c] -= ez[c];
        exj[c] -= ex[c];
        ezi[c] -= ez[c];
        eyi[c] -= ey[c];
    }
    R ikx = 1, iky = 1, ikzs[V] = {}, dbdx[V];
    const R dx = Tab<R>::dx(P), idx_ = R(1) / dx;
    if constexpr (EDGE) { ikx = Tab<R>::ld(P.ikh[0], i); iky = Tab<R>::ld(P.ikh[1], j); ldaxis<R, V>(ikzs, P.ikh[2], k); }
#pragma unroll
    for (int c = 0; c < V; c++) {
        if (c > 0 && !uni) Tab<R>::hcoef(P, cl, (cw >> (8 * c)) & 0xff, da, db);
        const bool klc = kl && c == V - 1;
        const R ikz = EDGE ? ikzs[c] : R(1);
        if (!(jl || klc)) hx[c] = fma1(da, hx[c], db, dyk[c] * ikz - ezj[c] * iky);
        if (!(il || klc)) hy[c] = fma1(da, hy[c], db, ezi[c] * ikx - dxk[c] * ikz);
        if (!(il || jl)) hz[c] = fma1(da, hz[c], db, exj[c] * iky - eyi[c] * ikx);
        dbdx[c] = db * dx;
    }
    if ((flags & FB_TSF) && tsf_hit<V>(P, i, j, k)) tsf_add_h<R, V>(P, i, j, k, hx, hy, hz);
#pragma unroll 1
    for (int turn = (ANY && !P.axis_order ? 0 : 2); turn <= (ANY && !P.axis_order ? 1 : 2); turn++) {
        auto now = [&]() { return turn == 2 || (S.f & 1) == turn; };
        // x faces: psi[1] <- dey_i (hz -= dbdx psi), psi[0] <- dez_i (hy += dbdx psi)
        if constexpr ((FACE & 1) != 0) {
            if constexpr (ANY) { on = false; if (flags & FB_X) { x_slab(); on = on && now(); load_psi(true, kin); } }
            if (on) {
                const R bh = Tab<R>::ld(P.bh[S.f], S.pos), ch = Tab<R>::ld(P.ch[S.f], S.pos);
#pragma unroll
                for (int c = 0; c < V; c++) {
                    if (!kin[c]) continue;
                    p1[c] = fma2(bh, p1[c], ch * eyi[c], idx_);
                    p0[c] = fma2(bh, p0[c], ch * ezi[c], idx_);
                    hy[c] = mad(dbdx[c], p0[c], hy[c]);
                    hz[c] = mad(-dbdx[c], p1[c], hz[c]);
                }
                stpsi<T, V>(P.psih_out[S.f][1], q, kall, kin, ps, p1, stp, 18 + 2 * S.f + 1);
                stpsi<T, V>(P.psih_out[S.f][0], q, kall, kin, ps, p0, stp, 18 + 2 * S.f + 0);
            }
        }
        // y faces: psi[0] <- dez_j (hx -= dbdx psi), psi[1] <- dex_j (hz += dbdx psi)
        if constexpr ((FACE & 2) != 0) {
            if constexpr (ANY) { on = false; if (flags & FB_Y) { y_slab(); on = on && now(); load_psi(true, kin); } }
            if (on) {
                const R bh = Tab<R>::ld(P.bh[S.f], S.pos), ch = Tab<R>::ld(P.ch[S.f], S.pos);
#pragma unroll
                for (int c = 0; c < V; c++) {
                    if (!kin[c]) continue;
                    p0[c] = fma2(bh, p0[c], ch * ezj[c], idx_);
                    p1[c] = fma2(bh, p1[c], ch * exj[c], idx_);
                    hx[c] = mad(-dbdx[c], p0[c], hx[c]);
                    hz[c] = mad(dbdx[c], p1[c], hz[c]);
                }
                stpsi<T, V>(P.psih_out[S.f][0], q, kall, kin, ps, p0, stp, 18 + 2 * S.f + 0);
                stpsi<T, V>(P.psih_out[S.f][1], q, kall, kin, ps, p1, stp, 18 + 2 * S.f + 1);
            }
        }
        // z faces: psi[1] <- dex_k (hy -= dbdx psi), psi[0] <- dey_k (hx += dbdx psi)
        if constexpr ((FACE & 4) != 0) {
#pragma unroll 1
            for (int f = Z0; f <= (ANY ? ZN : Z0); f++) {
                if constexpr (ANY) {
                    if (!(flags & FB_Z)) break;
                    z_slab(f);
                    on = on && now();
                    load_psi(V == 1 || S.d % V == 0, m);
                }
                if (!on) continue;
                const bool vec = V == 1 || S.d % V == 0;
                R bh[V], ch[V];
                ldtab<R, V>(bh, P.bh[S.f], S.pos, vec, m);
                ldtab<R, V>(ch, P.ch[S.f], S.pos, vec, m);
#pragma unroll
                for (int c = 0; c < V; c++) {
                    if (!m[c]) continue;
                    p1[c] = fma2(bh[c], p1[c], ch[c] * dxk[c], idx_);
                    p0[c] = fma2(bh[c], p0[c], ch[c] * dyk[c], idx_);
                    hy[c] = mad(-dbdx[c], p1[c], hy[c]);
                    hx[c] = mad(dbdx[c], p0[c], hx[c]);
                }
                stpsi<T, V>(P.psih_out[S.f][1], q, vec && mall, m, ps, p1, stp, 18 + 2 * S.f + 1);
                stpsi<T, V>(P.psih_out[S.f][0], q, vec && mall, m, ps, p0, stp, 18 + 2 * S.f + 0);
            }
        }
    }
    // the outer H planes boundary_hstep zeroes (boundary.c:418-420, 455-457, 490-492)
#pragma unroll
    for (int c = 0; c < V; c++) {
        const bool klc = kl && c == V - 1;
        if ((P.cp_on[XN] && il && jin && kin[c]) || (P.cp_on[YN] && jl && iin && kin[c]) || (P.cp_on[ZN] && klc && iin && jin))
            hx[c] = hy[c] = hz[c] = 0;
    }
    stv<T, V>(P.fout[3], c0, hx, P.hs, stp, 3);
    stv<T, V>(P.fout[4], c0, hy, P.hs, stp, 4);
    stv<T, V>(P.fout[5], c0, hz, P.hs, stp, 5);
}

// ------------------------------------------------------------ E half step

template <class R>
struct ECoef {
    R ca[3], cb[3];
    R cba;          // CPML coefficient of the dispersive branch (one value for the three components)
    unsigned fl;
    int ade;
};

template <class R>
__device__ __forceinline__ int ade_of(const DevPlan &P, int cls)
{
    if constexpr (sizeof(R) == 8) return Tab<double>::cls(P, cls).ade;
    else return __ldg(&P.classes[cls].ade);
}

template <class R>
__device__ __forceinline__ void ecoef(const DevPlan &P, const float4 *cl, int cls, int i, int j, int k, ECoef<R> &C)
{
    R cba[3];
    Tab<R>::ecoef(P, cl, cls, C.ca, C.cb, cba, C.fl, C.ade);
    C.cba = cba[0];
    if (C.fl & CF_DESIGN) {   // adjoint design region: coefficients per cell
        const int64_t q = ((int64_t)(i - P.dbox[0]) * (P.dbox[3] - P.dbox[2]) + (j - P.dbox[2])) * (P.dbox[5] - P.dbox[4]) + (k - P.dbox[4]);
#pragma unroll
        for (int a = 0; a < 3; a++) { C.ca[a] = Tab<R>::ld(P.dcoef, 6 * q + a); C.cb[a] = Tab<R>::ld(P.dcoef, 6 * q + 3 + a); }
    }
}

// NPOLES: 0 the Drude term alone, 2 the Drude term and both poles, 1 the first
// pole alone (a Lorentz medium: the state of the other terms is zero and stays
// so; 150 x 118 x 131, half of it one: 126 us a step with variant 2, 94 here).
template <bool ADE, int NPOLES, class T, int V, int FACE, bool ONE>
__device__ __forceinline__ void flat_e_group(const DevPlan &P, const FlatCell &g)
{
    using R = real_t<T>;
    constexpr bool ANY = FACE == 7, EDGE = FACE != 0, DRUDE = NPOLES != 1;
    const int i = g.i, j = g.j, k = g.k, flags = g.flags;
    const int xr = P.xr, yr = P.yr, zr = P.zr;
    const int64_t c0 = (int64_t)i * P.si + (int64_t)j * P.sj + k;
    const bool i0 = ANY && i == 0, j0 = ANY && j == 0, k0 = (FACE & 4) && k == 0;
    const float *HX = P.fout[3], *HY = P.fout[4], *HZ = P.fout[5];   // H^{n+1/2}, written this step
    const uint32_t cw = ONE ? (uint32_t)g.cls : class_word<V>(P, i, j, k);
    const float4 *cl = reinterpret_cast<const float4 *>(P.classes);
    const bool uni = ONE || one_class<V>(cw);   // (a design cell takes its own coefficients all the same)
    R hx[V], hy[V], hz[V], hxj[V], hzj[V], hyi[V], hzi[V], eo[3][V];
#pragma unroll
    for (int a = 0; a < 3; a++) ldv<T, V>(eo[a], P.fin[a], c0);
    ECoef<R> C;
    // components owned by the ADE in some cell of the group, their Q and E^{n-1}
    unsigned adem = 0;
    R qd[3][V], w[3][V];
    if (ADE && (flags & FB_ADE)) {
        if constexpr (ONE) {
            adem = CF_ADE_X | CF_ADE_Y | CF_ADE_Z;   // FB_ONE: all or none
        } else {
#pragma unroll
            for (int c = 0; c < V; c++) {
                unsigned fl;
                if constexpr (sizeof(R) == 8) fl = Tab<double>::cls(P, (cw >> (8 * c)) & 0xff).flags;
                else fl = __ldg(&P.classes[(cw >> (8 * c)) & 0xff].flags);
                if (fl & CF_ADE_BRANCH) adem |= fl & (CF_ADE_X | CF_ADE_Y | CF_ADE_Z);
                if (uni) break;
            }
        }
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (!(adem & (1u << a))) continue;
            if constexpr (DRUDE) ldstate<R, V>(qd[a], P.q[a], c0);
            ldv<T, V>(w[a], P.fout[a], c0);   // E^{n-1}: the output set before this step writes it
        }
    }
    // Everything so far and psi_E is older than this step's H kernel, beside whose
    // last blocks these may start; H itself is not.
    after_h();
    ldv<T, V>(hx, HX, c0);
    ldv<T, V>(hy, HY, c0);
    ldv<T, V>(hz, HZ, c0);
    if (!j0) {
        ldv<T, V>(hxj, HX, c0 - P.sj);
        ldv<T, V>(hzj, HZ, c0 - P.sj);
    }
    if (!i0) {
        ldv<T, V>(hyi, HY, c0 - P.si);
        ldv<T, V>(hzi, HZ, c0 - P.si);
    }
    R hxk1 = k0 ? R(0) : Stor<T>::ld(HX, c0 - 1), hyk1 = k0 ? R(0) : Stor<T>::ld(HY, c0 - 1);
    // psi_E of the slab, requested here when the box has no other
    const bool zero_ij = ANY && ((P.cp_on[X0] && i0) || (P.cp_on[Y0] && j0));
    const bool kz0 = k0 && P.cp_on[Z0];
    R p0[V], p1[V];
    Slab S{0, 0, 0};
    bool on = false, m[V];
    int64_t q = 0;
    auto xy_mask = [&]() {
#pragma unroll
        for (int c = 0; c < V; c++) m[c] = !(k0 && c == 0);
    };
    auto x_slab = [&]() {
        S = slab_of(P, 0, i, xr);
        on = P.cp_on[S.f] && S.pos >= 1 && !zero_ij && !j0;
        q = ((int64_t)S.pos * yr + j) * zr + k;
        xy_mask();
    };
    auto y_slab = [&]() {
        S = slab_of(P, 1, j, yr);
        on = P.cp_on[S.f] && S.pos >= 1 && !zero_ij && !i0;
        q = ((int64_t)i * S.d + S.pos) * zr + k;
        xy_mask();
    };
    auto z_slab = [&](int f) {
        S.f = f;
        S.d = P.cp_d[f];
        S.pos = f == Z0 ? k : k - (zr - S.d);
        on = false;
#pragma unroll
        for (int c = 0; c < V; c++) {
            m[c] = P.cp_on[f] && !zero_ij && !i0 && !j0 && S.pos + c >= 1 && S.pos + c < S.d && !(kz0 && c == 0);
            on = on || m[c];
        }
        q = ((int64_t)i * yr + j) * S.d + S.pos;
    };
    auto load_psi = [&](bool vec) {
        if (!on) return;
        ldpsi<T, V>(p0, P.psie[S.f][0], q, vec, m, P.ipse);
        ldpsi<T, V>(p1, P.psie[S.f][1], q, vec, m, P.ipse);
    };
    if constexpr (FACE == 1) { x_slab(); load_psi(true); }
    if constexpr (FACE == 2) { y_slab(); load_psi(true); }
    if constexpr (FACE == 4) { z_slab(k < P.cp_d[Z0] ? Z0 : ZN); load_psi(V == 1 || S.d % V == 0); }
    // the poles' part of E^{n+1} (their state is read again for its recursion,
    // from L1: holding it would take 12 V registers; one cell a thread holds it)
    R pole[3][V], pk[3][2], qk[3][2];
    if constexpr (NPOLES > 0) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
#pragma unroll
            for (int c = 0; c < V; c++) pole[a][c] = 0;
            if (!(adem & (1u << a))) continue;
#pragma unroll
            for (int n = 0; n < NPOLES; n++) {
                R pv[V], qv[V];
                ldstate<R, V>(pv, P.pc[a][n], c0);
                ldstate<R, V>(qv, P.qc[a][n], c0);
                if constexpr (V == 1) { pk[a][n] = pv[0]; qk[a][n] = qv[0]; }
#pragma unroll
                for (int c = 0; c < V; c++) {
                    const auto &A = Tab<R>::ade(P, ade_of<R>(P, ONE ? g.cls : (int)((cw >> (8 * c)) & 0xff)));
                    pole[a][c] += fma1(A.qpe[n], qv[c], A.pe[n], pv[c]);
                }
            }
        }
    }
    const uint32_t stp = sr_step<T>(P);
    if constexpr (Stor<T>::scaled) {
        const float s = P.ihs;
#pragma unroll
        for (int c = 0; c < V; c++) {
            hx[c] *= s; hy[c] *= s; hz[c] *= s;
            hxj[c] *= s; hzj[c] *= s; hyi[c] *= s; hzi[c] *= s;
        }
        hxk1 *= s; hyk1 *= s;
    }
    // backward H differences, zero at the lower grid edges; they take the neighbours' places
    R dxk[V], dyk[V];
#pragma unroll
    for (int c = 0; c < V; c++) {
        dxk[c] = hx[c] - (c ? hx[c > 0 ? c - 1 : 0] : hxk1);
        dyk[c] = hy[c] - (c ? hy[c > 0 ? c - 1 : 0] : hyk1);
    }
    if (k0) dxk[0] = dyk[0] = 0;
#pragma unroll
    for (int c = 0; c < V; c++) {
        hxj[c] = j0 ? R(0) : hx[c] - hxj[c];
        hzj[c] = j0 ? R(0) : hz[c] - hzj[c];
        hyi[c] = i0 ? R(0) : hy[c] - hyi[c];
        hzi[c] = i0 ? R(0) : hz[c] - hzi[c];
    }
    R ikx = 1, iky = 1, ikzs[V] = {};
    if constexpr (EDGE) { ikx = Tab<R>::ld(P.ike[0], i); iky = Tab<R>::ld(P.ike[1], j); ldaxis<R, V>(ikzs, P.ike[2], k); }
    // new values before the CPML corrections: the ADE's, the ordinary update and the PEC rule elsewhere
    const unsigned cm[3] = {CF_ADE_X, CF_ADE_Y, CF_ADE_Z}, pm[3] = {CF_PEC_X, CF_PEC_Y, CF_PEC_Z};
    constexpr unsigned OWN = CF_ADE_BRANCH | CF_ADE_X | CF_ADE_Y | CF_ADE_Z, ODD = CF_PEC_X | CF_PEC_Y | CF_PEC_Z | CF_DESIGN;
    R ne[3][V];
    ecoef<R>(P, cl, cw & 0xff, i, j, k, C);
    // one class, no PEC rule, no design cell, no lower edge, and all or none of
    // the components dispersive: straight-line code
    const bool even = ONE ? !k0 : uni && !(C.fl & ODD) && !i0 && !j0 && !k0;
    const bool all_own = ADE && even && (C.fl & OWN) == OWN;
    auto curl_of = [&](int c, R (&cu)[3]) {
        const R ikz = EDGE ? ikzs[c] : R(1);
        cu[0] = hzj[c] * iky - dyk[c] * ikz;
        cu[1] = dxk[c] * ikz - hzi[c] * ikx;
        cu[2] = hyi[c] * ikx - hxj[c] * iky;
    };
    if (all_own) {
        const auto &A = Tab<R>::ade(P, C.ade);
        const R c0dx = A.c0dx, qe = A.qe, c2 = A.c2, c3 = A.c3;
#pragma unroll
        for (int c = 0; c < V; c++) {
            R cu[3];
            curl_of(c, cu);
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const R ep = w[a][c], e0 = eo[a][c];
                R v = DRUDE ? fma1(c0dx, cu[a], qe, qd[a][c]) : fma1(c0dx, cu[a], R(0), R(0));
                if constexpr (NPOLES > 0) v += pole[a][c];
                v += fma1(c2, ep, c3, e0);
                ne[a][c] = v;
                if constexpr (NPOLES == 0) w[a][c] = mad(R(2), e0, ep);   // what the Q recursion reads
            }
        }
    } else if (even && !(ADE && (C.fl & OWN))) {
#pragma unroll
        for (int c = 0; c < V; c++) {
            R cu[3];
            curl_of(c, cu);
#pragma unroll
            for (int a = 0; a < 3; a++) ne[a][c] = fma1(C.ca[a], eo[a][c], C.cb[a], cu[a]);
        }
    } else {
#pragma unroll
        for (int c = 0; c < V; c++) {
            if (c > 0 && !ONE && (!uni || (C.fl & CF_DESIGN))) ecoef<R>(P, cl, (cw >> (8 * c)) & 0xff, i, j, k + c, C);
            R cu[3];
            curl_of(c, cu);
            const bool kz = k0 && c == 0;
            const bool gd[3] = {!j0 && !kz, !i0 && !kz, !i0 && !j0};
            const bool branch = ADE && (flags & FB_ADE) && (C.fl & CF_ADE_BRANCH);
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const R e0 = eo[a][c];
                ne[a][c] = e0;
                if (branch && (C.fl & cm[a])) {
                    const auto &A = Tab<R>::ade(P, C.ade);
                    const R ep = w[a][c];
                    if (gd[a]) {
                        R v = DRUDE ? fma1(A.c0dx, cu[a], A.qe, qd[a][c]) : fma1(A.c0dx, cu[a], R(0), R(0));
                        if constexpr (NPOLES > 0) v += pole[a][c];
                        v += fma1(A.c2, ep, A.c3, e0);
                        ne[a][c] = v;
                    }
                    if constexpr (NPOLES == 0) w[a][c] = mad(R(2), e0, ep);
                } else {
                    if (gd[a]) ne[a][c] = fma1(C.ca[a], e0, C.cb[a], cu[a]);
                    if (C.fl & pm[a]) ne[a][c] = 0;
                }
            }
        }
    }
    R zdx[V];   // deferred z0 corrections of Ex
    const R dx = Tab<R>::dx(P), idx_ = R(1) / dx;
    const float pse = P.pse;
    // C holds the class of a one-class group; a mixed group looks each cell's up
    auto cell_class = [&](int c) { if (!uni) ecoef<R>(P, cl, (cw >> (8 * c)) & 0xff, i, j, k + c, C); };
#pragma unroll
    for (int c = 0; c < V; c++) zdx[c] = 0;
    // Each face: the first psi update of the ADE branch with its corrections
    // (yee.c:950-1057), then boundary_estep's with the corrections of the
    // components the ADE does not own; the two touch disjoint components.
    // What does not apply to a cell is switched off through its coefficients
    // (psi * 1 + 0 * difference, 0 * psi).
#pragma unroll 1
    for (int turn = (ANY && !P.axis_order ? 0 : 2); turn <= (ANY && !P.axis_order ? 1 : 2); turn++) {
        auto now = [&]() { return turn == 2 || (S.f & 1) == turn; };
        // x faces: psi[0] <- dhz_i (ey -= dx cb psi), psi[1] <- dhy_i (ez += dx cb psi)
        if constexpr ((FACE & 1) != 0) {
            if constexpr (ANY) { on = false; if (flags & FB_X) { x_slab(); on = on && now(); load_psi(true); } }
            if (on) {
                const int f = S.f;
                const R be = Tab<R>::ld(P.be[f], S.pos), ce = Tab<R>::ld(P.ce[f], S.pos);
#pragma unroll
                for (int c = 0; c < V; c++) {
                    if (!m[c]) continue;
                    cell_class(c);
                    if constexpr (ADE) {
                        const bool first = (C.fl & CF_ADE_BRANCH) && (f == XN || i > 1);
                        const R b1 = first ? be : R(1), c1 = first ? ce : R(0);
                        // the x0 corrections are scaled by cb == 0 (yee.c:577)
                        const R ky = first && f == XN && (C.fl & CF_ADE_Y) ? dx * C.cba : R(0);
                        const R kz = first && f == XN && (C.fl & CF_ADE_Z) ? dx * C.cba : R(0);
                        p0[c] = fma1(b1, p0[c], c1 * hzi[c], idx_);
                        p1[c] = fma1(b1, p1[c], c1 * hyi[c], idx_);
                        ne[1][c] = mad(-ky, p0[c], ne[1][c]);
                        ne[2][c] = mad(kz, p1[c], ne[2][c]);
                    }
                    p0[c] = fma1(be, p0[c], ce * hzi[c], idx_);
                    p1[c] = fma1(be, p1[c], ce * hyi[c], idx_);
                    ne[1][c] = mad(-(ADE && (C.fl & CF_ADE_Y) ? R(0) : dx * C.cb[1]), p0[c], ne[1][c]);
                    ne[2][c] = mad((ADE && (C.fl & CF_ADE_Z) ? R(0) : dx * C.cb[2]), p1[c], ne[2][c]);
                }
                stpsi<T, V>(P.psie[f][0], q, true, m, pse, p0, stp, 6 + 2 * f + 0);
                stpsi<T, V>(P.psie[f][1], q, true, m, pse, p1, stp, 6 + 2 * f + 1);
            }
        }
        // y faces: psi[0] <- dhz_j (ex += dx cb psi), psi[1] <- dhx_j (ez -= dx cb psi)
        if constexpr ((FACE & 2) != 0) {
            if constexpr (ANY) { on = false; if (flags & FB_Y) { y_slab(); on = on && now(); load_psi(true); } }
            if (on) {
                const int f = S.f;
                const R be = Tab<R>::ld(P.be[f], S.pos), ce = Tab<R>::ld(P.ce[f], S.pos);
#pragma unroll
                for (int c = 0; c < V; c++) {
                    if (!m[c]) continue;
                    cell_class(c);
                    if constexpr (ADE) {
                        const bool first = (C.fl & CF_ADE_BRANCH) && (f == YN || j > 1);
                        const R b1 = first ? be : R(1), c1 = first ? ce : R(0);
                        const R kx = first && (C.fl & CF_ADE_X) ? dx * C.cba : R(0);
                        const R kz = first && (C.fl & CF_ADE_Z) ? dx * C.cba : R(0);
                        p0[c] = fma1(b1, p0[c], c1 * hzj[c], idx_);
                        p1[c] = fma1(b1, p1[c], c1 * hxj[c], idx_);
                        ne[0][c] = mad(kx, p0[c], ne[0][c]);
                        ne[2][c] = mad(-kz, p1[c], ne[2][c]);
                    }
                    p0[c] = fma1(be, p0[c], ce * hzj[c], idx_);
                    p1[c] = fma1(be, p1[c], ce * hxj[c], idx_);
                    ne[0][c] = mad((ADE && (C.fl & CF_ADE_X) ? R(0) : dx * C.cb[0]), p0[c], ne[0][c]);
                    ne[2][c] = mad(-(ADE && (C.fl & CF_ADE_Z) ? R(0) : dx * C.cb[2]), p1[c], ne[2][c]);
                }
                stpsi<T, V>(P.psie[f][0], q, true, m, pse, p0, stp, 6 + 2 * f + 0);
                stpsi<T, V>(P.psie[f][1], q, true, m, pse, p1, stp, 6 + 2 * f + 1);
            }
        }
        // z faces: psi[1] <- dhx_k (ey += dx cb psi), psi[0] <- dhy_k (ex -= dx cb psi).
        // The first face gates the ex correction by the z component
        // (boundary.c:758-759): a cell whose ADE owns Ex but not Ez gets it after
        // its polarisation recursion.
        if constexpr ((FACE & 4) != 0) {
#pragma unroll 1
            for (int z = Z0; z <= (ANY ? ZN : Z0); z++) {
                if constexpr (ANY) {
                    if (!(flags & FB_Z)) break;
                    z_slab(z);
                    on = on && now();
                    load_psi(V == 1 || S.d % V == 0);
                }
                if (!on) continue;
                const int f = S.f;
                const bool vec = V == 1 || S.d % V == 0;
                R be[V], ce[V];
                ldtab<R, V>(be, P.be[f], S.pos, vec, m);
                ldtab<R, V>(ce, P.ce[f], S.pos, vec, m);
#pragma unroll
                for (int c = 0; c < V; c++) {
                    if (!m[c]) continue;
                    cell_class(c);
                    const R b = be[c], cc = ce[c];
                    if constexpr (ADE) {
                        const bool first = (C.fl & CF_ADE_BRANCH) && (f == ZN || k + c > 1);
                        const R b1 = first ? b : R(1), c1 = first ? cc : R(0);
                        const R ky = first && (C.fl & CF_ADE_Y) ? dx * C.cba : R(0);
                        const R kx = first && (C.fl & CF_ADE_X) ? dx * C.cba : R(0);
                        p1[c] = fma1(b1, p1[c], c1 * dxk[c], idx_);
                        p0[c] = fma1(b1, p0[c], c1 * dyk[c], idx_);
                        ne[1][c] = mad(ky, p1[c], ne[1][c]);
                        ne[0][c] = mad(-kx, p0[c], ne[0][c]);
                    }
                    p1[c] = fma1(b, p1[c], cc * dxk[c], idx_);
                    p0[c] = fma1(b, p0[c], cc * dyk[c], idx_);
                    ne[1][c] = mad((ADE && (C.fl & CF_ADE_Y) ? R(0) : dx * C.cb[1]), p1[c], ne[1][c]);
                    const R kx = ADE && (C.fl & (f == Z0 ? CF_ADE_Z : CF_ADE_X)) ? R(0) : dx * C.cb[0];
                    if (ADE && f == Z0 && (C.fl & CF_ADE_X)) zdx[c] = kx * p0[c];
                    else ne[0][c] = mad(-kx, p0[c], ne[0][c]);
                }
                stpsi<T, V>(P.psie[f][0], q, vec, m, pse, p0, stp, 6 + 2 * f + 0);
                stpsi<T, V>(P.psie[f][1], q, vec, m, pse, p1, stp, 6 + 2 * f + 1);
            }
        }
    }
    // polarisation recursions of the owned components, their PEC rule
    if (ADE && adem) {
        if constexpr (NPOLES > 0) {
#pragma unroll
            for (int a = 0; a < 3; a++) {
                if (!(adem & (1u << a))) continue;
#pragma unroll
                for (int n = 0; n < NPOLES; n++) {
                    R pv[V], qv[V];
                    if constexpr (V == 1) {
                        pv[0] = pk[a][n];
                        qv[0] = qk[a][n];
                    } else {
                        ldstate<R, V>(pv, P.pc[a][n], c0);
                        ldstate<R, V>(qv, P.qc[a][n], c0);
                    }
#pragma unroll
                    for (int c = 0; c < V; c++) {
                        if (!uni) ecoef<R>(P, cl, (cw >> (8 * c)) & 0xff, i, j, k + c, C);
                        if (!(C.fl & CF_ADE_BRANCH) || !(C.fl & cm[a])) continue;
                        const auto &A = Tab<R>::ade(P, C.ade);
                        const R pc = pv[c], qc = qv[c];
                        const R qn = mad(A.bp4[n], ne[a][c], mad(A.bp3[n], eo[a][c], mad(A.bp2[n], w[a][c], fma1(A.rp[n], pc, A.rq[n], qc))));
                        qv[c] = qn;
                        pv[c] = pc + qn;
                    }
                    ststate<R, V>(P.qc[a][n], c0, qv);
                    ststate<R, V>(P.pc[a][n], c0, pv);
                }
            }
        }
        if (!DRUDE && all_own) {
        } else if (all_own) {
            const auto &A = Tab<R>::ade(P, C.ade);
            const R ma0 = A.ma0, a2 = A.a2;
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int c = 0; c < V; c++)
                    qd[a][c] = fma1(ma0, qd[a][c], a2, (NPOLES == 0 ? w[a][c] : mad(R(2), eo[a][c], w[a][c])) + ne[a][c]);
        } else {
#pragma unroll
            for (int c = 0; c < V; c++) {
                if (!uni) ecoef<R>(P, cl, (cw >> (8 * c)) & 0xff, i, j, k + c, C);
                if (!(C.fl & CF_ADE_BRANCH)) continue;
                const auto &A = Tab<R>::ade(P, C.ade);
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    if (!(C.fl & cm[a])) continue;
                    if constexpr (DRUDE) qd[a][c] = fma1(A.ma0, qd[a][c], A.a2, (NPOLES == 0 ? w[a][c] : mad(R(2), eo[a][c], w[a][c])) + ne[a][c]);
                    if (C.fl & pm[a]) ne[a][c] = 0;
                }
                ne[0][c] -= zdx[c];
            }
        }
#pragma unroll
        for (int a = 0; a < 3; a++)
            if (DRUDE && (adem & (1u << a))) ststate<R, V>(P.q[a], c0, qd[a]);
    }
    // the lower E planes boundary_estep zeroes (boundary.c:522-690)
#pragma unroll
    for (int c = 0; c < V; c++)
        if (zero_ij || (kz0 && c == 0)) ne[0][c] = ne[1][c] = ne[2][c] = 0;
    if ((flags & FB_TSF) && tsf_hit<V>(P, i, j, k)) tsf_add_e<R, V>(P, i, j, k, ne[0], ne[1], ne[2]);
    stv<T, V>(P.fout[0], c0, ne[0], 1.f, stp, 0);
    stv<T, V>(P.fout[1], c0, ne[1], 1.f, stp, 1);
    stv<T, V>(P.fout[2], c0, ne[2], 1.f, stp, 2);
}

// ------------------------------------------------------------ kernels

template <class T, int V>
__device__ __forceinline__ void flat_h(const DevPlan &P, const FlatCell &g)
{
    const int fl = g.flags;
    if ((fl & (FB_EDGE | FB_ONE)) == FB_ONE) {
        flat_h_group<T, V, 0, true>(P, g);
    } else if ((fl & FB_SPEC) && g.i > 0 && g.j > 0 && g.i < P.xr - 1 && g.j < P.yr - 1) {   // (edge planes and rows: general)
        if (fl & FB_X) flat_h_group<T, V, 1, true>(P, g);
        else if (fl & FB_Y) flat_h_group<T, V, 2, true>(P, g);
        else flat_h_group<T, V, 4, true>(P, g);
    } else if (fl & FB_EDGE) {
        flat_h_group<T, V, 7, false>(P, g);
    } else {
        flat_h_group<T, V, 0, false>(P, g);
    }
}

template <bool ADE, int NPOLES, class T, int V>
__device__ __forceinline__ void flat_e(const DevPlan &P, const FlatCell &g)
{
    const int fl = g.flags;
    if ((fl & (FB_EDGE | FB_ONE)) == FB_ONE) {
        flat_e_group<ADE, NPOLES, T, V, 0, true>(P, g);
    } else if ((fl & FB_SPEC) && g.i > 0 && g.j > 0) {
        if (fl & FB_X) flat_e_group<ADE, NPOLES, T, V, 1, true>(P, g);
        else if (fl & FB_Y) flat_e_group<ADE, NPOLES, T, V, 2, true>(P, g);
        else flat_e_group<ADE, NPOLES, T, V, 4, true>(P, g);
    } else if (fl & FB_EDGE) {
        flat_e_group<ADE, NPOLES, T, V, 7, false>(P, g);
    } else {
        flat_e_group<ADE, NPOLES, T, V, 0, false>(P, g);
    }
}

// Blocks ahead of which a block's descriptor is fetched into L2: about those in
// flight (a descriptor is read once a launch and would come from DRAM; 512^3
// without the bulk kernel: 3.13 -> 3.01 ms a step).
constexpr int H_AHEAD = 1536, E_AHEAD = 1024;

// Resident blocks asked for.  H: 24 warps an SM at 80 registers (20 at 88:
// 256^3 rough surface 405 -> 393 us a step).  E: 16 warps at 128; 20 warps spill
// the dispersive variant (403 us).  Single cells: 40 and 28 warps.  What still
// spills (bytes a thread, stores / loads): E of groups with two poles 48 / 112, H
// of groups 32 / 56, BF16 H 156 / 212; the batch forms, which read the plan
// through a pointer, 140 / 428 with two poles; FP64 single cells, whose bounds are
// FP32's, up to 1664 / 1696 with two poles (96 x 96 x 97, metal in half of it: 99
// us a step, 170 with the kernels of one cell a thread before).
template <int V>
constexpr int H_BLOCKS = V == 1 ? 10 : 6;
template <int V>
constexpr int E_BLOCKS = V == 1 ? 7 : 4;

template <class T, int V>
__global__ void __launch_bounds__(FLAT_NT, H_BLOCKS<V>) flat_h_kernel(const __grid_constant__ DevPlan P, const FlatBlock *blocks)
{
    e_may_start();
    FlatCell g;
    if (flat_cell<V>(blocks, blockIdx.x, H_AHEAD, g)) flat_h<T, V>(P, g);
}

template <class T, int V>
__global__ void __launch_bounds__(FLAT_NT, H_BLOCKS<V>) flat_h_batch(const DevPlan *plans, const FlatBlock *blocks)
{
    e_may_start();
    FlatCell g;
    if (flat_cell<V>(blocks, blockIdx.x, H_AHEAD, g)) flat_h<T, V>(plans[g.inst], g);
}

// E walks the blocks backwards: what H touched last is still in L2
template <bool ADE, int NPOLES, class T, int V>
__global__ void __launch_bounds__(FLAT_NT, E_BLOCKS<V>) flat_e_kernel(const __grid_constant__ DevPlan P, const FlatBlock *blocks)
{
    FlatCell g;
    if (flat_cell<V>(blocks, gridDim.x - 1 - blockIdx.x, -E_AHEAD, g)) flat_e<ADE, NPOLES, T, V>(P, g);
}

template <bool ADE, int NPOLES, class T, int V>
__global__ void __launch_bounds__(FLAT_NT, E_BLOCKS<V>) flat_e_batch(const DevPlan *plans, const FlatBlock *blocks)
{
    FlatCell g;
    if (flat_cell<V>(blocks, gridDim.x - 1 - blockIdx.x, -E_AHEAD, g)) flat_e<ADE, NPOLES, T, V>(plans[g.inst], g);
}

template <class T, int V>
cudaError_t flat_h_v(const DevPlan *p, const DevPlan *plans, const FlatList &l, cudaStream_t st)
{
    if (plans) flat_h_batch<T, V><<<l.n, FLAT_NT, 0, st>>>(plans, l.blocks);
    else flat_h_kernel<T, V><<<l.n, FLAT_NT, 0, st>>>(*p, l.blocks);
    return cudaGetLastError();
}

template <bool ADE, int NPOLES, class T, int V>
void flat_e_v(const DevPlan *p, const DevPlan *plans, const FlatList &l, bool beside_h, cudaStream_t st)
{
    if (plans) {
        flat_e_batch<ADE, NPOLES, T, V><<<l.n, FLAT_NT, 0, st>>>(plans, l.blocks);
        return;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at = {};
    cfg.gridDim = dim3(l.n);
    cfg.blockDim = dim3(FLAT_NT);
    cfg.stream = st;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = beside_h ? 1 : 0;
    cudaLaunchKernelEx(&cfg, flat_e_kernel<ADE, NPOLES, T, V>, *p, l.blocks);
}

template <class T, int V>
cudaError_t flat_e_v(const DevPlan *p, const DevPlan *plans, const FlatList &l, bool ade, int npoles, bool beside_h, cudaStream_t st)
{
    if (!ade) flat_e_v<false, 0, T, V>(p, plans, l, beside_h, st);
    else if (npoles == 0) flat_e_v<true, 0, T, V>(p, plans, l, beside_h, st);
    else if (npoles == 1) flat_e_v<true, 1, T, V>(p, plans, l, beside_h, st);
    else flat_e_v<true, 2, T, V>(p, plans, l, beside_h, st);
    return cudaGetLastError();
}

}  // namespace

// cells per thread when the k rows are whole vectors
template <class T>
constexpr int FLAT_VEC = sizeof(T) == 8 ? 2 : 4;

template <class T>
cudaError_t flat_h_t(const DevPlan *p, const DevPlan *plans, const FlatList &l, int width, cudaStream_t st)
{
    return width > 1 ? flat_h_v<T, FLAT_VEC<T>>(p, plans, l, st) : flat_h_v<T, 1>(p, plans, l, st);
}

template <class T>
cudaError_t flat_e_t(const DevPlan *p, const DevPlan *plans, const FlatList &l, int width, bool ade, int npoles, bool beside_h, cudaStream_t st)
{
    return width > 1 ? flat_e_v<T, FLAT_VEC<T>>(p, plans, l, ade, npoles, beside_h, st) : flat_e_v<T, 1>(p, plans, l, ade, npoles, beside_h, st);
}

#define FLAT_INSTANCE(T)                                                                                        \
    template cudaError_t flat_h_t<T>(const DevPlan *, const DevPlan *, const FlatList &, int, cudaStream_t);    \
    template cudaError_t flat_e_t<T>(const DevPlan *, const DevPlan *, const FlatList &, int, bool, int, bool, cudaStream_t);
