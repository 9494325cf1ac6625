// resident.cuh — time steps of a grid that stays on the SMs.
//
// The split half-steps (yee.cuh) read every field value from L2 or HBM and
// write it back once per half-step, and every step waits for two rounds of
// launches with their forks and joins. A grid whose state fits the registers
// and shared memory of the device needs neither: one cooperative launch loads
// the state once, advances it by a chunk of steps, and stores it once.
//
// Blocks. CTA b owns full x rows of a band of y rows times a slab of z planes
// (resident.cpp cuts the grid so that the slowest block is as fast as it can
// be). A thread owns a run of up to L planes of one column (x, y), with all
// six fields of its cells in registers. What the neighbouring columns read is
// in shared memory too, at [component][plane of the run][thread]: with L and
// the thread count known at compile time every access is a per-thread base
// and a constant offset, so a cell costs its arithmetic, four loads and three
// stores. (Holding the fields in shared memory alone, with run-time strides,
// measured 9.0 us against 5.6 us per step on a 40 x 40 x 200 FP32 cell; the
// split half-steps take 13.8 us.) CPML psi of z is in shared memory, psi of x
// and y and the recursive-convolution psi (18 values per cell for three poles)
// in global
// memory; the latter's update reads only the block's own E and runs before
// the block waits for its neighbours.
//
// Exchange. An E update needs H of the y-1 and z-1 blocks, an H update E of
// the y+1 and z+1 blocks (fdtd_core.cpp:363-969; both wrap). The thread that
// owns a cell at such a face stores each value, together with the number of
// the half-step, as one 64-bit word into the neighbour's inbox (FP64: two
// words of 32 data bits each), and the one thread there that needs it reads
// the word until it carries the number it waits for: data and flag arrive
// together, so there is no fence and no second round trip, and threads inside
// the block do not wait at all. One inbox slot per value is enough: a value
// is overwritten only by its owner's next update of that field, which needs
// the neighbour's next value at the same place, which the neighbour computed
// after it had read the slot. All CTAs are resident (cooperative launch) and
// a wait only looks back one half-step, so every wait ends; each is bounded
// all the same, and one that runs out raises the device error flag, after
// which every CTA leaves at its next barrier.
//
// The arithmetic per cell is that of the split kernels in the same order:
// FP64 fields are bit-identical.
//
// Bound: per half-step the slowest block's issue slots (about 12 cycles per
// warp and plane in FP32, 20 in FP64, twice that in a z-CPML slab) and one
// inbox round trip of 1000 to 1300 cycles. Measured per step, resident against
// split: 12 x 10 x 90 FP64 4.3 / 13.4 us, 48 x 48 x 128 FP64 7.5 / 16.2,
// 40 x 40 x 200 FP32 5.6 / 13.8, 64 x 64 x 128 FP32 with two 61-wavelength flux
// planes 8.3 / 15.1.
#pragma once

#include <cuda_runtime.h>

#include "kernels.hpp"
#include "yee.cuh"

namespace aefdtd {

// Inbox words: FP32 one 64-bit word {data, number}; FP64 two such words with 32
// data bits each. Every word is read and written as one 64-bit element, which
// is atomic; a pair moves in one instruction.
template <typename T> struct InboxWords { unsigned long long w[sizeof(T) / 4]; };
__device__ __forceinline__ void inbox_read(const unsigned long long *p, InboxWords<float> &x) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x.w[0]) : "l"(p) : "memory");
}
__device__ __forceinline__ void inbox_read(const unsigned long long *p, InboxWords<double> &x) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x.w[0]), "=l"(x.w[1]) : "l"(p) : "memory");
}
// No memory clobber: nothing else of this launch reads the word, and the cell
// loops must stay free to move around it.
__device__ __forceinline__ void inbox_put(unsigned long long *p, float v, unsigned seq) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)seq << 32) | __float_as_uint(v)));
}
__device__ __forceinline__ void inbox_put(unsigned long long *p, double v, unsigned seq) {
    const unsigned long long n = (unsigned long long)seq << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(n | (unsigned)__double2loint(v)),
                 "l"(n | (unsigned)__double2hiint(v)));
}
// Whether the value numbered seq has arrived (then in v).
__device__ __forceinline__ bool inbox_take(const InboxWords<float> &x, float &v, unsigned seq) {
    v = __uint_as_float((unsigned)x.w[0]);
    return (unsigned)(x.w[0] >> 32) == seq;
}
__device__ __forceinline__ bool inbox_take(const InboxWords<double> &x, double &v, unsigned seq) {
    v = __hiloint2double((int)(unsigned)x.w[1], (int)(unsigned)x.w[0]);
    return (unsigned)(x.w[0] >> 32) == seq && (unsigned)(x.w[1] >> 32) == seq;
}

// Coefficients of material m: four or six consecutive values of one entry.
template <typename T> struct Coef4 { T C1, C2x, C2y, C2z; };
__device__ __forceinline__ Coef4<float> coef4(const MatCoef<float> *c) {
    const float2 a = *reinterpret_cast<const float2 *>(&c->C1), b = *reinterpret_cast<const float2 *>(&c->C2y);
    return {a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ Coef4<double> coef4(const MatCoef<double> *c) {
    const double2 a = *reinterpret_cast<const double2 *>(&c->C1), b = *reinterpret_cast<const double2 *>(&c->C2y);
    return {a.x, a.y, b.x, b.y};
}

// Shared memory of a CTA, in values of T from the start: E [3][L][threads],
// H [3][L][threads], z-CPML psi [E 0, E 1, H 0, H 1][npsi][threads].
extern __shared__ __align__(16) unsigned char res_sm[];
template <typename T, int L, int NT> __device__ __forceinline__ T *res_e(int c) { return reinterpret_cast<T *>(res_sm) + c * L * NT; }
template <typename T, int L, int NT> __device__ __forceinline__ T *res_h(int c) { return reinterpret_cast<T *>(res_sm) + (3 + c) * L * NT; }
// psi q of the thread's first plane, its planes NT apart; only blocks with CPML
// planes need one slot per plane (npsi of them), all others keep zeros
template <typename T, int L, int NT> __device__ __forceinline__ T *res_pz(int npsi, int q) {
    return reinterpret_cast<T *>(res_sm) + (6 * L + q * npsi) * NT + threadIdx.x;
}

// The injection plane alone (kFMisc adds the oscillator boxes).
constexpr unsigned kFInject = 16;

// What a thread knows about its run of cells for the whole launch.
template <typename T, int L> struct ResThread {
    T e0[L], e1[L], e2[L], h0[L], h1[L], h2[L];
    int t, i, J, K, nk;                 // thread; column; first plane and number of planes
    int xm, xp;                         // threads of the neighbouring columns along x
    bool mixed;                         // more than one material in the run
    Coef4<T> v;                         // the run's coefficients otherwise
    T C4;
    unsigned ids[(L + 3) / 4];          // material ids, a byte each
};
// z-CPML values of one of the block's planes for E and for H. Outside a side's
// range b keeps psi (which is zero there) and c adds nothing, so the updates
// need no branch.
template <typename T> struct alignas(16) ResZ { T ik, b, c, pad; };
template <typename T, int L> __device__ __forceinline__ int res_id(const ResThread<T, L> &s, int k) {
    return (s.ids[k >> 2] >> (8 * (k & 3))) & 0xff;
}

// ---- one cell
// E of one cell at plane K (run plane k), feature set F: e the cell's E, h its
// H, hxj, hzj the row below, hyi, hzi the column before, hxm, hym the plane
// below; writes the new E to n.
template <typename T, int L, int NT, unsigned F>
__device__ __forceinline__ void res_cell_e(const StepArgs<T, uint8_t> &a, const ResBlock &B, const Coef4<T> v, int m, int i,
                                           int J, int K, int k, int t, int q, const T e[3], const T h[3], T hxj, T hzj,
                                           T hyi, T hzi, T hxm, T hym, T n[3]) {
    T ikx = 1, iky = 1, ikz = 1;
    if constexpr ((F & kFPmlXY) != 0) { ikx = __ldg(a.ikx + i); iky = __ldg(a.iky + J); }
    if constexpr ((F & kFPmlZ) != 0) ikz = __ldg(a.ikz + K);
    const T dHz_y = h[2] - hzj, dHy_z = h[1] - hym, dHx_z = h[0] - hxm, dHz_x = h[2] - hzi, dHy_x = h[1] - hyi, dHx_y = h[0] - hxj;
    T nex = (v.C1 * e[0] + (v.C2y * iky) * dHz_y) - (v.C2z * ikz) * dHy_z;
    T ney = (v.C1 * e[1] + (v.C2z * ikz) * dHx_z) - (v.C2x * ikx) * dHz_x;
    T nez = (v.C1 * e[2] + (v.C2x * ikx) * dHy_x) - (v.C2y * iky) * dHx_y;
    const MatCoef<T> *coef = reinterpret_cast<const MatCoef<T> *>(res_sm + B.o_coef) + m;
    if constexpr ((F & kFDisp) != 0) {
        if (B.disp_n > 0) {
            const int r = reinterpret_cast<const uint16_t *>(res_sm + B.o_rank)[k * NT + t];
            if (r != kResNoRank) {
                const T C3 = coef->C3;
                const T *sum = reinterpret_cast<const T *>(res_sm + B.o_sum) + 3 * r;
                nex += C3 * sum[0];
                ney += C3 * sum[1];
                nez += C3 * sum[2];
            }
        }
    }
    if constexpr ((F & (kFPmlXY | kFPmlZ)) != 0) {
        const T C4 = coef->C4;
        // E-side ranges [1, pml_m) and [N - pml_p + 1, N) (fdtd_pml.cpp:518,527,547,559)
        const bool ze = a.pz && ((K >= 1 && K < a.pml_zm) || (K >= a.Nz - a.pml_zp + 1));
        bool xe = false, ye = false;
        T bx = 0, cx = 0, by = 0, cy = 0, bz = 0, cz = 0;
        long long ox = 0, oy = 0;
        T qx0 = 0, qx1 = 0, qy0 = 0, qy1 = 0, qz0 = 0, qz1 = 0;
        if constexpr ((F & kFPmlXY) != 0) {
            xe = a.px && ((i >= 1 && i < a.pml_xm) || (i >= a.Nx - a.pml_xp + 1));
            ye = a.py && ((J >= 1 && J < a.pml_ym) || (J >= a.Ny - a.pml_yp + 1));
            if (xe) {
                ox = ((i < a.pml_xm) ? i : i - (a.Nx - a.pml_xp) + a.pml_xm) + (long long)(a.pml_xm + a.pml_xp) * (J + (long long)a.Ny * K);
                bx = __ldg(a.bx + i); cx = __ldg(a.cx + i); qx0 = a.psi_x0[ox]; qx1 = a.psi_x1[ox];
            }
            if (ye) {
                oy = i + (long long)a.Nx * (((J < a.pml_ym) ? J : J - (a.Ny - a.pml_yp) + a.pml_ym) + (long long)(a.pml_ym + a.pml_yp) * K);
                by = __ldg(a.by + J); cy = __ldg(a.cy + J); qy0 = a.psi_y0[oy]; qy1 = a.psi_y1[oy];
            }
        }
        T *p0 = res_pz<T, L, NT>(B.npsi, 0) + k * NT, *p1 = res_pz<T, L, NT>(B.npsi, 1) + k * NT;
        if (ze) { bz = __ldg(a.bz + K); cz = __ldg(a.cz + K); qz0 = *p0; qz1 = *p1; }
        // Ex: y block, then z block
        if constexpr ((F & kFPmlXY) != 0) {
            if (ye) { const T ps = cpml_rec(by, qy0, cy, dHz_y); a.psi_y0[oy] = ps; nex += C4 * ps; }
            if (a.py && J == 0) nex = 0;
        }
        if (ze) { const T ps = cpml_rec(bz, qz0, cz, dHy_z); *p0 = ps; nex -= C4 * ps; }
        if (a.pz && K == 0) nex = 0;
        // Ey: x block, then z block
        if constexpr ((F & kFPmlXY) != 0) {
            if (xe) { const T ps = cpml_rec(bx, qx0, cx, dHz_x); a.psi_x0[ox] = ps; ney -= C4 * ps; }
            if (a.px && i == 0) ney = 0;
        }
        if (ze) { const T ps = cpml_rec(bz, qz1, cz, dHx_z); *p1 = ps; ney += C4 * ps; }
        if (a.pz && K == 0) ney = 0;
        // Ez: x block, then y block
        if constexpr ((F & kFPmlXY) != 0) {
            if (xe) { const T ps = cpml_rec(bx, qx1, cx, dHy_x); a.psi_x1[ox] = ps; nez += C4 * ps; }
            if (a.px && i == 0) nez = 0;
            if (ye) { const T ps = cpml_rec(by, qy1, cy, dHx_y); a.psi_y1[oy] = ps; nez -= C4 * ps; }
            if (a.py && J == 0) nez = 0;
        }
    }
    if constexpr ((F & (kFMisc | kFInject)) != 0) {
        if (K == a.kinj) {
            nex = nex - (T)a.sc[q].inj_eA;
            ney = ney + (T)a.sc[q].inj_eB;
        }
    }
    if constexpr ((F & kFMisc) != 0) {
        for (int u = 0; u < a.nsrc; ++u) {
            const int *b = a.src_box[u];
            if (i >= b[0] && i < b[1] && J >= b[2] && J < b[3] && K >= b[4] && K < b[5]) {
                const T sv = (T)a.sc[q].src[u];
                if (a.src_comp[u] == 0) nex += sv;
                else if (a.src_comp[u] == 1) ney += sv;
                else nez += sv;
            }
        }
    }
    n[0] = nex; n[1] = ney; n[2] = nez;
}

// H of one cell: exj, ezj the row above, eyi, ezi the column after, exk, eyk
// the plane above.
template <typename T, int L, int NT, unsigned F>
__device__ __forceinline__ void res_cell_h(const StepArgs<T, uint8_t> &a, const ResBlock &B, int i, int J, int K, int k, int t, int q, const T e[3],
                                           const T h[3], T exj, T ezj, T eyi, T ezi, T exk, T eyk, T n[3]) {
    T ax = a.dtdmx, ay = a.dtdmy, az = a.dtdmz;
    if constexpr ((F & kFPmlXY) != 0) { ax = a.dtdmx * __ldg(a.ikx + i); ay = a.dtdmy * __ldg(a.iky + J); }
    if constexpr ((F & kFPmlZ) != 0) az = a.dtdmz * __ldg(a.ikz + K);
    const T dEy_z = eyk - e[1], dEz_y = ezj - e[2], dEz_x = ezi - e[2], dEx_z = exk - e[0], dEx_y = exj - e[0], dEy_x = eyi - e[1];
    T nhx = h[0] + (az * dEy_z - ay * dEz_y);
    T nhy = h[1] + (ax * dEz_x - az * dEx_z);
    T nhz = h[2] + (ay * dEx_y - ax * dEy_x);
    if constexpr ((F & (kFPmlXY | kFPmlZ)) != 0) {
        // H-side ranges [0, pml_m) and [N - pml_p, N - 1) (fdtd_pml.cpp:750,756,775,784)
        const bool zh = a.pz && ((K < a.pml_zm) || (K >= a.Nz - a.pml_zp && K < a.Nz - 1));
        bool xh = false, yh = false;
        T bx = 0, cx = 0, by = 0, cy = 0, bz = 0, cz = 0;
        long long ox = 0, oy = 0;
        T qx0 = 0, qx1 = 0, qy0 = 0, qy1 = 0, qz0 = 0, qz1 = 0;
        if constexpr ((F & kFPmlXY) != 0) {
            xh = a.px && ((i < a.pml_xm) || (i >= a.Nx - a.pml_xp && i < a.Nx - 1));
            yh = a.py && ((J < a.pml_ym) || (J >= a.Ny - a.pml_yp && J < a.Ny - 1));
            if (xh) {
                ox = ((i < a.pml_xm) ? i : i - (a.Nx - a.pml_xp) + a.pml_xm) + (long long)(a.pml_xm + a.pml_xp) * (J + (long long)a.Ny * K);
                bx = __ldg(a.bx + i); cx = __ldg(a.cx + i); qx0 = a.psi_x0[ox]; qx1 = a.psi_x1[ox];
            }
            if (yh) {
                oy = i + (long long)a.Nx * (((J < a.pml_ym) ? J : J - (a.Ny - a.pml_yp) + a.pml_ym) + (long long)(a.pml_ym + a.pml_yp) * K);
                by = __ldg(a.by + J); cy = __ldg(a.cy + J); qy0 = a.psi_y0[oy]; qy1 = a.psi_y1[oy];
            }
        }
        T *p0 = res_pz<T, L, NT>(B.npsi, 2) + k * NT, *p1 = res_pz<T, L, NT>(B.npsi, 3) + k * NT;
        if (zh) { bz = __ldg(a.bz + K); cz = __ldg(a.cz + K); qz0 = *p0; qz1 = *p1; }
        // Hx: y block, then z block
        if constexpr ((F & kFPmlXY) != 0) {
            if (yh) { const T ps = cpml_rec(by, qy0, cy, dEz_y); a.psi_y0[oy] = ps; nhx -= a.dtm * ps; }
            if (a.py && J == a.Ny - 1) nhx = 0;
        }
        if (zh) { const T ps = cpml_rec(bz, qz0, cz, dEy_z); *p0 = ps; nhx += a.dtm * ps; }
        if (a.pz && K == a.Nz - 1) nhx = 0;
        // Hy: x block, then z block
        if constexpr ((F & kFPmlXY) != 0) {
            if (xh) { const T ps = cpml_rec(bx, qx0, cx, dEz_x); a.psi_x0[ox] = ps; nhy += a.dtm * ps; }
            if (a.px && i == a.Nx - 1) nhy = 0;
        }
        if (zh) { const T ps = cpml_rec(bz, qz1, cz, dEx_z); *p1 = ps; nhy -= a.dtm * ps; }
        if (a.pz && K == a.Nz - 1) nhy = 0;
        // Hz: x block, then y block
        if constexpr ((F & kFPmlXY) != 0) {
            if (xh) { const T ps = cpml_rec(bx, qx1, cx, dEy_x); a.psi_x1[ox] = ps; nhz -= a.dtm * ps; }
            if (a.px && i == a.Nx - 1) nhz = 0;
            if (yh) { const T ps = cpml_rec(by, qy1, cy, dEx_y); a.psi_y1[oy] = ps; nhz += a.dtm * ps; }
            if (a.py && J == a.Ny - 1) nhz = 0;
        }
    }
    if constexpr ((F & (kFMisc | kFInject)) != 0) {
        if (K == a.kinj) {
            nhx = nhx + (T)a.sc[q].inj_hA;
            nhy = nhy - (T)a.sc[q].inj_hB;
        }
    }
    n[0] = nhx; n[1] = nhy; n[2] = nhz;
}

// ---- one run
// Where a run finds the row next to it: component 0 at element p of shared
// memory, the other at p + d, planes sj apart, in the block's own arrays or in
// the halo; and the plane next to it: elements z and z + dz. Two records per
// thread (for E, for H), computed once per launch.
struct alignas(16) ResNext {
    int p, sj_d, z, dz;   // sj_d: sj | d << 12
};
template <typename T, int L, int NT, int HALF> __device__ __forceinline__ ResNext res_next(int nx, const ResBlock &B, int t) {
    const int ncol = nx * B.by, last = B.nseg - 1, run = t / ncol;
    // threads past the last run read what the first column reads
    const bool live = run <= last;
    const int seg = live ? run : 0, col = live ? t - run * ncol : 0, j = col / nx, i = col - j * nx, kb = seg * L;
    const int base = HALF ? 0 : 3 * L * NT, halo = B.o_halo / (int)sizeof(T), own = live ? t : 0;
    ResNext r;
    const bool edge = HALF ? j == B.by - 1 : j == 0;
    if (!edge || B.self_y) {
        r.p = base + own + (HALF ? (edge ? -j * nx : nx) : (edge ? (B.by - 1) * nx : -nx));
        r.sj_d = NT | (2 * L * NT) << 12;
    } else {
        r.p = halo + kb * nx + i;
        r.sj_d = nx | (nx * B.bz) << 12;
    }
    const bool end = HALF ? seg == last : seg == 0;
    if (!end || B.self_z) {
        const int k = HALF ? 0 : end ? B.bz - last * L - 1 : L - 1;
        r.z = base + k * NT + own + (HALF ? (end ? -last * ncol : ncol) : (end ? last * ncol : -ncol));
        r.dz = L * NT;
    } else {
        r.z = halo + 2 * nx * B.bz + col;
        r.dz = ncol;
    }
    return r;
}
template <typename T> __device__ __forceinline__ const T *res_at(int element) { return reinterpret_cast<const T *>(res_sm) + element; }
template <int HALF> __device__ __forceinline__ ResNext res_record(const ResBlock &B, int nt) {
    return reinterpret_cast<const ResNext *>(res_sm + B.o_next)[HALF * nt + threadIdx.x];
}

// The run in registers, fully unrolled: any of pole sums, z CPML and the
// injection plane; Mixed: the run holds several materials. Shared-memory
// reads of a few planes at a time are issued together, psi is stored after
// each such group and the fields after the whole run, so that no read waits
// behind a store it cannot be told apart from. Planes past nk compute values
// that nobody reads.
template <typename T, int L, int NT, unsigned F, bool Mixed>
__device__ __forceinline__ void res_run_e(const ResArgs<T> &A, const ResBlock &B, ResThread<T, L> &s, int q) {
    constexpr int C = sizeof(T) == 8 ? 2 : 4;
    const ResNext next = res_record<0>(B, NT);
    const T *row = res_at<T>(next.p), *plane = res_at<T>(next.z);
    const int sj = next.sj_d & 0xfff, dj = next.sj_d >> 12, npsi = B.npsi;
    const MatCoef<T> *coef = reinterpret_cast<const MatCoef<T> *>(res_sm + B.o_coef);
    const ResZ<T> *zt = reinterpret_cast<const ResZ<T> *>(res_sm + B.o_z) + (s.K - B.k0);
    // the run's plane that takes the injection, and its conducting plane
    const int kin = A.e.kinj - s.K, kpec = A.e.pz ? -s.K : -1;
    T injA = 0, injB = 0;
    if ((F & kFInject) != 0 && A.e.kinj >= 0) {
        const T *inj = reinterpret_cast<const T *>(res_sm + B.o_inject) + 4 * q;
        injA = inj[0];
        injB = inj[1];
    }
    T hxm = plane[0], hym = plane[next.dz];
#pragma unroll
    for (int k0 = 0; k0 < L; k0 += C) {
        if (k0 > 0 && k0 >= s.nk) break;
        T yx[C], yz[C], x1[C], x2[C], p0[C], p1[C];
        Coef4<T> v[C];
        ResZ<T> z[C];
#pragma unroll
        for (int u = 0; u < C; ++u) {
            const int k = k0 + u;
            if (k >= L) continue;
            yx[u] = row[k * sj];
            yz[u] = row[dj + k * sj];
            x1[u] = res_h<T, L, NT>(1)[k * NT + s.xm];
            x2[u] = res_h<T, L, NT>(2)[k * NT + s.xm];
            if constexpr (Mixed) v[u] = coef4(coef + res_id(s, k));
            if constexpr ((F & kFPmlZ) != 0) {
                z[u] = zt[k];
                p0[u] = res_pz<T, L, NT>(npsi, 0)[min(k, npsi - 1) * NT];
                p1[u] = res_pz<T, L, NT>(npsi, 1)[min(k, npsi - 1) * NT];
            }
        }
#pragma unroll
        for (int u = 0; u < C; ++u) {
            const int k = k0 + u;
            if (k >= L) continue;
            const Coef4<T> c = Mixed ? v[u] : s.v;
            const T hx = s.h0[k], hy = s.h1[k], hz = s.h2[k];
            const T dHz_y = hz - yz[u], dHy_z = hy - hym, dHx_z = hx - hxm, dHz_x = hz - x2[u], dHy_x = hy - x1[u], dHx_y = hx - yx[u];
            T ikz = 1;
            if constexpr ((F & kFPmlZ) != 0) ikz = z[u].ik;
            T nex = (c.C1 * s.e0[k] + c.C2y * dHz_y) - (c.C2z * ikz) * dHy_z;
            T ney = (c.C1 * s.e1[k] + (c.C2z * ikz) * dHx_z) - c.C2x * dHz_x;
            T nez = (c.C1 * s.e2[k] + c.C2x * dHy_x) - c.C2y * dHx_y;
            if constexpr ((F & kFDisp) != 0) {
                const int rank = reinterpret_cast<const uint16_t *>(res_sm + B.o_rank)[k * NT + s.t];
                if (rank != kResNoRank) {
                    const T C3 = coef[res_id(s, k)].C3;
                    const T *sum = reinterpret_cast<const T *>(res_sm + B.o_sum) + 3 * rank;
                    nex += C3 * sum[0];
                    ney += C3 * sum[1];
                    nez += C3 * sum[2];
                }
            }
            if constexpr ((F & kFPmlZ) != 0) {
                const T C4 = Mixed ? coef[res_id(s, k)].C4 : s.C4;
                p0[u] = cpml_rec(z[u].b, p0[u], z[u].c, dHy_z);
                nex -= C4 * p0[u];
                p1[u] = cpml_rec(z[u].b, p1[u], z[u].c, dHx_z);
                ney += C4 * p1[u];
                nex = k == kpec ? T(0) : nex;
                ney = k == kpec ? T(0) : ney;
            }
            if constexpr ((F & kFInject) != 0) {
                nex = k == kin ? nex - injA : nex;
                ney = k == kin ? ney + injB : ney;
            }
            s.e0[k] = nex; s.e1[k] = ney; s.e2[k] = nez;
            hxm = hx;
            hym = hy;
        }
        if constexpr ((F & kFPmlZ) != 0) {
#pragma unroll
            for (int u = 0; u < C; ++u)
                if (k0 + u < L && k0 + u < min(s.nk, npsi)) {
                    res_pz<T, L, NT>(npsi, 0)[(k0 + u) * NT] = p0[u];
                    res_pz<T, L, NT>(npsi, 1)[(k0 + u) * NT] = p1[u];
                }
        }
    }
#pragma unroll
    for (int k = 0; k < L; ++k) {
        res_e<T, L, NT>(0)[k * NT + s.t] = s.e0[k];
        res_e<T, L, NT>(1)[k * NT + s.t] = s.e1[k];
        res_e<T, L, NT>(2)[k * NT + s.t] = s.e2[k];
    }
}
template <typename T, int L, int NT, unsigned F>
__device__ __forceinline__ void res_run_h(const ResArgs<T> &A, const ResBlock &B, ResThread<T, L> &s, int q) {
    constexpr int C = sizeof(T) == 8 ? 2 : 4;
    const ResNext next = res_record<1>(B, NT);
    const T *row = res_at<T>(next.p), *plane = res_at<T>(next.z);
    const int sj = next.sj_d & 0xfff, dj = next.sj_d >> 12, npsi = B.npsi;
    const ResZ<T> *zt = reinterpret_cast<const ResZ<T> *>(res_sm + B.o_z) + B.bz + L + (s.K - B.k0);
    const int kin = A.h.kinj - s.K, kpec = A.h.pz ? A.h.Nz - 1 - s.K : -1;
    T injA = 0, injB = 0;
    if ((F & kFInject) != 0 && A.h.kinj >= 0) {
        const T *inj = reinterpret_cast<const T *>(res_sm + B.o_inject) + 4 * q;
        injA = inj[2];
        injB = inj[3];
    }
    const T ax = A.h.dtdmx, ay = A.h.dtdmy, dtdmz = A.h.dtdmz, dtm = A.h.dtm;
    const T zx = plane[0], zy = plane[next.dz];
#pragma unroll
    for (int k0 = 0; k0 < L; k0 += C) {
        if (k0 > 0 && k0 >= s.nk) break;
        T yx[C], yz[C], x1[C], x2[C], p0[C], p1[C];
        ResZ<T> z[C];
#pragma unroll
        for (int u = 0; u < C; ++u) {
            const int k = k0 + u;
            if (k >= L) continue;
            yx[u] = row[k * sj];
            yz[u] = row[dj + k * sj];
            x1[u] = res_e<T, L, NT>(1)[k * NT + s.xp];
            x2[u] = res_e<T, L, NT>(2)[k * NT + s.xp];
            if constexpr ((F & kFPmlZ) != 0) {
                z[u] = zt[k];
                p0[u] = res_pz<T, L, NT>(npsi, 2)[min(k, npsi - 1) * NT];
                p1[u] = res_pz<T, L, NT>(npsi, 3)[min(k, npsi - 1) * NT];
            }
        }
#pragma unroll
        for (int u = 0; u < C; ++u) {
            const int k = k0 + u;
            if (k >= L) continue;
            const T ex = s.e0[k], ey = s.e1[k], ez = s.e2[k];
            const bool end = k == L - 1 || k + 1 >= s.nk;
            const T exk = end ? zx : s.e0[k + (k < L - 1)], eyk = end ? zy : s.e1[k + (k < L - 1)];
            T az = dtdmz;
            if constexpr ((F & kFPmlZ) != 0) az = dtdmz * z[u].ik;
            const T dEy_z = eyk - ey, dEz_y = yz[u] - ez, dEz_x = x2[u] - ez, dEx_z = exk - ex, dEx_y = yx[u] - ex, dEy_x = x1[u] - ey;
            T nhx = s.h0[k] + (az * dEy_z - ay * dEz_y);
            T nhy = s.h1[k] + (ax * dEz_x - az * dEx_z);
            const T nhz = s.h2[k] + (ay * dEx_y - ax * dEy_x);
            if constexpr ((F & kFPmlZ) != 0) {
                p0[u] = cpml_rec(z[u].b, p0[u], z[u].c, dEy_z);
                nhx += dtm * p0[u];
                p1[u] = cpml_rec(z[u].b, p1[u], z[u].c, dEx_z);
                nhy -= dtm * p1[u];
                nhx = k == kpec ? T(0) : nhx;
                nhy = k == kpec ? T(0) : nhy;
            }
            if constexpr ((F & kFInject) != 0) {
                nhx = k == kin ? nhx + injA : nhx;
                nhy = k == kin ? nhy - injB : nhy;
            }
            s.h0[k] = nhx; s.h1[k] = nhy; s.h2[k] = nhz;
        }
        if constexpr ((F & kFPmlZ) != 0) {
#pragma unroll
            for (int u = 0; u < C; ++u)
                if (k0 + u < L && k0 + u < min(s.nk, npsi)) {
                    res_pz<T, L, NT>(npsi, 2)[(k0 + u) * NT] = p0[u];
                    res_pz<T, L, NT>(npsi, 3)[(k0 + u) * NT] = p1[u];
                }
        }
    }
#pragma unroll
    for (int k = 0; k < L; ++k) {
        res_h<T, L, NT>(0)[k * NT + s.t] = s.h0[k];
        res_h<T, L, NT>(1)[k * NT + s.t] = s.h1[k];
        res_h<T, L, NT>(2)[k * NT + s.t] = s.h2[k];
    }
}

// Every feature, rolled: the run is read from and written to shared memory
// (which holds the same values) and taken back into registers at the end, so
// that the long body exists once and needs few registers.
template <typename T, int L, int NT>
__device__ __forceinline__ void res_run_e_all(const ResArgs<T> &A, const ResBlock &B, ResThread<T, L> &s, int q) {
    const ResNext next = res_record<0>(B, NT);
    const T *row = res_at<T>(next.p), *plane = res_at<T>(next.z);
    const int sj = next.sj_d & 0xfff, dj = next.sj_d >> 12, npsi = B.npsi;
    const MatCoef<T> *coef = reinterpret_cast<const MatCoef<T> *>(res_sm + B.o_coef);
    T hxm = plane[0], hym = plane[next.dz];
#pragma unroll 1
    for (int k = 0; k < s.nk; ++k) {
        const int c = k * NT + s.t, x = k * NT + s.xm;
        const T e[3] = {res_e<T, L, NT>(0)[c], res_e<T, L, NT>(1)[c], res_e<T, L, NT>(2)[c]};
        const T h[3] = {res_h<T, L, NT>(0)[c], res_h<T, L, NT>(1)[c], res_h<T, L, NT>(2)[c]};
        const int m = reinterpret_cast<const uint8_t *>(res_sm + B.o_ids)[c];
        T n[3];
        res_cell_e<T, L, NT, kFAll>(A.e, B, coef4(coef + m), m, s.i, s.J, s.K + k, k, s.t, q, e, h, row[k * sj], row[dj + k * sj],
                                res_h<T, L, NT>(1)[x], res_h<T, L, NT>(2)[x], hxm, hym, n);
        res_e<T, L, NT>(0)[c] = n[0];
        res_e<T, L, NT>(1)[c] = n[1];
        res_e<T, L, NT>(2)[c] = n[2];
        hxm = h[0];
        hym = h[1];
    }
#pragma unroll
    for (int k = 0; k < L; ++k) {
        const int c = k * NT + s.t;
        s.e0[k] = res_e<T, L, NT>(0)[c]; s.e1[k] = res_e<T, L, NT>(1)[c]; s.e2[k] = res_e<T, L, NT>(2)[c];
        s.h0[k] = res_h<T, L, NT>(0)[c]; s.h1[k] = res_h<T, L, NT>(1)[c]; s.h2[k] = res_h<T, L, NT>(2)[c];
    }
}
template <typename T, int L, int NT>
__device__ __forceinline__ void res_run_h_all(const ResArgs<T> &A, const ResBlock &B, ResThread<T, L> &s, int q) {
    const ResNext next = res_record<1>(B, NT);
    const T *row = res_at<T>(next.p), *plane = res_at<T>(next.z);
    const int sj = next.sj_d & 0xfff, dj = next.sj_d >> 12, npsi = B.npsi;
#pragma unroll 1
    for (int k = 0; k < s.nk; ++k) {
        const int c = k * NT + s.t, x = k * NT + s.xp;
        const T e[3] = {res_e<T, L, NT>(0)[c], res_e<T, L, NT>(1)[c], res_e<T, L, NT>(2)[c]};
        const T h[3] = {res_h<T, L, NT>(0)[c], res_h<T, L, NT>(1)[c], res_h<T, L, NT>(2)[c]};
        const bool end = k + 1 >= s.nk;
        const T exk = end ? plane[0] : res_e<T, L, NT>(0)[c + NT], eyk = end ? plane[next.dz] : res_e<T, L, NT>(1)[c + NT];
        T n[3];
        res_cell_h<T, L, NT, kFPmlXY | kFPmlZ | kFMisc>(A.h, B, s.i, s.J, s.K + k, k, s.t, q, e, h, row[k * sj], row[dj + k * sj],
                                                    res_e<T, L, NT>(1)[x], res_e<T, L, NT>(2)[x], exk, eyk, n);
        res_h<T, L, NT>(0)[c] = n[0];
        res_h<T, L, NT>(1)[c] = n[1];
        res_h<T, L, NT>(2)[c] = n[2];
    }
#pragma unroll
    for (int k = 0; k < L; ++k) {
        const int c = k * NT + s.t;
        s.e0[k] = res_e<T, L, NT>(0)[c]; s.e1[k] = res_e<T, L, NT>(1)[c]; s.e2[k] = res_e<T, L, NT>(2)[c];
        s.h0[k] = res_h<T, L, NT>(0)[c]; s.h1[k] = res_h<T, L, NT>(1)[c]; s.h2[k] = res_h<T, L, NT>(2)[c];
    }
}

// A run's face values into the neighbours' inboxes: E to the blocks below
// (HALF 0), H to the blocks above (HALF 1); y, z: the run's places there (-1:
// not at that face), in values.
struct alignas(8) ResSend { int y, z; };
template <int L, int NT, int HALF> __device__ __forceinline__ ResSend res_places(int nx, const ResBlock &B, int t) {
    const int ncol = nx * B.by, run = t / ncol, col = t - run * ncol, j = col / nx;
    ResSend r{-1, -1};
    if (run >= B.nseg) return r;
    const int put_y = HALF ? B.put_hy : B.put_ey, put_z = HALF ? B.put_hz : B.put_ez;
    if (put_y >= 0 && j == (HALF ? B.by - 1 : 0)) r.y = put_y + run * L * nx + col - j * nx;
    if (put_z >= 0 && run == (HALF ? B.nseg - 1 : 0)) r.z = put_z + col;
    return r;
}
template <typename T, int L, int NT, int HALF>
__device__ __forceinline__ void res_send(const ResArgs<T> &A, const ResBlock &B, const ResThread<T, L> &s, unsigned seq) {
    const ResSend at = reinterpret_cast<const ResSend *>(res_sm + B.o_send)[HALF * NT + threadIdx.x];
    constexpr int kWords = sizeof(T) / 4;
    const int nx = A.e.Nx;
    const T *c0 = HALF ? s.h0 : s.e0, *c1 = HALF ? s.h1 : s.e1, *c2 = HALF ? s.h2 : s.e2;
    if (at.z >= 0) {
        T x = c0[0], y = c1[0];
        if constexpr (HALF) {   // the run's last plane
#pragma unroll
            for (int k = 1; k < L; ++k)
                if (k < s.nk) { x = c0[k]; y = c1[k]; }
        }
        unsigned long long *p = A.inbox + (size_t)at.z * kWords;
        inbox_put(p, x, seq);
        inbox_put(p + nx * B.by * kWords, y, seq);
    }
    if (at.y >= 0) {
        unsigned long long *p = A.inbox + (size_t)at.y * kWords, *p2 = p + nx * B.bz * kWords;
#pragma unroll
        for (int k = 0; k < L; ++k) {
            if (k < s.nk) {
                inbox_put(p, c0[k], seq);
                inbox_put(p2, c2[k], seq);
            }
            p += nx * kWords;
            p2 += nx * kWords;
        }
    }
}

// Brings a half-step's halo into shared memory: H before E (HALF 0), E before
// H (HALF 1). The halo buffer has the inbox's layout, so a word's place is its
// number; each thread has a few reads in flight. False when a wait ran out.
template <typename T, int NT, int HALF>
__device__ __forceinline__ bool res_halo(const ResArgs<T> &A, const ResBlock &B, unsigned seq) {
    constexpr int U = NT == 512 || sizeof(T) == 8 ? 4 : NT == 384 ? 6 : 8;
    const int nx = A.e.Nx, ny = 2 * nx * B.bz, n = ny + 2 * nx * B.by;
    const int first = B.self_y ? ny : 0, last = B.self_z ? ny : n;   // words that come from the inbox
    constexpr int kWords = sizeof(T) / 4;
    const unsigned long long *box = A.inbox + (size_t)(HALF ? B.get_e : B.get_h) * kWords;
    T *const halo = reinterpret_cast<T *>(res_sm + B.o_halo);
    const int lane = threadIdx.x & 31;
    for (int w0 = first + threadIdx.x; w0 - lane < last; w0 += U * NT) {   // whole warps
        InboxWords<T> in[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (w0 + u * NT < last) inbox_read(box + (w0 + u * NT) * kWords, in[u]);
        unsigned late = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            T v;
            if (w0 + u * NT >= last) continue;
            if (inbox_take(in[u], v, seq)) halo[w0 + u * NT] = v;
            else late |= 1u << u;
        }
        if (__any_sync(0xffffffffu, late != 0)) {
            // Two lanes watch the last word of each face; the others read again
            // once it is there. (Every thread spinning on its own word keeps the
            // neighbours' stores waiting in L2.)
            const long long t0 = clock64();
            const int watch = lane == 0 ? ny - 1 : n - 1;
            bool there = lane > 1 || (lane == 0 ? B.self_y : B.self_z);
            for (;;) {
                if (!there) {
                    InboxWords<T> x;
                    T v;
                    inbox_read(box + watch * kWords, x);
                    there = inbox_take(x, v, seq);
                }
                if (__all_sync(0xffffffffu, there)) {
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (late >> u & 1) inbox_read(box + (w0 + u * NT) * kWords, in[u]);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        T v;
                        if ((late >> u & 1) && inbox_take(in[u], v, seq)) {
                            halo[w0 + u * NT] = v;
                            late &= ~(1u << u);
                        }
                    }
                    if (!__any_sync(0xffffffffu, late != 0)) break;
                }
                const bool over = lane == 0 && (clock64() - t0 > A.wait_cycles || *(volatile int *)A.abort);
                if (__any_sync(0xffffffffu, over)) {
                    if (lane == 0) {
                        *(volatile int *)A.abort = 1;
                        atomicExch(A.e.err, 1);
                    }
                    return false;
                }
            }
        }
    }
    return true;
}

// Recursive-convolution "ante" update of the block's dispersive cells with
// E^n (mats_RC.cpp:21-36), in the split kernels' order; the sums over poles
// are kept for the E update. Cells, materials and pole coefficients are in
// shared memory, so that a cell costs one round trip for its psi.
template <typename T> struct ResPole { Cplx<T> crec, dchi; };
struct ResMat { int np, pole, box; };
template <typename T, int L, int NT> __device__ __forceinline__ void res_ante(const ResArgs<T> &A, const ResBlock &B) {
    const StepArgs<T, uint8_t> &a = A.e;
    T *sum = reinterpret_cast<T *>(res_sm + B.o_sum);
    const ResDisp *cells = reinterpret_cast<const ResDisp *>(res_sm + B.o_disp);
    const ResMat *mats = reinterpret_cast<const ResMat *>(res_sm + B.o_mats);
    const ResPole<T> *poles = reinterpret_cast<const ResPole<T> *>(res_sm + B.o_poles);
    constexpr int kPoles = (NT == 512 ? 2 : 4) * 4 / (int)sizeof(T);   // in flight, beside the run's registers
    for (int r = threadIdx.x; r < B.disp_n; r += NT) {
        const ResDisp e = cells[r];
        const ResMat m = mats[e.place >> 16];
        const int c = e.place & 0xffff;
        Cplx<T> *__restrict__ P = a.psi + e.psi;
        const T ev[3] = {res_e<T, L, NT>(0)[c], res_e<T, L, NT>(1)[c], res_e<T, L, NT>(2)[c]};
        T s[3] = {0, 0, 0};
        for (int p0 = 0; p0 < m.np; p0 += kPoles) {
            const int pn = min(kPoles, m.np - p0);
            Cplx<T> v[kPoles][3];
#pragma unroll
            for (int p = 0; p < kPoles; ++p)
                if (p < pn)
#pragma unroll
                    for (int dd = 0; dd < 3; ++dd) v[p][dd] = P[(3 * (p0 + p) + dd) * m.box];
#pragma unroll
            for (int p = 0; p < kPoles; ++p)
                if (p < pn) {
                    const ResPole<T> x = poles[m.pole + p0 + p];
#pragma unroll
                    for (int dd = 0; dd < 3; ++dd) {
                        Cplx<T> w;
                        if constexpr (Exact<T>::value) {
                            w.re = (x.crec.re * v[p][dd].re - x.crec.im * v[p][dd].im) + x.dchi.re * ev[dd];
                            w.im = (x.crec.re * v[p][dd].im + x.crec.im * v[p][dd].re) + x.dchi.im * ev[dd];
                        } else {
                            w.re = v[p][dd].re + ((x.crec.re * v[p][dd].re - x.crec.im * v[p][dd].im) + x.dchi.re * ev[dd]);
                            w.im = v[p][dd].im + ((x.crec.re * v[p][dd].im + x.crec.im * v[p][dd].re) + x.dchi.im * ev[dd]);
                        }
                        P[(3 * (p0 + p) + dd) * m.box] = w;
                        s[dd] = s[dd] + w.re;
                    }
                }
        }
        sum[3 * r] = s[0];
        sum[3 * r + 1] = s[1];
        sum[3 * r + 2] = s[2];
    }
}

// This step's values at the sites the sensors read (plane sums, DFT planes):
// E (half 0) or H (half 1) from shared memory into the step's record, a site
// per thread, region by region.
template <typename T, int L, int NT>
__device__ __forceinline__ void res_taps(const ResArgs<T> &A, const ResBlock &B, int q, int half) {
    T *rec = A.raw + (size_t)q * A.rec;
    const T *f = half ? res_h<T, L, NT>(0) : res_e<T, L, NT>(0);
    const ResTaps *region = reinterpret_cast<const ResTaps *>(res_sm + B.o_taps);
    const uint2 *site = reinterpret_cast<const uint2 *>(res_sm + B.o_sites);
    for (int r = 0; r < B.tap_n; ++r) {
        const ResTaps g = region[r];
        if (half && !g.h) continue;
        T *out = rec + (half ? 3 * (size_t)g.stride : 0);
#pragma unroll 2
        for (int t = g.first + threadIdx.x; t < g.first + g.n; t += NT) {
            const uint2 e = site[t];
            const T v0 = f[e.x], v1 = f[L * NT + e.x], v2 = f[2 * L * NT + e.x];
            T *o = out + e.y;
            o[0] = v0;
            o[g.stride] = v1;
            o[2 * (size_t)g.stride] = v2;
        }
    }
}

// z-CPML psi of a thread's run between global and shared memory.
template <typename T, int L, int NT, bool Store>
__device__ __forceinline__ void res_psi(const ResArgs<T> &A, const ResBlock &B, const ResThread<T, L> &s) {
    const StepArgs<T, uint8_t> &a = A.e;
    T *const g[4] = {A.e.psi_z0, A.e.psi_z1, A.h.psi_z0, A.h.psi_z1};
    // a block with CPML planes has a slot for each of its run's planes
    const int n = Store ? min(s.nk, B.npsi) : B.npsi;
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        const int K = s.K + k;
        const int zn = k >= s.nk ? -1 : K < a.pml_zm ? K : K >= a.Nz - a.pml_zp ? K - (a.Nz - a.pml_zp) + a.pml_zm : -1;
        const long long o = s.i + (long long)s.J * a.Nx + zn * a.NxNy;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            T *p = res_pz<T, L, NT>(B.npsi, q) + k * NT;
            if constexpr (Store) {
                if (zn >= 0) g[q][o] = *p;
            } else {
                *p = zn >= 0 ? g[q][o] : T(0);
            }
        }
    }
}

template <typename T, int L, int NT>
__global__ void __launch_bounds__(NT, 1) resident_steps(const __grid_constant__ ResArgs<T> A) {
    __shared__ ResBlock B;
    const int tid = threadIdx.x;
    for (int t = tid; t < (int)(sizeof(ResBlock) / 4); t += NT)
        reinterpret_cast<int *>(&B)[t] = reinterpret_cast<const int *>(A.blocks + blockIdx.x)[t];
    __syncthreads();
    const StepArgs<T, uint8_t> &a = A.e;
    const int nx = a.Nx;
    ResThread<T, L> s;
    {
        // threads past the last run shadow the first column with no planes of their own
        const int ncol = nx * B.by, run = tid / ncol, col = run < B.nseg ? tid - run * ncol : 0, j = col / nx;
        const bool live = run < B.nseg;
        s.t = tid;
        s.i = col - j * nx;
        s.J = B.j0 + j;
        s.K = B.k0 + (live ? run * L : 0);
        s.nk = !live ? 0 : min(L, B.bz - run * L);
        s.xm = !live ? tid : s.i ? tid - 1 : tid + nx - 1;
        s.xp = !live ? tid : s.i < nx - 1 ? tid + 1 : tid - (nx - 1);
    }
    MatCoef<T> *coef = reinterpret_cast<MatCoef<T> *>(res_sm + B.o_coef);
    uint8_t *ids = res_sm + B.o_ids;
    for (int t = tid; t < a.nmat; t += NT) coef[t] = a.coef[t];
    if (B.disp_n > 0)
        for (int t = tid; t < L * NT; t += NT) reinterpret_cast<uint16_t *>(res_sm + B.o_rank)[t] = kResNoRank;
    // ---- load the run
    const long long first = s.i + (long long)s.J * nx + s.K * a.NxNy;
    s.mixed = false;
    int id0 = 0;
#pragma unroll
    for (int k = 0; k < L; ++k) {
        const bool live = k < s.nk;
        const long long o = first + k * a.NxNy;
        s.e0[k] = live ? a.Ex[o] : T(0);
        s.e1[k] = live ? a.Ey[o] : T(0);
        s.e2[k] = live ? a.Ez[o] : T(0);
        s.h0[k] = live ? a.Hx[o] : T(0);
        s.h1[k] = live ? a.Hy[o] : T(0);
        s.h2[k] = live ? a.Hz[o] : T(0);
        const int m = live ? a.mat[s.i + (long long)a.mpitch * (s.J + (long long)a.Ny * (s.K + k))] : 0;
        if ((k & 3) == 0) s.ids[k >> 2] = 0;
        s.ids[k >> 2] |= (unsigned)m << (8 * (k & 3));
        if (k == 0) id0 = m;
        s.mixed |= live && m != id0;
        const int c = k * NT + tid;
        ids[c] = (uint8_t)m;
        res_e<T, L, NT>(0)[c] = s.e0[k]; res_e<T, L, NT>(1)[c] = s.e1[k]; res_e<T, L, NT>(2)[c] = s.e2[k];
        res_h<T, L, NT>(0)[c] = s.h0[k]; res_h<T, L, NT>(1)[c] = s.h1[k]; res_h<T, L, NT>(2)[c] = s.h2[k];
    }
    res_psi<T, L, NT, false>(A, B, s);
    {
        // the first E update's H halo, from the arrays
        const int jm = B.j0 == 0 ? a.Ny - 1 : B.j0 - 1, km = B.k0 == 0 ? a.Nz - 1 : B.k0 - 1;
        const int ny = nx * B.bz, nz = nx * B.by;
        T *halo = reinterpret_cast<T *>(res_sm + B.o_halo);
        for (int t = tid; t < ny; t += NT) {
            const int k = t / nx;
            const long long o = (t - k * nx) + (long long)jm * nx + (B.k0 + k) * a.NxNy;
            halo[t] = a.Hx[o];
            halo[ny + t] = a.Hz[o];
        }
        for (int t = tid; t < nz; t += NT) {
            const long long o = t + (long long)B.j0 * nx + km * a.NxNy;
            halo[2 * ny + t] = a.Hx[o];
            halo[2 * ny + nz + t] = a.Hy[o];
        }
    }
    __syncthreads();
    s.v = coef4(coef + id0);
    s.C4 = coef[id0].C4;
    // runs cut short read past the block's planes: those entries change nothing
    for (int t = tid; t < 2 * (B.bz + L); t += NT) {
        const bool h = t >= B.bz + L;
        const int k = h ? t - B.bz - L : t, K = min(B.k0 + k, a.Nz - 1);
        const StepArgs<T, uint8_t> &x = h ? A.h : A.e;
        // E-side range [1, pml_zm) and [Nz - pml_zp + 1, Nz), H-side [0, pml_zm)
        // and [Nz - pml_zp, Nz - 1) (fdtd_pml.cpp:547,559,775,784)
        const bool on = a.pz && k < B.bz && (h ? K < a.pml_zm || (K >= a.Nz - a.pml_zp && K < a.Nz - 1)
                                   : (K >= 1 && K < a.pml_zm) || K >= a.Nz - a.pml_zp + 1);
        ResZ<T> z;
        z.ik = x.ikz[K];
        z.b = on ? x.bz[K] : (Exact<T>::value ? T(1) : T(0));   // FP32 holds b - 1
        z.c = on ? x.cz[K] : T(0);
        z.pad = 0;
        reinterpret_cast<ResZ<T> *>(res_sm + B.o_z)[t] = z;
    }
    // this launch's injection values
    if (a.kinj >= 0)
        for (int q = tid; q < A.steps; q += NT) {
            T *inj = reinterpret_cast<T *>(res_sm + B.o_inject) + 4 * q;
            inj[0] = (T)a.sc[q].inj_eA; inj[1] = (T)a.sc[q].inj_eB;
            inj[2] = (T)a.sc[q].inj_hA; inj[3] = (T)a.sc[q].inj_hB;
        }
    {
        ResNext *rec = reinterpret_cast<ResNext *>(res_sm + B.o_next);
        rec[tid] = res_next<T, L, NT, 0>(nx, B, tid);
        rec[NT + tid] = res_next<T, L, NT, 1>(nx, B, tid);
        ResSend *places = reinterpret_cast<ResSend *>(res_sm + B.o_send);
        places[tid] = res_places<L, NT, 0>(nx, B, tid);
        places[NT + tid] = res_places<L, NT, 1>(nx, B, tid);
    }
    for (int t = tid; t < B.tap_n; t += NT) reinterpret_cast<ResTaps *>(res_sm + B.o_taps)[t] = A.taps[B.tap_off + t];
    for (int t = tid; t < B.site_n; t += NT) reinterpret_cast<uint2 *>(res_sm + B.o_sites)[t] = A.sites[B.site_off + t];
    const bool mixed = __any_sync(0xffffffffu, s.mixed);   // a warp takes one of the two forms
    if (B.disp_n > 0) {
        for (int t = tid; t < B.disp_n; t += NT) {
            const ResDisp e = A.disp[B.disp_off + t];
            reinterpret_cast<ResDisp *>(res_sm + B.o_disp)[t] = e;
            reinterpret_cast<uint16_t *>(res_sm + B.o_rank)[e.place & 0xffff] = (uint16_t)t;
        }
        for (int t = tid; t < a.nmat; t += NT) {
            const DispInfo d = a.disp[t];
            reinterpret_cast<ResMat *>(res_sm + B.o_mats)[t] = ResMat{d.np, d.pole_off, (int)d.box};
        }
        for (int t = tid; t < A.npoles; t += NT) reinterpret_cast<ResPole<T> *>(res_sm + B.o_poles)[t] = ResPole<T>{a.crec[t], a.dchi[t]};
    }
    __syncthreads();
    if (B.disp_n > 0) res_ante<T, L, NT>(A, B);
    // half-step h of this launch carries number seq0 + h + 1
    bool ok = true;
#pragma unroll 1
    for (int q = 0; q < A.steps; ++q) {
        const unsigned seq = A.seq0 + 2 * q;
        if (q > 0) ok = res_halo<T, NT, 0>(A, B, seq);   // H of the step before
        if (!__syncthreads_and(ok)) return;
        switch (B.feat_e) {
            case 0:
                if (mixed) res_run_e<T, L, NT, 0, true>(A, B, s, q);
                else res_run_e<T, L, NT, 0, false>(A, B, s, q);
                break;
            case kFPmlZ | kFInject:
                if (mixed) res_run_e<T, L, NT, kFPmlZ | kFInject, true>(A, B, s, q);
                else res_run_e<T, L, NT, kFPmlZ | kFInject, false>(A, B, s, q);
                break;
            case kFDisp | kFPmlZ | kFInject: res_run_e<T, L, NT, kFDisp | kFPmlZ | kFInject, true>(A, B, s, q); break;
            default: res_run_e_all<T, L, NT>(A, B, s, q); break;
        }
        res_send<T, L, NT, 0>(A, B, s, seq + 1);
        __syncthreads();
        if (B.tap_n) res_taps<T, L, NT>(A, B, q, 0);
        // the next step's pole update, while the neighbours' E is on its way
        if (B.disp_n > 0 && q + 1 < A.steps) res_ante<T, L, NT>(A, B);
        ok = res_halo<T, NT, 1>(A, B, seq + 1);
        if (!__syncthreads_and(ok)) return;
        if (!(A.withhold && blockIdx.x == 0)) {
            switch (B.feat_h) {
                case 0: res_run_h<T, L, NT, 0>(A, B, s, q); break;
                case kFPmlZ | kFInject: res_run_h<T, L, NT, kFPmlZ | kFInject>(A, B, s, q); break;
                default: res_run_h_all<T, L, NT>(A, B, s, q); break;
            }
            res_send<T, L, NT, 1>(A, B, s, seq + 2);
        }
        __syncthreads();
        if (B.tap_n) res_taps<T, L, NT>(A, B, q, 1);
    }
    // ---- store the run
#pragma unroll
    for (int k = 0; k < L; ++k)
        if (k < s.nk) {
            const long long o = first + k * a.NxNy;
            a.Ex[o] = s.e0[k]; a.Ey[o] = s.e1[k]; a.Ez[o] = s.e2[k];
            a.Hx[o] = s.h0[k]; a.Hy[o] = s.h1[k]; a.Hz[o] = s.h2[k];
        }
    if (B.nzp > 0) res_psi<T, L, NT, true>(A, B, s);
}

template <typename T, int L, int NT> cudaError_t launch_resident_run(const ResArgs<T> &A, int grid, int smem, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(resident_steps<T, L, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, resident_steps<T, L, NT>, A);
}

}  // namespace aefdtd
