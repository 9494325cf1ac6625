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
// in global memory; the latter's update reads only the block's own E and runs
// before the block waits for its neighbours. The longest runs share one array
// between E and H (Tight).
//
// Exchange. An E update needs H of the y-1 and z-1 blocks, an H update E of
// the y+1 and z+1 blocks (fdtd_core.cpp:363-969; both wrap). The thread that
// owns a cell at such a face stores each value, together with the number of
// the half-step, as one 64-bit word into the neighbour's inbox (FP64: two
// words of 32 data bits each), and the neighbour brings its inbox into
// shared memory before its update, reading until every word carries the number
// it waits for: data and flag arrive together, so there is no fence and no
// second round trip. One inbox slot per value is enough: a value
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
// split: 12 x 10 x 90 FP64 4.5 / 13.5 us, 48 x 48 x 128 FP64 7.8 / 16.2,
// 64 x 64 x 128 FP64 12.9 / 20.0, 40 x 40 x 200 FP32 with a disk of poles
// 5.9 / 13.9, 64 x 64 x 128 FP32 with two 61-wavelength flux planes 8.6 / 15.1,
// 64 x 64 x 250 FP32 11.7 / 17.8.
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
// H [3][L][threads] (Tight: in the same place, see resident_steps), z-CPML psi
// [E 0, E 1, H 0, H 1][npsi][threads], a slot for each CPML plane of a run.
extern __shared__ __align__(16) unsigned char res_sm[];
template <typename T, int L, int NT> __device__ __forceinline__ T *res_e(int c) { return reinterpret_cast<T *>(res_sm) + c * L * NT; }
template <typename T, int L, int NT, bool Tight> __device__ __forceinline__ T *res_h(int c) {
    return reinterpret_cast<T *>(res_sm) + ((Tight ? 0 : 3) + c) * L * NT;
}
// psi q of the thread's first slot, its slots NT apart
template <typename T, int L, int NT, bool Tight> __device__ __forceinline__ T *res_pz(int npsi, int q) {
    return reinterpret_cast<T *>(res_sm) + ((Tight ? 3 : 6) * L + q * npsi) * NT + threadIdx.x;
}

// The injection plane alone (kFMisc adds the oscillator boxes).
constexpr unsigned kFInject = 16;

// A thread's run of cells for the whole launch. Its geometry is in the thread's
// records in shared memory (ResNext), read where it is used: kept in registers
// across the steps it would push the fields of the longer runs out of them.
template <typename T, int L> struct ResThread {
    T e0[L], e1[L], e2[L], h0[L], h1[L], h2[L];
    int K;                              // first plane
};
// z-CPML values of one of the block's planes for E and for H. The updates need no
// branch on the range (taking one cost a 60 x 60 x 200 FP32 cell 9 %): outside it
// psi is zero, chosen after the recursion, as its c = 0 would add 0 * inf, a NaN
// where the split kernels have none.
template <typename T> struct alignas(16) ResZ { T ik, b, c, pad; };
// Material id of a thread's run plane k: a word of shared memory per four planes.
template <int NT> __device__ __forceinline__ int res_id(const ResBlock &B, int k) {
    return (res_sm + B.o_ids)[((k >> 2) * NT + threadIdx.x) * 4 + (k & 3)];
}

// ---- one cell
// E of one cell at plane K (run plane k), feature set F: e the cell's E, h its
// H, hxj, hzj the row below, hyi, hzi the column before, hxm, hym the plane
// below; writes the new E to n.
template <typename T, int L, int NT, unsigned F>
__device__ __forceinline__ void res_cell_e(const StepArgs<T, uint8_t> &a, const ResBlock &B, const Coef4<T> v, int m, int i,
                                           int J, int K, int k, int slot, int t, int q, const T e[3], const T h[3], T hxj, T hzj,
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
        T *p0 = res_pz<T, L, NT, false>(B.npsi, 0) + slot * NT, *p1 = res_pz<T, L, NT, false>(B.npsi, 1) + slot * NT;
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
__device__ __forceinline__ void res_cell_h(const StepArgs<T, uint8_t> &a, const ResBlock &B, int i, int J, int K, int slot, int q, const T e[3],
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
        T *p0 = res_pz<T, L, NT, false>(B.npsi, 2) + slot * NT, *p1 = res_pz<T, L, NT, false>(B.npsi, 3) + slot * NT;
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
// the halo; the plane next to it: elements z and z + dz; and the thread of the
// column next to it. A run that reads a halo is also at the face whose values
// the block sends there, so the same places give those in the neighbour's
// inbox (p - halo along y, z - halo along z).
template <typename T> struct ResRow {
    const T *row, *plane;
    int sj, dj, dz, x;
    int nk, lo, from, np; // the run's planes, its first z-CPML plane (of either half-step), this half-step's first and how many
    int face_y, face_z;   // places in the halo, -1 for none
};
// The record: two words per half-step and thread, computed once per launch.
// p: element | halo << 16 | x << 17 | lo << 26; z: element | halo << 16 | nk << 17 | from << 22 | np << 27.
template <int L> struct ResPack {
    static_assert(L < 32, "a run's planes are packed in five bits");
    static constexpr unsigned kHalo = 1u << 16;   // above any element of 227 KB
};
template <typename T, int L, int NT, bool Tight, int HALF>
__device__ __forceinline__ uint2 res_pack(const StepArgs<T, uint8_t> &a, const ResBlock &B, int t) {
    const int nx = a.Nx, ncol = nx * B.by, last = B.nseg - 1, run = t / ncol;
    // threads past the last run read what the first column reads
    const bool live = run <= last;
    const int seg = live ? run : 0, col = live ? t - run * ncol : 0, j = col / nx, i = col - j * nx, kb = seg * L;
    const int base = HALF || Tight ? 0 : 3 * L * NT, halo = B.o_halo / (int)sizeof(T), own = live ? t : 0;
    unsigned p, z;
    const bool edge = HALF ? j == B.by - 1 : j == 0;
    if (!edge || B.self_y) p = base + own + (HALF ? (edge ? -j * nx : nx) : (edge ? (B.by - 1) * nx : -nx));
    else p = (halo + kb * nx + i) | ResPack<L>::kHalo;
    const bool end = HALF ? seg == last : seg == 0;
    if (!end || B.self_z) {
        const int k = HALF ? 0 : end ? B.bz - last * L - 1 : L - 1;
        z = base + k * NT + own + (HALF ? (end ? -last * ncol : ncol) : (end ? last * ncol : -ncol));
    } else {
        z = (halo + 2 * nx * B.bz + col) | ResPack<L>::kHalo;
    }
    const int x = !live ? t : HALF ? (i < nx - 1 ? t + 1 : t - (nx - 1)) : (i ? t - 1 : t + nx - 1);
    // planes of the run in the range of E, [1, pml_zm) and [Nz - pml_zp + 1, Nz), or
    // of H, [0, pml_zm) and [Nz - pml_zp, Nz - 1) (fdtd_pml.cpp:547,559,775,784);
    // no run holds planes of both ends (resident.cpp)
    const int K = B.k0 + kb, nk = live ? min(L, B.bz - kb) : 0;
    const int low = a.pz ? max(0, min(nk, a.pml_zm - K)) : 0, high = a.pz ? min(nk, max(0, a.Nz - a.pml_zp - K)) : nk;
    const int lo = low > 0 ? 0 : high;
    const int from = low > 0 ? (!HALF && K == 0) : min(nk, high + (!HALF && high < nk && K + high == a.Nz - a.pml_zp));
    const int to = low > 0 ? low : HALF && nk > high && K + nk == a.Nz ? nk - 1 : nk;
    return make_uint2(p | x << 17 | unsigned(lo) << 26, z | nk << 17 | from << 22 | unsigned(to - from) << 27);
}
template <typename T> __device__ __forceinline__ const T *res_at(int element) { return reinterpret_cast<const T *>(res_sm) + element; }
template <typename T, int L, int NT, int HALF> __device__ __forceinline__ ResRow<T> res_record(int nx, const ResBlock &B) {
    const uint2 w = reinterpret_cast<const uint2 *>(res_sm + B.o_next)[HALF * NT + threadIdx.x];
    const bool hp = (w.x & ResPack<L>::kHalo) != 0, hz = (w.y & ResPack<L>::kHalo) != 0;
    ResRow<T> r;
    const int p = w.x & 0xffff, z = w.y & 0xffff, halo = B.o_halo / (int)sizeof(T);
    r.row = res_at<T>(p);
    r.plane = res_at<T>(z);
    r.sj = hp ? nx : NT;
    r.dj = hp ? nx * B.bz : 2 * L * NT;
    r.dz = hz ? nx * B.by : L * NT;
    r.x = w.x >> 17 & 511;
    r.nk = w.y >> 17 & 31;
    r.lo = w.x >> 26;
    r.from = w.y >> 22 & 31;
    r.np = w.y >> 27;
    r.face_y = hp && r.nk > 0 ? p - halo : -1;
    r.face_z = hz && r.nk > 0 ? z - halo : -1;
    return r;
}

// The run in registers, fully unrolled: any of pole sums, z CPML and the
// injection plane; Mixed: the run holds several materials. Shared-memory
// reads of a few planes at a time are issued together, psi is stored after
// each such group and the fields (res_publish) after the whole run, so that no
// read waits behind a store it cannot be told apart from. Planes past nk compute values
// that nobody reads.
template <typename T, int L, int NT, bool Tight, unsigned F, bool Mixed>
__device__ __forceinline__ void res_run_e(const ResArgs<T> &A, const ResBlock &B, ResThread<T, L> &s, int q) {
    constexpr int C = (sizeof(T) == 8 ? 2 : 4) / (L * (int)sizeof(T) > 104 ? 2 : 1);
    const ResRow<T> next = res_record<T, L, NT, 0>(A.e.Nx, B);
    const T *row = next.row, *plane = next.plane;
    const int sj = next.sj, dj = next.dj, nk = next.nk, lo = next.lo;
    const auto on = [&](int k) { return unsigned(k - next.from) < unsigned(next.np); };   // in the z-CPML range
    const MatCoef<T> *coef = reinterpret_cast<const MatCoef<T> *>(res_sm + B.o_coef);
    const ResZ<T> *zt = reinterpret_cast<const ResZ<T> *>(res_sm + B.o_z) + (s.K - B.k0);
    // the run's coefficients where it has one material
    const MatCoef<T> *const one = coef + res_id<NT>(B, 0);
    const Coef4<T> v1 = coef4(one);
    const T C41 = one->C4;
    // the run's plane that takes the injection, and its conducting plane
    const int kin = A.e.kinj - s.K, kpec = A.e.pz ? -s.K : -1;
    T injA = 0, injB = 0;
    if ((F & kFInject) != 0 && A.e.kinj >= 0) {
        const T *inj = reinterpret_cast<const T *>(res_sm + B.o_inject) + 4 * q;
        injA = inj[0];
        injB = inj[1];
    }
    T *pz0 = res_pz<T, L, NT, Tight>(B.npsi, 0) - lo * NT, *pz1 = pz0 + B.npsi * NT;
    T hxm = plane[0], hym = plane[next.dz];
    constexpr bool kBatchSums = sizeof(T) == 4;   // FP64 has no registers for a group's pole sums
#pragma unroll
    for (int k0 = 0; k0 < L; k0 += C) {
        if (k0 > 0 && k0 >= nk) break;
        T yx[C], yz[C], x1[C], x2[C], p0[C], p1[C], d0[C], d1[C], d2[C], C3[C];
        int rank[C];
        Coef4<T> v[C];
        ResZ<T> z[C];
#pragma unroll
        for (int u = 0; u < C; ++u) {
            const int k = k0 + u;
            if (k >= L) continue;
            yx[u] = row[k * sj];
            yz[u] = row[dj + k * sj];
            x1[u] = res_h<T, L, NT, Tight>(1)[k * NT + next.x];
            x2[u] = res_h<T, L, NT, Tight>(2)[k * NT + next.x];
            if constexpr (Mixed) v[u] = coef4(coef + res_id<NT>(B, k));
            if constexpr ((F & kFDisp) != 0) rank[u] = reinterpret_cast<const uint16_t *>(res_sm + B.o_rank)[k * NT + threadIdx.x];
            if constexpr ((F & kFPmlZ) != 0) {
                z[u] = zt[k];
                p0[u] = on(k) ? pz0[k * NT] : T(0);
                p1[u] = on(k) ? pz1[k * NT] : T(0);
            }
        }
        if constexpr ((F & kFDisp) != 0 && kBatchSums) {
            bool some = false;
#pragma unroll
            for (int u = 0; u < C; ++u) some |= k0 + u < L && rank[u] != kResNoRank;
            if (some) {
                const T *sum = reinterpret_cast<const T *>(res_sm + B.o_sum);
#pragma unroll
                for (int u = 0; u < C; ++u) {
                    if (k0 + u >= L) continue;
                    const int r = rank[u] != kResNoRank ? 3 * rank[u] : 0;
                    d0[u] = sum[r];
                    d1[u] = sum[r + 1];
                    d2[u] = sum[r + 2];
                    C3[u] = coef[res_id<NT>(B, k0 + u)].C3;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < C; ++u) {
            const int k = k0 + u;
            if (k >= L) continue;
            const Coef4<T> c = Mixed ? v[u] : v1;
            const T hx = s.h0[k], hy = s.h1[k], hz = s.h2[k];
            const T dHz_y = hz - yz[u], dHy_z = hy - hym, dHx_z = hx - hxm, dHz_x = hz - x2[u], dHy_x = hy - x1[u], dHx_y = hx - yx[u];
            T ikz = 1;
            if constexpr ((F & kFPmlZ) != 0) ikz = z[u].ik;
            T nex = (c.C1 * s.e0[k] + c.C2y * dHz_y) - (c.C2z * ikz) * dHy_z;
            T ney = (c.C1 * s.e1[k] + (c.C2z * ikz) * dHx_z) - c.C2x * dHz_x;
            T nez = (c.C1 * s.e2[k] + c.C2x * dHy_x) - c.C2y * dHx_y;
            if constexpr ((F & kFDisp) != 0)
                if (rank[u] != kResNoRank) {
                    if constexpr (!kBatchSums) {
                        const T *sum = reinterpret_cast<const T *>(res_sm + B.o_sum) + 3 * rank[u];
                        d0[u] = sum[0];
                        d1[u] = sum[1];
                        d2[u] = sum[2];
                        C3[u] = coef[res_id<NT>(B, k)].C3;
                    }
                    nex += C3[u] * d0[u];
                    ney += C3[u] * d1[u];
                    nez += C3[u] * d2[u];
                }
            if constexpr ((F & kFPmlZ) != 0) {
                const T C4 = Mixed ? coef[res_id<NT>(B, k)].C4 : C41;
                p0[u] = on(k) ? cpml_rec(z[u].b, p0[u], z[u].c, dHy_z) : T(0);
                nex -= C4 * p0[u];
                p1[u] = on(k) ? cpml_rec(z[u].b, p1[u], z[u].c, dHx_z) : T(0);
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
                if (k0 + u < L && on(k0 + u)) {
                    pz0[(k0 + u) * NT] = p0[u];
                    pz1[(k0 + u) * NT] = p1[u];
                }
        }
    }
}
template <typename T, int L, int NT, bool Tight, unsigned F>
__device__ __forceinline__ void res_run_h(const ResArgs<T> &A, const ResBlock &B, ResThread<T, L> &s, int q) {
    constexpr int C = (sizeof(T) == 8 ? 2 : 4) / (L * (int)sizeof(T) > 104 ? 2 : 1);
    const ResRow<T> next = res_record<T, L, NT, 1>(A.e.Nx, B);
    const T *row = next.row, *plane = next.plane;
    const int sj = next.sj, dj = next.dj, nk = next.nk, lo = next.lo;
    const auto on = [&](int k) { return unsigned(k - next.from) < unsigned(next.np); };   // in the z-CPML range
    const ResZ<T> *zt = reinterpret_cast<const ResZ<T> *>(res_sm + B.o_z) + B.bz + L + (s.K - B.k0);
    const int kin = A.h.kinj - s.K, kpec = A.h.pz ? A.h.Nz - 1 - s.K : -1;
    T injA = 0, injB = 0;
    if ((F & kFInject) != 0 && A.h.kinj >= 0) {
        const T *inj = reinterpret_cast<const T *>(res_sm + B.o_inject) + 4 * q;
        injA = inj[2];
        injB = inj[3];
    }
    const T ax = A.h.dtdmx, ay = A.h.dtdmy, dtdmz = A.h.dtdmz, dtm = A.h.dtm;
    T *pz0 = res_pz<T, L, NT, Tight>(B.npsi, 2) - lo * NT, *pz1 = pz0 + B.npsi * NT;
    const T zx = plane[0], zy = plane[next.dz];
#pragma unroll
    for (int k0 = 0; k0 < L; k0 += C) {
        if (k0 > 0 && k0 >= nk) break;
        T yx[C], yz[C], x1[C], x2[C], p0[C], p1[C];
        ResZ<T> z[C];
#pragma unroll
        for (int u = 0; u < C; ++u) {
            const int k = k0 + u;
            if (k >= L) continue;
            yx[u] = row[k * sj];
            yz[u] = row[dj + k * sj];
            x1[u] = res_e<T, L, NT>(1)[k * NT + next.x];
            x2[u] = res_e<T, L, NT>(2)[k * NT + next.x];
            if constexpr ((F & kFPmlZ) != 0) {
                z[u] = zt[k];
                p0[u] = on(k) ? pz0[k * NT] : T(0);
                p1[u] = on(k) ? pz1[k * NT] : T(0);
            }
        }
#pragma unroll
        for (int u = 0; u < C; ++u) {
            const int k = k0 + u;
            if (k >= L) continue;
            const T ex = s.e0[k], ey = s.e1[k], ez = s.e2[k];
            const bool end = k == L - 1 || k + 1 >= nk;
            const T exk = end ? zx : s.e0[k + (k < L - 1)], eyk = end ? zy : s.e1[k + (k < L - 1)];
            T az = dtdmz;
            if constexpr ((F & kFPmlZ) != 0) az = dtdmz * z[u].ik;
            const T dEy_z = eyk - ey, dEz_y = yz[u] - ez, dEz_x = x2[u] - ez, dEx_z = exk - ex, dEx_y = yx[u] - ex, dEy_x = x1[u] - ey;
            T nhx = s.h0[k] + (az * dEy_z - ay * dEz_y);
            T nhy = s.h1[k] + (ax * dEz_x - az * dEx_z);
            const T nhz = s.h2[k] + (ay * dEx_y - ax * dEy_x);
            if constexpr ((F & kFPmlZ) != 0) {
                p0[u] = on(k) ? cpml_rec(z[u].b, p0[u], z[u].c, dEy_z) : T(0);
                nhx += dtm * p0[u];
                p1[u] = on(k) ? cpml_rec(z[u].b, p1[u], z[u].c, dEx_z) : T(0);
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
                if (k0 + u < L && on(k0 + u)) {
                    pz0[(k0 + u) * NT] = p0[u];
                    pz1[(k0 + u) * NT] = p1[u];
                }
        }
    }
}

// A run's field into its exchange array f.
template <typename T, int L, int NT> __device__ __forceinline__ void res_publish(T *f, const T *c0, const T *c1, const T *c2) {
    f += threadIdx.x;
#pragma unroll
    for (int k = 0; k < L; ++k) {
        f[k * NT] = c0[k];
        f[(L + k) * NT] = c1[k];
        f[(2 * L + k) * NT] = c2[k];
    }
}

// Every feature, rolled: the run is read from and written to shared memory
// (which holds the same values) and taken back into registers at the end, so
// that the long body exists once and needs few registers.
template <typename T, int L, int NT>
__device__ __forceinline__ void res_run_e_all(const ResArgs<T> &A, const ResBlock &B, ResThread<T, L> &s, int q) {
    const ResRow<T> next = res_record<T, L, NT, 0>(A.e.Nx, B);
    const T *row = next.row, *plane = next.plane;
    const int sj = next.sj, dj = next.dj, t = threadIdx.x;
    const int col = t - (s.K - B.k0) / L * (A.e.Nx * B.by), j = col / A.e.Nx, i = col - j * A.e.Nx, J = B.j0 + j;   // of a live run
    const MatCoef<T> *coef = reinterpret_cast<const MatCoef<T> *>(res_sm + B.o_coef);
    T hxm = plane[0], hym = plane[next.dz];
#pragma unroll 1
    for (int k = 0; k < next.nk; ++k) {
        const int c = k * NT + t, x = k * NT + next.x;
        const T e[3] = {res_e<T, L, NT>(0)[c], res_e<T, L, NT>(1)[c], res_e<T, L, NT>(2)[c]};
        const T h[3] = {res_h<T, L, NT, false>(0)[c], res_h<T, L, NT, false>(1)[c], res_h<T, L, NT, false>(2)[c]};
        const int m = res_id<NT>(B, k);
        T n[3];
        res_cell_e<T, L, NT, kFAll>(A.e, B, coef4(coef + m), m, i, J, s.K + k, k, k - next.lo, t, q, e, h, row[k * sj], row[dj + k * sj],
                                res_h<T, L, NT, false>(1)[x], res_h<T, L, NT, false>(2)[x], hxm, hym, n);
        res_e<T, L, NT>(0)[c] = n[0];
        res_e<T, L, NT>(1)[c] = n[1];
        res_e<T, L, NT>(2)[c] = n[2];
        hxm = h[0];
        hym = h[1];
    }
#pragma unroll
    for (int k = 0; k < L; ++k) {
        const int c = k * NT + t;
        s.e0[k] = res_e<T, L, NT>(0)[c]; s.e1[k] = res_e<T, L, NT>(1)[c]; s.e2[k] = res_e<T, L, NT>(2)[c];
        s.h0[k] = res_h<T, L, NT, false>(0)[c]; s.h1[k] = res_h<T, L, NT, false>(1)[c]; s.h2[k] = res_h<T, L, NT, false>(2)[c];
    }
}
template <typename T, int L, int NT>
__device__ __forceinline__ void res_run_h_all(const ResArgs<T> &A, const ResBlock &B, ResThread<T, L> &s, int q) {
    const ResRow<T> next = res_record<T, L, NT, 1>(A.e.Nx, B);
    const T *row = next.row, *plane = next.plane;
    const int sj = next.sj, dj = next.dj, t = threadIdx.x;
    const int col = t - (s.K - B.k0) / L * (A.e.Nx * B.by), j = col / A.e.Nx, i = col - j * A.e.Nx, J = B.j0 + j;   // of a live run
#pragma unroll 1
    for (int k = 0; k < next.nk; ++k) {
        const int c = k * NT + t, x = k * NT + next.x;
        const T e[3] = {res_e<T, L, NT>(0)[c], res_e<T, L, NT>(1)[c], res_e<T, L, NT>(2)[c]};
        const T h[3] = {res_h<T, L, NT, false>(0)[c], res_h<T, L, NT, false>(1)[c], res_h<T, L, NT, false>(2)[c]};
        const bool end = k + 1 >= next.nk;
        const T exk = end ? plane[0] : res_e<T, L, NT>(0)[c + NT], eyk = end ? plane[next.dz] : res_e<T, L, NT>(1)[c + NT];
        T n[3];
        res_cell_h<T, L, NT, kFPmlXY | kFPmlZ | kFMisc>(A.h, B, i, J, s.K + k, k - next.lo, q, e, h, row[k * sj], row[dj + k * sj],
                                                    res_e<T, L, NT>(1)[x], res_e<T, L, NT>(2)[x], exk, eyk, n);
        res_h<T, L, NT, false>(0)[c] = n[0];
        res_h<T, L, NT, false>(1)[c] = n[1];
        res_h<T, L, NT, false>(2)[c] = n[2];
    }
#pragma unroll
    for (int k = 0; k < L; ++k) {
        const int c = k * NT + t;
        s.e0[k] = res_e<T, L, NT>(0)[c]; s.e1[k] = res_e<T, L, NT>(1)[c]; s.e2[k] = res_e<T, L, NT>(2)[c];
        s.h0[k] = res_h<T, L, NT, false>(0)[c]; s.h1[k] = res_h<T, L, NT, false>(1)[c]; s.h2[k] = res_h<T, L, NT, false>(2)[c];
    }
}

// A run's face values into the neighbours' inboxes: E to the blocks below
// (HALF 0), H to the blocks above (HALF 1).
template <typename T, int L, int NT, int HALF>
__device__ __forceinline__ void res_send(const ResArgs<T> &A, const ResBlock &B, const ResThread<T, L> &s, unsigned seq) {
    constexpr int kWords = sizeof(T) / 4;
    const int nx = A.e.Nx;
    const T *c0 = HALF ? s.h0 : s.e0, *c1 = HALF ? s.h1 : s.e1, *c2 = HALF ? s.h2 : s.e2;
    const ResRow<T> at = res_record<T, L, NT, HALF>(nx, B);
    if (at.face_z >= 0) {
        T x = c0[0], y = c1[0];
        if constexpr (HALF) {   // the run's last plane
#pragma unroll
            for (int k = 1; k < L; ++k)
                if (k < at.nk) { x = c0[k]; y = c1[k]; }
        }
        unsigned long long *p = A.inbox + (size_t)((HALF ? B.put_hz : B.put_ez) + at.face_z - 2 * nx * B.bz) * kWords;
        inbox_put(p, x, seq);
        inbox_put(p + nx * B.by * kWords, y, seq);
    }
    if (at.face_y >= 0) {
        unsigned long long *p = A.inbox + (size_t)((HALF ? B.put_hy : B.put_ey) + at.face_y) * kWords, *p2 = p + nx * B.bz * kWords;
#pragma unroll
        for (int k = 0; k < L; ++k) {
            if (k < at.nk) {
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
// shared memory, so that a cell costs one round trip for its psi (and its
// record one read: chains of table reads cost more than the psi). A thread
// takes one component of a cell at a time, kResPoles poles of it per trip (with
// whole cells the values in flight pushed the longer runs' fields out of the
// registers).
template <typename T> struct ResPole { Cplx<T> crec, dchi; };
struct alignas(16) ResCell { int psi, pole, box; unsigned short cell, np; };
// Where the tables are, read once: shared memory is reread after every store.
template <typename T> struct ResTables {
    const ResCell *cells;
    const ResPole<T> *poles;
    T *sum;
    Cplx<T> *psi;
    int n;
    __device__ ResTables(const ResArgs<T> &A, const ResBlock &B)
        : cells(reinterpret_cast<const ResCell *>(res_sm + B.o_disp)), poles(reinterpret_cast<const ResPole<T> *>(res_sm + B.o_poles)),
          sum(reinterpret_cast<T *>(res_sm + B.o_sum)), psi(A.e.psi), n(B.disp_n) {}
};
template <typename T> __device__ __forceinline__ Cplx<T> res_pole(const ResPole<T> &x, const Cplx<T> y, T e) {
    Cplx<T> w;
    if constexpr (Exact<T>::value) {
        w.re = (x.crec.re * y.re - x.crec.im * y.im) + x.dchi.re * e;
        w.im = (x.crec.re * y.im + x.crec.im * y.re) + x.dchi.im * e;
    } else {
        w.re = y.re + ((x.crec.re * y.re - x.crec.im * y.im) + x.dchi.re * e);
        w.im = y.im + ((x.crec.re * y.im + x.crec.im * y.re) + x.dchi.im * e);
    }
    return w;
}
// Item t: component t / n of dispersive cell t % n: its psi, E, poles, and where its sum goes.
template <typename T> struct ResItem {
    Cplx<T> *P;
    T e;
    int sum, pole, np, box;
};
template <typename T, int L, int NT> __device__ __forceinline__ ResItem<T> res_item(const ResTables<T> &X, int t) {
    const int dd = (t >= X.n) + (t >= 2 * X.n), r = t - dd * X.n;
    const ResCell c = X.cells[r];
    return {X.psi + c.psi + dd * c.box, res_e<T, L, NT>(dd)[c.cell], 3 * r + dd, c.pole, c.np, 3 * c.box};
}
// Poles p0 to p0 + kResPoles of an item, their psi in v.
template <typename T> __device__ __forceinline__ void res_poles(const ResPole<T> *poles, const ResItem<T> &x, int p0, const Cplx<T> *v, T &s) {
#pragma unroll
    for (int p = 0; p < kResPoles; ++p)
        if (p0 + p < x.np) {
            const Cplx<T> w = res_pole(poles[x.pole + p0 + p], v[p], x.e);
            x.P[(p0 + p) * x.box] = w;
            s = s + w.re;
        }
}
template <typename T> __device__ __forceinline__ void res_poles_load(const ResItem<T> &x, int p0, Cplx<T> *v) {
#pragma unroll
    for (int p = 0; p < kResPoles; ++p)
        if (p0 + p < x.np) v[p] = x.P[(p0 + p) * x.box];
}
// Asynchronous copy of one complex value to shared memory.
__device__ __forceinline__ void res_fetch(Cplx<float> *to, const Cplx<float> *from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void res_fetch(Cplx<double> *to, const Cplx<double> *from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}
// Short runs: U items in flight in registers.
template <typename T, int L, int NT, int U> __device__ __forceinline__ void res_ante_direct(const ResArgs<T> &A, const ResBlock &B) {
    const ResTables<T> X(A, B);
    const int n = 3 * X.n;
    for (int t0 = threadIdx.x; t0 < n; t0 += U * NT) {
        ResItem<T> x[U];
        Cplx<T> v[U][kResPoles];
        T s[U];
        int most = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            x[u].np = 0;
            s[u] = 0;
            if (t0 + u * NT < n) x[u] = res_item<T, L, NT>(X, t0 + u * NT);
            most = max(most, x[u].np);
        }
        for (int p0 = 0; p0 < most; p0 += kResPoles) {
#pragma unroll
            for (int u = 0; u < U; ++u) res_poles_load(x[u], p0, v[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) res_poles(X.poles, x[u], p0, v[u], s[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (t0 + u * NT < n) X.sum[x[u].sum] = s[u];
    }
}
// Long runs leave no registers for psi in flight: the first poles of a thread's
// next cells are copied ahead into shared memory, each thread its own.
// Whole cells here, as with two warps per scheduler the instructions of a round
// are what it costs: reading the tables once per cell instead of once per
// component takes a third of them.
template <typename T, int L, int NT> __device__ __forceinline__ void res_ante_staged(const ResArgs<T> &A, const ResBlock &B) {
    const ResTables<T> X(A, B);
    Cplx<T> *stage = reinterpret_cast<Cplx<T> *>(res_sm + B.o_stage) + threadIdx.x;
    constexpr int D = res_stage(sizeof(T)), kVal = 3 * kResPoles;
    const auto fetch = [&](int r) {
        const int t = threadIdx.x + r * NT;
        if (t < X.n) {
            const ResCell c = X.cells[t];
            const Cplx<T> *P = X.psi + c.psi;
#pragma unroll
            for (int p = 0; p < kResPoles; ++p)
                if (p < c.np)
#pragma unroll
                    for (int dd = 0; dd < 3; ++dd) res_fetch(stage + (r % D * kVal + 3 * p + dd) * NT, P + (3 * p + dd) * c.box);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int r = 0; r < D; ++r) fetch(r);
#pragma unroll 1
    for (int r = 0; (int)threadIdx.x + r * NT < X.n; ++r) {
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
        const int t = threadIdx.x + r * NT;
        const ResCell c = X.cells[t];
        // FP64: a component at a time, for the registers
        constexpr int W = sizeof(T) == 8 ? 1 : 3;
#pragma unroll 1
        for (int d0 = 0; d0 < 3; d0 += W) {
            Cplx<T> *__restrict__ P = X.psi + c.psi + d0 * c.box;
            const Cplx<T> *from = stage + (r % D * kVal + d0) * NT;
            T e[W], s[W];
#pragma unroll
            for (int w = 0; w < W; ++w) { e[w] = res_e<T, L, NT>(d0 + w)[c.cell]; s[w] = 0; }
            const auto pole = [&](int p, bool staged) {
                const ResPole<T> x = X.poles[c.pole + p];
                Cplx<T> v[W];
#pragma unroll
                for (int w = 0; w < W; ++w) v[w] = staged ? from[(3 * p + w) * NT] : P[(3 * p + w) * c.box];
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    const Cplx<T> y = res_pole(x, v[w], e[w]);
                    P[(3 * p + w) * c.box] = y;
                    s[w] = s[w] + y.re;
                }
            };
#pragma unroll
            for (int p = 0; p < kResPoles; ++p)
                if (p < c.np) pole(p, true);
#pragma unroll 1
            for (int p = kResPoles; p < c.np; ++p) pole(p, false);
#pragma unroll
            for (int w = 0; w < W; ++w) X.sum[3 * t + d0 + w] = s[w];
        }
        fetch(r + D);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}
template <typename T, int L, int NT> __device__ __forceinline__ void res_ante(const ResArgs<T> &A, const ResBlock &B) {
    if constexpr (res_staged(L, sizeof(T))) res_ante_staged<T, L, NT>(A, B);
    else res_ante_direct<T, L, NT, (NT > 256 ? 1 : 3)>(A, B);
}

// This step's values at the sites the sensors read (plane sums, DFT planes):
// E (half 0) or H (half 1) from shared memory into the step's record, a site
// per thread, region by region.
template <typename T, int L, int NT, bool Tight>
__device__ __forceinline__ void res_taps(const ResArgs<T> &A, const ResBlock &B, int q, int half) {
    T *rec = A.raw + (size_t)q * A.rec;
    const T *f = half ? res_h<T, L, NT, Tight>(0) : res_e<T, L, NT>(0);
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
template <typename T, int L, int NT, bool Tight, bool Store>
__device__ __forceinline__ void res_psi(const ResArgs<T> &A, const ResBlock &B, const ResThread<T, L> &s, int i, int J) {
    const ResRow<T> at = res_record<T, L, NT, 0>(A.e.Nx, B);
    const StepArgs<T, uint8_t> &a = A.e;
    T *const g[4] = {A.e.psi_z0, A.e.psi_z1, A.h.psi_z0, A.h.psi_z1};
#pragma unroll 1
    for (int n = 0; at.lo + n < at.nk; ++n) {
        const int K = s.K + at.lo + n;
        if (K >= a.pml_zm && K < a.Nz - a.pml_zp) break;
        const int zn = K < a.pml_zm ? K : K - (a.Nz - a.pml_zp) + a.pml_zm;
        const long long o = i + (long long)J * a.Nx + zn * a.NxNy;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            T *p = res_pz<T, L, NT, Tight>(B.npsi, q) + n * NT;
            if constexpr (Store) g[q][o] = *p;
            else *p = g[q][o];
        }
    }
}

// Tight: E and H take turns in one exchange array. An update's neighbours' values
// are read before its own result is published, with a barrier between, so the
// field that a phase reads is always the one there. Half the shared memory per
// cell for one barrier more per half-step; the blocks need the run updates
// (res_run_e_all keeps both fields in shared memory).
template <typename T, int L, int NT, bool Tight>
__global__ void __launch_bounds__(NT, 1) resident_steps(const __grid_constant__ ResArgs<T> A) {
    __shared__ ResBlock B;
    const int tid = threadIdx.x;
    for (int t = tid; t < (int)(sizeof(ResBlock) / 4); t += NT)
        reinterpret_cast<int *>(&B)[t] = reinterpret_cast<const int *>(A.blocks + blockIdx.x)[t];
    __syncthreads();
    const StepArgs<T, uint8_t> &a = A.e;
    const int nx = a.Nx;
    ResThread<T, L> s;
    uint2 *const rec = reinterpret_cast<uint2 *>(res_sm + B.o_next);
    rec[tid] = res_pack<T, L, NT, Tight, 0>(a, B, tid);
    rec[NT + tid] = res_pack<T, L, NT, Tight, 1>(a, B, tid);
    // threads past the last run shadow the first column with no planes of their own
    const auto column = [&](int &i, int &J, int &nk) {
        const int ncol = nx * B.by, run = tid / ncol, col = run < B.nseg ? tid - run * ncol : 0, j = col / nx;
        i = col - j * nx;
        J = B.j0 + j;
        s.K = B.k0 + (run < B.nseg ? run * L : 0);
        nk = run < B.nseg ? min(L, B.bz - run * L) : 0;
    };
    int i, J, nk;
    column(i, J, nk);
    MatCoef<T> *coef = reinterpret_cast<MatCoef<T> *>(res_sm + B.o_coef);
    unsigned *ids = reinterpret_cast<unsigned *>(res_sm + B.o_ids);
    for (int t = tid; t < a.nmat; t += NT) coef[t] = a.coef[t];
    if (B.disp_n > 0)
        for (int t = tid; t < L * NT; t += NT) reinterpret_cast<uint16_t *>(res_sm + B.o_rank)[t] = kResNoRank;
    // ---- load the run
    const long long first = i + (long long)J * nx + s.K * a.NxNy;
    bool mixed = false;   // more than one material in the run
    unsigned id0 = 0, word = 0;
#pragma unroll
    for (int k = 0; k < L; ++k) {
        const bool live = k < nk;
        const long long o = first + k * a.NxNy;
        s.e0[k] = live ? a.Ex[o] : T(0);
        s.e1[k] = live ? a.Ey[o] : T(0);
        s.e2[k] = live ? a.Ez[o] : T(0);
        s.h0[k] = live ? a.Hx[o] : T(0);
        s.h1[k] = live ? a.Hy[o] : T(0);
        s.h2[k] = live ? a.Hz[o] : T(0);
        const unsigned m = live ? a.mat[i + (long long)a.mpitch * (J + (long long)a.Ny * (s.K + k))] : 0;
        word = (k & 3) == 0 ? m : word | m << (8 * (k & 3));
        if ((k & 3) == 3 || k == L - 1) ids[(k >> 2) * NT + tid] = word;
        if (k == 0) id0 = m;
        mixed |= live && m != id0;
    }
    res_publish<T, L, NT>(res_e<T, L, NT>(0), s.e0, s.e1, s.e2);
    if constexpr (!Tight) res_publish<T, L, NT>(res_h<T, L, NT, false>(0), s.h0, s.h1, s.h2);
    res_psi<T, L, NT, Tight, false>(A, B, s, i, J);
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
    for (int t = tid; t < B.tap_n; t += NT) reinterpret_cast<ResTaps *>(res_sm + B.o_taps)[t] = A.taps[B.tap_off + t];
    for (int t = tid; t < B.site_n; t += NT) reinterpret_cast<uint2 *>(res_sm + B.o_sites)[t] = A.sites[B.site_off + t];
    mixed = __any_sync(0xffffffffu, mixed);   // a warp takes one of the two forms
    if (B.disp_n > 0) {
        for (int t = tid; t < B.disp_n; t += NT) {
            const ResDisp e = A.disp[B.disp_off + t];
            const DispInfo d = a.disp[e.place >> 16];
            ResCell c;
            c.psi = e.psi;
            c.pole = d.pole_off;
            c.box = (int)d.box;
            c.cell = (unsigned short)e.place;
            c.np = (unsigned short)d.np;
            reinterpret_cast<ResCell *>(res_sm + B.o_disp)[t] = c;
            reinterpret_cast<uint16_t *>(res_sm + B.o_rank)[e.place & 0xffff] = (uint16_t)t;
        }
        for (int t = tid; t < A.npoles; t += NT) reinterpret_cast<ResPole<T> *>(res_sm + B.o_poles)[t] = ResPole<T>{a.crec[t], a.dchi[t]};
    }
    __syncthreads();
    if (B.disp_n > 0) res_ante<T, L, NT>(A, B);
    if constexpr (Tight) {
        __syncthreads();
        res_publish<T, L, NT>(res_h<T, L, NT, true>(0), s.h0, s.h1, s.h2);
    }
    // half-step h of this launch carries number seq0 + h + 1
    bool ok = true;
#pragma unroll 1
    for (int q = 0; q < A.steps; ++q) {
        const unsigned seq = A.seq0 + 2 * q;
        if (q > 0) ok = res_halo<T, NT, 0>(A, B, seq);   // H of the step before
        if (!__syncthreads_and(ok)) return;
        switch (B.feat_e) {
            case 0:
                if (mixed) res_run_e<T, L, NT, Tight, 0, true>(A, B, s, q);
                else res_run_e<T, L, NT, Tight, 0, false>(A, B, s, q);
                break;
            case kFPmlZ | kFInject:
                if (mixed) res_run_e<T, L, NT, Tight, kFPmlZ | kFInject, true>(A, B, s, q);
                else res_run_e<T, L, NT, Tight, kFPmlZ | kFInject, false>(A, B, s, q);
                break;
            case kFDisp | kFPmlZ | kFInject: res_run_e<T, L, NT, Tight, kFDisp | kFPmlZ | kFInject, true>(A, B, s, q); break;
            default:
                if constexpr (!Tight) res_run_e_all<T, L, NT>(A, B, s, q);
                break;
        }
        if constexpr (Tight) __syncthreads();
        res_publish<T, L, NT>(res_e<T, L, NT>(0), s.e0, s.e1, s.e2);
        res_send<T, L, NT, 0>(A, B, s, seq + 1);
        __syncthreads();
        if (B.tap_n) res_taps<T, L, NT, Tight>(A, B, q, 0);
        // the next step's pole update, while the neighbours' E is on its way
        if (B.disp_n > 0 && q + 1 < A.steps) res_ante<T, L, NT>(A, B);
        ok = res_halo<T, NT, 1>(A, B, seq + 1);
        if (!__syncthreads_and(ok)) return;
        if (!(A.withhold && blockIdx.x == 0)) {
            switch (B.feat_h) {
                case 0: res_run_h<T, L, NT, Tight, 0>(A, B, s, q); break;
                case kFPmlZ | kFInject: res_run_h<T, L, NT, Tight, kFPmlZ | kFInject>(A, B, s, q); break;
                default:
                    if constexpr (!Tight) res_run_h_all<T, L, NT>(A, B, s, q);
                    break;
            }
            if constexpr (Tight) __syncthreads();
            res_publish<T, L, NT>(res_h<T, L, NT, Tight>(0), s.h0, s.h1, s.h2);
            res_send<T, L, NT, 1>(A, B, s, seq + 2);
        }
        __syncthreads();
        if (B.tap_n) res_taps<T, L, NT, Tight>(A, B, q, 1);
    }
    // ---- store the run
    column(i, J, nk);
    const long long out = i + (long long)J * nx + s.K * a.NxNy;
#pragma unroll
    for (int k = 0; k < L; ++k)
        if (k < nk) {
            const long long o = out + k * a.NxNy;
            a.Ex[o] = s.e0[k]; a.Ey[o] = s.e1[k]; a.Ez[o] = s.e2[k];
            a.Hx[o] = s.h0[k]; a.Hy[o] = s.h1[k]; a.Hz[o] = s.h2[k];
        }
    if (B.nzp > 0) res_psi<T, L, NT, Tight, true>(A, B, s, i, J);
}

template <typename T> struct ResEntry {
    void (*kernel)(const ResArgs<T>) = nullptr;
    int threads = 0;
};
template <typename T, int L, int NT, bool Tight = false> ResEntry<T> resident_entry() { return {resident_steps<T, L, NT, Tight>, NT}; }

// The attribute belongs to the kernel, not to a simulation: threads that step
// simulations with different plans all set the same value, the device's limit.
template <typename T> cudaError_t prepare_resident_entry(const ResEntry<T> &k, int most, int smem, int &per_sm) {
    per_sm = 0;
    if (!k.kernel) return cudaErrorInvalidValue;
    const cudaError_t e = cudaFuncSetAttribute(k.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    return e != cudaSuccess ? e : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k.kernel, k.threads, smem);
}

template <typename T>
cudaError_t launch_resident_entry(const ResEntry<T> &k, const ResArgs<T> &A, int grid, int smem, cudaStream_t st) {
    if (!k.kernel) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(k.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k.kernel, A);
}

}  // namespace aefdtd
