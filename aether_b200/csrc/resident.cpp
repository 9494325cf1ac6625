// resident.cpp — host side of the resident time steps (resident.cuh): the cut
// of the grid into blocks, their shared-memory layout, inboxes, dispersive
// cells and sensor sites, and the launches of a chunk of steps.
#include "sim.hpp"

namespace aefdtd {
namespace {

constexpr unsigned kXY = 1, kZ = 2, kDisp = 4, kMisc = 8, kInject = 16;   // kF* of yee.cuh and resident.cuh

// The unrolled updates exist for these feature sets; any other takes the full one.
unsigned kernel_feat(unsigned f) {
    if (f == 0) return 0;
    if ((f & (kXY | kMisc)) == 0) return (f & kDisp) | kZ | kInject;
    return kXY | kZ | kDisp | kMisc;
}

// Cut of n weighted rows into `parts` runs of about equal weight, each at least one row.
std::vector<int> cut(const std::vector<double> &w, int parts) {
    const int n = (int)w.size();
    std::vector<double> cum(n + 1, 0.0);
    for (int i = 0; i < n; i++) cum[i + 1] = cum[i] + w[i];
    std::vector<int> c(parts + 1, 0);
    c[parts] = n;
    int p = 0;
    for (int m = 1; m < parts; m++) {
        const double want = cum[n] * m / parts;
        while (p < n && cum[p] < want) p++;
        if (p > 0 && want - cum[p - 1] < cum[p] - want) p--;
        p = std::clamp(p, c[m - 1] + 1, n - (parts - m));
        c[m] = p;
    }
    return c;
}

size_t up16(size_t b) { return (b + 15) / 16 * 16; }

}  // namespace
}  // namespace aefdtd

// Whether the next n steps can run resident: the drivers and sensors that the
// resident kernel records sites for, ids of one byte, and a plan that fits.
// The knobs that pin other kernels (and timing runs, which time the split
// groups) keep their path.
bool aefdtd_sim::resident_ready(int n) {
    if (!use_resident || batch || obl || timing || cc_coeff > 0 || !fmaps.empty() || id_bytes != 1 ||
        sensors.size() > (size_t)kMaxGather || fused_eligible() || use_tma)
        return false;
    // A call of one step pays for loading and storing the whole state. The split
    // kernels give the same bits in FP64 and take over there past 10 MB of
    // fields; us per call, resident / split, without and with two flux planes:
    // 12 x 10 x 90 24.7 / 27.9 and 31.3 / 37.0, 70 x 58 x 50 30.6 / 26.4 and 35.0
    // / 37.1, 48 x 48 x 128 32.9 / 28.1 and 41.7 / 34.7, 64 x 64 x 128 43.1 / 31.7
    // and 52.2 / 38.2; at two steps 31.6 / 33.4 per step. FP32 kernels round
    // differently, so FP32 keeps to one path however a run is cut into calls (64 x
    // 64 x 250: 47.2 / 30.5 per call of one step, 27.8 / 27.9 per step at two).
    if (fp64 && n == 1 && 48.0 * Nx * Ny * Nz > 10e6) return false;
    if (res_dirty) build_resident();
    return res.grid > 0;
}

// Chooses the cut and the run length with the smallest estimated step time and
// fills the blocks.
//
// Cost of a step, in SM cycles of the slowest block (measured on cells of 12 to
// 64 rows): per half-step 300, and per plane of its runs 40 (sending the
// face) and per warp 11.5 (FP32), 20 or, past 13 planes, 30 (FP64), twice that
// with z CPML, 2.5 times with poles, eight times in the rolled update (x/y
// CPML, oscillators); per round of the threads over the dispersive cells 1700,
// or 3500 in the long FP64 runs, in the short runs with 12 values per pole read
// and written in L2 besides; the halo values past those that the threads read
// in one round trip 0.75 (FP32) or 1.5 (FP64) each; and 2600 for the two round
// trips of the inbox. Rows and planes are cut to equal weights; pole state is
// concentrated in few rows and planes, so cuts with its weight raised are tried
// too, and nearly equal cuts for the grids that fit no other.
//
// Where the line to the split half-steps lies: past kSlowest cycles the pole
// state of a few blocks keeps all others waiting, which the split kernels
// spread over the device. 60 x 60 x 200 FP32 with a disk of radius 18 (estimate
// 24000): 13.1 against 16.8 us per step; with a sphere of radius 20 (34000)
// 20.2 against 20.6; 48 x 48 x 200 FP64, disk of radius 12 (33000) 16.7 against
// 20.1.
void aefdtd_sim::build_resident() {
    res_dirty = false;
    res.grid = 0;
    res.mem.release(dev_bytes);
    int nsm = 0, optin = 0, coop = 0;
    AE_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
    AE_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    AE_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
    const size_t es = fp64 ? 8 : 4;
    const ResKernel *kernels = fp64 ? kResKernels64 : kResKernels32;
    const size_t nkernels = fp64 ? std::size(kResKernels64) : std::size(kResKernels32);
    const ResKernel &longest = kernels[nkernels - 1];
    const size_t limit = optin > 4096 ? size_t(optin) - 1024 : 0;   // the kernel's own block record
    if (!coop || Nx > 512 || (long long)Nx * Ny * Nz > (long long)nsm * longest.threads * longest.run || Nmat > 128)
        return;
    const bool px = pml[0] || pml[1], py = pml[2] || pml[3], pz = pml[4] || pml[5];
    // dispersive cells per (plane, row), and times their poles
    std::vector<int> dc(size_t(Ny) * Nz, 0), dp(size_t(Ny) * Nz, 0);
    std::vector<char> rc(Nmat, 0);
    int poles = 0;
    long long psi_n = 0;
    for (unsigned m = 0; m < Nmat; m++) {
        const HostMat &h = mats[m];
        rc[m] = h.rc && h.np > 0;
        if (!rc[m]) continue;
        poles += h.np;
        psi_n += 3LL * h.np * (h.x2 + 1 - h.x1) * (h.y2 + 1 - h.y1) * (h.z2 + 1 - h.z1);
    }
    if (psi_n >= (1LL << 31)) return;   // the kernel addresses psi in 32 bits
    for (unsigned m = 0; m < Nmat; m++) {
        const HostMat &h = mats[m];
        if (!rc[m]) continue;
        for (int k = h.z1; k <= h.z2; k++)
            for (int j = h.y1; j <= h.y2; j++) {
                const uint32_t *row = &map[size_t(j) * Nx + size_t(k) * Nx * Ny];
                int c = 0;
                for (int i = h.x1; i <= h.x2; i++) c += row[i] == m;
                dc[size_t(k) * Ny + j] += c;
                dp[size_t(k) * Ny + j] += c * h.np;
            }
    }
    auto prefix = [&](const std::vector<int> &v) {
        std::vector<long long> p(size_t(Ny + 1) * (Nz + 1), 0);
        for (int k = 0; k < Nz; k++)
            for (int j = 0; j < Ny; j++)
                p[size_t(k + 1) * (Ny + 1) + j + 1] = v[size_t(k) * Ny + j] + p[size_t(k) * (Ny + 1) + j + 1] +
                                                      p[size_t(k + 1) * (Ny + 1) + j] - p[size_t(k) * (Ny + 1) + j];
        return p;
    };
    const std::vector<long long> sum_c = prefix(dc), sum_p = prefix(dp);
    auto within = [&](const std::vector<long long> &p, int j0, int j1, int k0, int k1) {
        return p[size_t(k1) * (Ny + 1) + j1] - p[size_t(k0) * (Ny + 1) + j1] - p[size_t(k1) * (Ny + 1) + j0] +
               p[size_t(k0) * (Ny + 1) + j0];
    };
    const double per = fp64 ? 1.25 : 0.5, per_pole = 12.0 * 2 * es / 50.0;
    auto pole_cost = [&](int j0, int j1, int k0, int k1) {
        return per_pole * within(sum_p, j0, j1, k0, k1) + 2.0 * within(sum_c, j0, j1, k0, k1);
    };
    auto in_pml = [](int i, int N, int lo, int hi) { return i < lo || i >= N - hi; };
    auto weights = [&](std::vector<double> &wy, std::vector<double> &wz, double raise, double slab) {
        wy.assign(Ny, 0.0);
        wz.assign(Nz, 0.0);
        for (int j = 0; j < Ny; j++)
            wy[j] = per * Nx * Nz * ((py && in_pml(j, Ny, pml[2], pml[3])) ? slab : 1.0) + raise * pole_cost(j, j + 1, 0, Nz);
        for (int k = 0; k < Nz; k++)
            wz[k] = per * Nx * Ny * ((pz && in_pml(k, Nz, pml[4], pml[5])) ? slab : 1.0) + raise * pole_cost(0, Ny, k, k + 1);
    };
    // sensor sites: the two plane-sum planes, then each DFT plane's box of
    // cells with the neighbours its interpolation reads
    res.nregions = 0;
    res.rec = 0;
    auto region = [&](int x1, int y1, int z1, int sx, int sy, int sz, bool h) {
        ResRegion &r = res.region[res.nregions++];
        r.base = res.rec;
        r.x1 = x1; r.y1 = y1; r.z1 = z1;
        r.sx = sx; r.sy = sy; r.sz = sz;
        r.stride = size_t(sx) * sy * sz;
        r.h = h;
        res.rec += r.stride * (h ? 6 : 3);
    };
    if (normal) {
        region(0, 0, zs_e - 2, Nx, Ny, 1, false);
        region(0, 0, zs_s, Nx, Ny, 1, false);
    }
    for (auto *p : sensors) {
        if (p->type <= 1) region(p->x1, p->y1, p->z1, 2, p->span1 + 1, p->span2 + 1, true);
        else if (p->type <= 3) region(p->x1, p->y1, p->z1, p->span1 + 1, 2, p->span2 + 1, true);
        else region(p->x1, p->y1, p->z1, p->span1 + 1, p->span2 + 1, 2, true);
    }
    // Steps per launch: at most a segment, and the sensor record within 8 MiB, or
    // within 64 with DFT planes and where 8 hold fewer than `least` steps. A
    // launch of few steps does not pay for loading and storing the state and for
    // its sensor launches; us per step of 64 steps, resident / split, where a
    // segment has 4 and 8 steps: 64 x 64 x 128 FP64 with two flux planes 30.9 /
    // 26.0 and 20.4 / 21.4, 64 x 64 x 250 FP32 31.7 / 25.0 and 18.7 / 20.0; without
    // flux planes, at 2 and 4 steps: 26.4 / 23.2 and 18.0 / 20.0, 27.8 / 23.6 and
    // 18.8 / 20.0.
    const size_t least = sensors.empty() ? 4 : 8, bytes = res.rec * es, most = size_t(64) << 20;
    res.cap = bytes ? (int)std::min<size_t>(seg_len, std::max(least, (sensors.empty() ? most / 8 : most) / bytes)) : seg_len;
    if (res.cap < (int)least || bytes * res.cap > most) return;
    // sensor sites in a block: the cells of each region's box that fall in it, with wraps
    auto sites_in = [&](const ResBlock &x) {
        size_t n = 0;
        auto hits = [](int a, int len, int lo, int hi, int N) {   // a .. a + len - 1 mod N within [lo, hi)
            int c = 0;
            for (int m = a; m < a + len;) {
                const int p = m % N, e = std::min(a + len - m, N - p);
                c += std::max(0, std::min(p + e, hi) - std::max(p, lo));
                m += e;
            }
            return c;
        };
        for (int r = 0; r < res.nregions; r++) {
            const ResRegion &g = res.region[r];
            n += size_t(g.sx) * hits(g.y1, g.sy, x.j0, x.j0 + x.by, Ny) * hits(g.z1, g.sz, x.k0, x.k0 + x.bz, Nz);
        }
        return n;
    };
    // what a block over [j0, j1) x [k0, k1) holds, for runs of at most `run` planes
    auto fill = [&](ResBlock &x, int j0, int j1, int k0, int k1, int run) {
        x.j0 = j0;
        x.by = j1 - j0;
        x.k0 = k0;
        x.bz = k1 - k0;
        x.nseg = (x.bz + run - 1) / run;
        x.nzp = std::max(0, std::min(k1, pml[4]) - k0) + std::max(0, k1 - std::max(k0, Nz - pml[5]));
        x.disp_n = (int)within(sum_c, j0, j1, k0, k1);
        const bool yp = py && (j0 < std::max(pml[2], 1) || j1 > Ny - std::max(pml[3], 1));
        unsigned f = (px || yp ? kXY : 0u) | (pz && (x.nzp > 0 || k0 == 0 || k1 == Nz) ? kZ : 0u);
        if (normal && zs_e - 1 >= k0 && zs_e - 1 < k1) f |= kInject;
        unsigned fe = f | (x.disp_n > 0 ? kDisp : 0u);
        for (auto &o : oscs)
            if (o.box[4] < k1 && o.box[5] > k0 && o.box[2] < j1 && o.box[3] > j0) fe |= kMisc;
        x.feat_e = kernel_feat(fe);
        x.feat_h = kernel_feat(f);
    };
    // psi slots of a block's runs: a run's z-CPML planes, of one end of the axis
    // (-1: a run reaches both, which its record has no room for)
    auto slots = [&](const ResBlock &x, int run) {
        int n = 0;
        for (int r = 0; pz && r < x.nseg; r++) {
            const int k = x.k0 + r * run, e = std::min(k + run, x.k0 + x.bz);
            const int low = std::min(e, pml[4]) - k, high = e - std::max(k, Nz - pml[5]);
            if (low > 0 && high > 0) return -1;
            n = std::max({n, low, high});
        }
        return n;
    };
    // shared memory: fields, z psi, halo (runs cut short read on behind it),
    // coefficients, z tables, injection values, thread records, sensor sites,
    // ids, pole sums and their ranks
    auto layout = [&](ResBlock &x, const ResKernel &K) -> size_t {
        const int run = K.run;
        x.npsi = slots(x, run);
        size_t o = size_t((K.tight ? 3 : 6) * run + 4 * x.npsi) * K.threads * es;
        x.o_halo = (int)o;
        o += up16(2 * size_t(Nx) * (x.by + x.bz) * es);
        const size_t past = o + std::max(run * Nx, K.threads) * es;
        x.o_next = (int)o;
        o += size_t(2) * K.threads * 8;
        x.o_taps = (int)o;
        o += up16(size_t(kResRegions) * sizeof(ResTaps));
        x.o_sites = (int)o;
        o += up16(sites_in(x) * sizeof(uint2));
        x.o_coef = (int)o;
        o += up16(size_t(Nmat) * 6 * es);
        x.o_z = (int)o;
        o += size_t(2) * (x.bz + run) * 4 * es;
        x.o_inject = (int)o;
        o += normal ? size_t(seg_len) * 4 * es : 0;
        x.o_ids = (int)o;
        o += size_t((run + 3) / 4) * 4 * K.threads;
        x.o_sum = (int)o;
        o += up16(size_t(x.disp_n) * 3 * es);
        x.o_rank = (int)o;
        o += x.disp_n ? up16(size_t(run) * K.threads * 2) : 0;
        x.o_disp = (int)o;
        o += size_t(x.disp_n) * 16;
        x.o_poles = (int)o;
        o += x.disp_n ? size_t(poles) * 4 * es : 0;
        x.o_stage = (int)o;
        o += x.disp_n && res_staged(run, (int)es) ? size_t(K.threads) * res_stage((int)es) * kResPoles * 6 * es : 0;
        return std::max(o, past);
    };
    // cycles of a half-step of a block of rows x planes with features f, and of a whole step
    auto half = [&](int rows, int planes, int runs, int run, unsigned f) {
        const double c = (fp64 ? run > 13 ? 30 : 20 : 11.5) * (f == 0 ? 1.0 : f & kXY ? 8.0 : f & kDisp ? 2.5 : 2.0);
        const double warps = (Nx * rows * runs + 31) / 32, n = std::min(run, planes);
        return 300 + n * std::max(warps * c, 60.0) + 40.0 * n;
    };
    auto cost = [&](const ResBlock &x, const ResKernel &K) {
        const bool staged = res_staged(K.run, (int)es);
        const double words = 2.0 * Nx * (x.by + x.bz);
        const double ante = x.disp_n == 0 ? 0
                            : staged ? (fp64 ? 3500.0 : 1700.0) * ((x.disp_n + K.threads - 1) / K.threads)
                                     : 1700.0 * ((x.disp_n + K.threads - 1) / K.threads) + pole_cost(x.j0, x.j0 + x.by, x.k0, x.k0 + x.bz);
        return (K.tight ? 200 : 0) + half(x.by, x.bz, x.nseg, K.run, x.feat_e) + half(x.by, x.bz, x.nseg, K.run, x.feat_h) +
               2 * (0.1 * words + (fp64 ? 1.5 * std::max(0.0, words - 4 * K.threads) : 0.75 * std::max(0.0, words - 8 * K.threads))) + ante;
    };
    const double kSlowest = fp64 ? 36000 : 30000;
    double best = kSlowest;
    ResKernel kernel{0, 0, false};
    std::vector<int> cy, cz;
    for (const auto &w : {std::array{1.0, 1.25}, {1.0, 1.8}, {1.0, 1.1}, {0.0, 1.5}, {4.0, 1.5}}) {
        if (w[0] != 1.0 && sum_p.back() == 0) continue;
        std::vector<double> wy, wz;
        weights(wy, wz, w[0], w[1]);
        for (int nb = 1; nb <= std::min(Ny, nsm); nb++) {
            const std::vector<int> yc = cut(wy, nb);
            int tall = 0;   // the widest band
            for (int b = 0; b < nb; b++) tall = std::max(tall, yc[b + 1] - yc[b]);
            if (Nx * tall > 512) continue;
            int tried = 0;
            for (int part : {1, 2, 4}) {
                // as many slabs as the device has room for; a half or a quarter may do for small grids
                const int ns = std::min(Nz, std::max(1, nsm / nb / part));
                if (ns == tried) continue;
                tried = ns;
                const std::vector<int> zc = cut(wz, ns);
                int deep = 0;
                for (int s = 0; s < ns; s++) deep = std::max(deep, zc[s + 1] - zc[s]);
                const double waits = nb * ns > 1 ? 2600 : 600;
                std::vector<ResBlock> x;   // filled for the first kernel that may be better
                for (size_t n = 0; n < nkernels; n++) {
                    const ResKernel &K = kernels[n];
                    const int runs = (deep + K.run - 1) / K.run;
                    if (Nx * tall * runs > K.threads) continue;
                    if (waits + 2 * half(tall, deep, runs, K.run, 0) >= best) continue;
                    double worst = waits;
                    bool better = true;
                    if (x.empty()) {
                        x.resize(size_t(nb) * ns);
                        for (int s = 0; s < ns; s++)
                            for (int b = 0; b < nb; b++) fill(x[size_t(s) * nb + b], yc[b], yc[b + 1], zc[s], zc[s + 1], K.run);
                    }
                    for (size_t m = 0; m < x.size() && better; m++) {
                        ResBlock &y = x[m];
                        y.nseg = (y.bz + K.run - 1) / K.run;
                        worst = std::max(worst, waits + cost(y, K));
                        better = y.disp_n < kResNoRank && worst < best && slots(y, K.run) >= 0 && !(K.tight && ((y.feat_e | y.feat_h) & kXY));
                    }
                    for (size_t m = 0; m < x.size() && better; m++) better = layout(x[m], K) <= limit;
                    if (!better) continue;
                    best = worst;
                    kernel = K;
                    cy = yc;
                    cz = zc;
                }
            }
        }
    }
    if (cy.empty()) return;
    const int run = kernel.run;
    const int nb = (int)cy.size() - 1, ns = (int)cz.size() - 1;
    std::vector<ResBlock> B(size_t(nb) * ns);
    auto at = [&](int s, int b) -> ResBlock & { return B[size_t((s + ns) % ns) * nb + (b + nb) % nb]; };
    size_t smem = 0;
    long long words = 0;
    int ndisp = 0;
    for (int s = 0; s < ns; s++)
        for (int b = 0; b < nb; b++) {
            ResBlock &x = at(s, b);
            fill(x, cy[b], cy[b + 1], cz[s], cz[s + 1], run);
            smem = std::max(smem, layout(x, kernel));
            x.disp_off = ndisp;
            ndisp += x.disp_n;
            x.self_y = nb == 1;
            x.self_z = ns == 1;
            // E halo, then H halo: y face, z face
            const long long n = 2LL * Nx * (x.by + x.bz);
            x.get_e = (int)words;
            x.get_h = (int)(words + n);
            words += 2 * n;
        }
    for (int s = 0; s < ns; s++)
        for (int b = 0; b < nb; b++) {
            ResBlock &x = at(s, b);
            const ResBlock &ym = at(s, b - 1), &yp = at(s, b + 1), &zm = at(s - 1, b), &zp = at(s + 1, b);
            // E goes down (to the blocks whose H reads it), H goes up
            x.put_ey = x.self_y ? -1 : ym.get_e;
            x.put_ez = x.self_z ? -1 : zm.get_e + 2 * Nx * zm.bz;
            x.put_hy = x.self_y ? -1 : yp.get_h;
            x.put_hz = x.self_z ? -1 : zp.get_h + 2 * Nx * zp.bz;
        }
    // What the device refuses (blocks that are not all resident at once, memory
    // for the plan) is no error: the split kernels run in what there is.
    int per_sm = 0;
    if ((fp64 ? prepare_resident_f64(run, (int)limit, (int)smem, per_sm)
              : prepare_resident_f32(run, (int)limit, (int)smem, per_sm)) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (per_sm * nsm < nb * ns || res.refuse == 2) return;
    std::vector<int> yb(Ny), zb(Nz);   // owner band / slab
    for (int b = 0; b < nb; b++) for (int j = cy[b]; j < cy[b + 1]; j++) yb[j] = b;
    for (int s = 0; s < ns; s++) for (int k = cz[s]; k < cz[s + 1]; k++) zb[k] = s;
    // a cell's place in its block's arrays: plane of the run, then thread
    auto cell_of = [&](const ResBlock &x, int i, int j, int k) {
        const int z = k - x.k0;
        return (z % run) * kernel.threads + (z / run) * Nx * x.by + i + Nx * (j - x.j0);
    };
    std::vector<ResDisp> disp_cells(ndisp);
    {
        std::vector<DispInfo> di(Nmat);
        if (ndisp) AE_CUDA(cudaMemcpy(di.data(), disp.p, sizeof(DispInfo) * Nmat, cudaMemcpyDeviceToHost));
        std::vector<int> fill(B.size(), 0);
        for (int k = 0; k < Nz && ndisp; k++)
            for (int j = 0; j < Ny; j++) {
                if (!dc[size_t(k) * Ny + j]) continue;
                const size_t n = size_t(zb[k]) * nb + yb[j];
                const ResBlock &x = B[n];
                const uint32_t *row = &map[size_t(j) * Nx + size_t(k) * Nx * Ny];
                for (int i = 0; i < Nx; i++) {
                    const uint32_t m = row[i];
                    if (!rc[m]) continue;
                    const DispInfo &d = di[m];
                    ResDisp &e = disp_cells[x.disp_off + fill[n]++];
                    e.place = (unsigned)cell_of(x, i, j, k) | m << 16;
                    e.psi = int(d.psi_off + (i - d.x1) + (long long)(j - d.y1) * d.xs + (long long)(k - d.z1) * d.xs * d.ys);
                }
            }
    }
    // sites per block, region by region
    std::vector<std::vector<uint2>> site(B.size());
    std::vector<std::vector<ResTaps>> part(B.size());
    for (int r = 0; r < res.nregions; r++) {
        const ResRegion &g = res.region[r];
        for (int w = 0; w < g.sz; w++)
            for (int v = 0; v < g.sy; v++) {
                const int j = (g.y1 + v) % Ny, k = (g.z1 + w) % Nz;
                const size_t n = size_t(zb[k]) * nb + yb[j];
                if (part[n].empty() || part[n].back().region != r)
                    part[n].push_back(ResTaps{(int)site[n].size(), 0, int(g.stride), g.h, r});
                for (int u = 0; u < g.sx; u++)
                    site[n].push_back(make_uint2(unsigned(cell_of(B[n], (g.x1 + u) % Nx, j, k)),
                                                 unsigned(g.base + u + size_t(g.sx) * (v + size_t(g.sy) * w))));
                part[n].back().n += g.sx;
            }
    }
    std::vector<ResTaps> taps;
    std::vector<uint2> sites;
    for (size_t n = 0; n < B.size(); n++) {
        B[n].tap_off = (int)taps.size();
        B[n].tap_n = (int)part[n].size();
        B[n].site_off = (int)sites.size();
        B[n].site_n = (int)site[n].size();
        taps.insert(taps.end(), part[n].begin(), part[n].end());
        sites.insert(sites.end(), site[n].begin(), site[n].end());
    }
    std::vector<char> host;
    auto put = [&](const void *p, size_t n) {
        const size_t o = host.size();
        host.resize((o + n + 255) / 256 * 256);
        if (n) std::memcpy(host.data() + o, p, n);
        return o;
    };
    put(B.data(), sizeof(ResBlock) * B.size());
    res.disp = put(disp_cells.data(), sizeof(ResDisp) * disp_cells.size());
    res.taps = put(taps.data(), sizeof(ResTaps) * taps.size());
    res.sites = put(sites.data(), sizeof(uint2) * sites.size());
    res.inbox = host.size();
    res.raw = (res.inbox + up16(size_t(words) * 2 * es) + 255) / 256 * 256;
    const size_t need = res.raw + res.rec * es * res.cap;
    if (res.refuse == 1 || cudaMalloc(&res.mem.p, need) != cudaSuccess) {
        cudaGetLastError();
        res.mem.p = nullptr;
        return;
    }
    res.mem.n = need;
    dev_bytes += need;
    AE_CUDA(cudaMemcpy(res.mem.p, host.data(), host.size(), cudaMemcpyHostToDevice));
    AE_CUDA(cudaMemsetAsync(res.at<char>(res.inbox), 0, res.raw - res.inbox, stream));
    res.seq = 0;
    res.smem = (int)smem;
    res.run = run;
    res.grid = nb * ns;
}

// n steps in chunks of at most res.cap, each one cooperative launch and the
// sensor launches over the sites it recorded; a chunk ends where a DFT sample
// buffer fills, and the block is accumulated at once. Returns the steps made:
// fewer than n when a launch was refused, after which res.grid is 0.
template <typename T> int aefdtd_sim::run_resident(int n) {
    for (auto *s : sensors) launch_pending<T>(*s, stream);
    std::vector<StepScalars> host(seg_len);
    int done = 0;
    while (done < n) {
        int L = std::min(n - done, res.cap);
        for (auto *s : sensors) L = std::min(L, dft_k - s->nbuf);
        StepScalars *tbl = tables.as<StepScalars>() + size_t(seg_slot) * seg_len;
        seg_slot ^= 1;
        for (int q = 0; q < L; q++) fill_scalars(tstep + q, q, host[q]);
        AE_CUDA(cudaMemcpyAsync(tbl, host.data(), sizeof(StepScalars) * L, cudaMemcpyHostToDevice, stream));
        ResArgs<T> A{};
        make_step_args(A.e, A.h, tbl);
        A.blocks = res.at<ResBlock>(0);
        A.disp = res.at<ResDisp>(res.disp);
        A.npoles = (int)(crec.n / (2 * sizeof(T)));
        A.taps = res.at<ResTaps>(res.taps);
        A.sites = res.at<uint2>(res.sites);
        A.inbox = res.at<unsigned long long>(res.inbox);
        A.raw = res.at<T>(res.raw);
        A.rec = res.rec;
        A.steps = L;
        A.seq0 = res.seq;
        res.seq += 2u * (unsigned)L + 2u;
        A.abort = err.as<int>() + 1;
        A.wait_cycles = res.wait_cycles;
        A.withhold = res.withhold;
        const cudaError_t refused =
            res.refuse == 3 ? cudaErrorCooperativeLaunchTooLarge : launch_resident(A, res.run, res.grid, res.smem, stream);
        // fewer SMs for this process than the device has, or no memory for the kernel's stack
        if (refused == cudaErrorCooperativeLaunchTooLarge || refused == cudaErrorLaunchOutOfResources ||
            refused == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            res.release(dev_bytes);
            return done;
        }
        AE_CUDA(refused);
        launches++;
        int reg = 0;
        if (normal) {
            SensorStepArgs<T> sa;
            make_sensor_args(sa, tbl);
            launch_resident_planes(sa, res.at<T>(res.raw), res.rec, L, stream);
            launch_plane_reduce(psum_partial.as<double>(), sa.nbp, tbl, psums.as<double>(), L, stream);
            launches += 2;
            reg = 2;
        }
        for (PlaneSensor *s : sensors) {
            const ResRegion &r = res.region[reg++];
            if (s->nbuf == 0) s->buf_step0 = s->step;
            ResGatherArgs<T> g{};
            g.raw = res.at<T>(res.raw) + r.base;
            g.rec = res.rec;
            g.stride = r.stride;
            g.sx = r.sx; g.sy = r.sy; g.sz = r.sz;
            g.type = s->type;
            g.span1 = s->span1;
            g.P = s->P;
            g.S = s->S.as<T>() + (size_t(s->half) * dft_k + s->nbuf) * 6 * s->P;
            launch_resident_gather(g, L, stream);
            launches++;
            s->nbuf += L;
            s->step += L;
            if (s->nbuf == dft_k) {
                flush_block<T>(*s, s->half, dft_k, nullptr, s->buf_step0, stream);
                s->nbuf = 0;
            }
        }
        for (auto &o : oscs) o.step += L;
        tstep += L;
        done += L;
    }
    AE_CUDA(cudaGetLastError());
    return done;
}
template int aefdtd_sim::run_resident<double>(int);
template int aefdtd_sim::run_resident<float>(int);
