// post.cu — per-pixel finalisation in FP64.
//
//   k_ipss      IPSS spherical single-scatter correction kappa and the
//               ray-traced direct-beam slant depth (rt_ipss.c:24-644), one
//               thread per line-of-sight quadrature node, a pixel's nodes over
//               several blocks
//   k_finalize  Fourier reconstruction (rt_fourier.c:9-33), rho = X/mu0, kappa,
//               direct sunglint (shared/surface.c:1813-1907) and the
//               transmittance diagnostics (rt_solver.c:1100-1275), a warp per
//               pixel with the modes over its lanes
//
// Everything here is FP64, which issues at about 2 lanes per clock and SM on
// this part, so the bound is the FP64 pipe of the SMs that take part: the
// node sums skip the shells below a node where they hold no path, prefix sums
// and the plane-parallel sum run over threads, mirrored azimuths of a LUT grid
// are evaluated once, and a single pixel's nodes are spread over many SMs.
// Whole solves: look-up tables of 3 pixels x 5040 directions x 100 layers
// 21.9 -> 6.6 ms by this alone (5.2 ms with the rest of the solve as it is now), a 400-layer
// pixel with 242 modes 8.4 -> 5.2 ms (1.6 now).
#include "kernels.cuh"
#include "physics.cuh"

#define IPSS_RE 6371.0

// Slant optical depth from rB toward the sun; +inf when the ray meets the
// ground (shadow).  Per-shell path lengths are taken in closed form: with
// tau' = t + b and p^2 = |rB|^2 - b^2, shell j holds |tau'| in [A_j, A_j+1],
// A = sqrt(max(0, R^2 - p^2)), intersected with tau' > b.  This is the
// reference's sorted-crossing sum (rt_ipss.c:233-318) regrouped by shell.
// R[0..nl]: shell radii; j0: the shell that holds rB (0 when unknown).  With
// the sun above rB's horizon (b >= 0) the ray leaves upward and the shells
// below j0 hold no path, so the sum starts there.
__device__ double ipss_tau_sun(const double *R, const double *beta, int nl, double mu0, const double *rB, int j0)
{
    const double sn = sqrt(fmax(0.0, 1.0 - mu0 * mu0));
    const double un = sqrt(sn * sn + mu0 * mu0);
    const double ux = -sn / un, uz = mu0 / un;
    const double b = rB[0] * ux + rB[2] * uz;
    const double c0 = rB[0] * rB[0] + rB[1] * rB[1] + rB[2] * rB[2];
    const double dg = b * b - (c0 - IPSS_RE * IPSS_RE);
    if (dg >= 0.0) {
        const double sq = sqrt(dg);
        if (-b - sq > 1e-9 || -b + sq > 1e-9) return INFINITY;
    }
    const double p2 = c0 - b * b;
    double tau = 0.0;
    if (b >= 0.0) {
        double Alo = b;
        for (int j = j0; j < nl; ++j) {
            const double d2 = R[j + 1] * R[j + 1] - p2;
            const double Ahi = d2 > 0.0 ? sqrt(d2) : 0.0;
            if (Ahi > Alo) { tau += (Ahi - Alo) * beta[j]; Alo = Ahi; }
        }
        return tau;
    }
    double Alo = sqrt(fmax(0.0, R[0] * R[0] - p2));
    for (int j = 0; j < nl; ++j) {
        const double d2 = R[j + 1] * R[j + 1] - p2;
        if (d2 > 0.0) {
            const double Ahi = sqrt(d2);
            // branch tau' in [Alo, Ahi] with tau' > b
            double len = 0.0;
            const double a1 = fmax(Alo, b);
            if (Ahi > a1) len += Ahi - a1;
            // branch tau' in [-Ahi, -Alo] with tau' > b
            const double a2 = fmax(-Ahi, b);
            if (-Alo > a2) len += -Alo - a2;
            tau += len * beta[j];
            Alo = Ahi;
        } else {
            Alo = 0.0;
        }
    }
    return tau;
}

// Block-wide inclusive prefix sums of v[0..n) in place (n any, blockDim a
// multiple of 32, at most 1024).  red: 33 doubles.
__device__ void block_prefix(double *v, int n, double *red)
{
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
    const int per = (n + blockDim.x - 1) / blockDim.x, b = min(n, tid * per), e = min(n, b + per);
    double s = 0.0;
    for (int i = b; i < e; ++i) { s += v[i]; v[i] = s; }
    double x = s;
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) red[w] = x;
    __syncthreads();
    if (w == 0) {
        double t = lane < nw ? red[lane] : 0.0;
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        red[lane] = t;
    }
    __syncthreads();
    const double off = (w ? red[w - 1] : 0.0) + x - s;
    for (int i = b; i < e; ++i) v[i] += off;
    __syncthreads();
}

// Sum over the block, valid in every thread.
__device__ double block_sum_d(double v, double *red)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    return t;
}

struct IpssMem { double *R, *beta, *wsrc, *above, *lt, *ltau, *red; };

// shared-memory doubles of the IPSS kernels at nl layers
size_t ipss_smem_bytes(int nl) { return sizeof(double) * (6 * ((size_t)nl + 1) + 40); }

__device__ inline IpssMem ipss_mem(double *sm, int nl)
{
    IpssMem m;
    m.R = sm; m.beta = m.R + nl + 1; m.wsrc = m.beta + nl + 1; m.above = m.wsrc + nl + 1;
    m.lt = m.above + nl + 1; m.ltau = m.lt + nl + 1; m.red = m.ltau + nl + 1;
    return m;
}

// What does not depend on the view direction: shell radii, extinction per km
// of the layers in ascending altitude, vertical depth above every shell edge.
// Returns whether any layer holds aerosol.
__device__ int ipss_pixel(const PixDev &d, const double *h, const double *z, const double *xd, const IpssMem &m)
{
    const int nl = d.nt;
    const long long lo = d.lev_off;
    for (int k = threadIdx.x; k <= nl; k += blockDim.x) m.R[k] = IPSS_RE + z[lo + nl - k];
    int have = 0;
    for (int j = threadIdx.x; j < nl; j += blockDim.x) {
        const int k = nl - 1 - j;
        const double dz = z[lo + k] - z[lo + k + 1], dtau = h[lo + k + 1] - h[lo + k];
        const double be = (dz > 0.0 && dtau > 0.0) ? dtau / dz : 0.0;
        m.beta[j] = be;
        m.above[nl - 1 - j] = be * dz;               // from the top down, for the prefix sum
        if (xd[lo + k + 1] > 0.0) have = 1;
    }
    have = __syncthreads_or(have);
    block_prefix(m.above, nl, m.red);                // above[i]: depth above edge nl - 1 - i
    return have;
}

// One view direction by the whole block (after ipss_pixel): the partial
// line-of-sight sum of the nodes q0, q0 + qstep, ... of this thread, and, when
// pp is set, the plane-parallel sum.  Both are block sums.
__device__ void ipss_view(const PixDev &d, int have_aer, double vza_deg, double raa_deg, const double *h,
                          const double *xd, const double *yd, const double *tabs, const double *mb,
                          const double *vk_th, const double *vk_p11, const IpssMem &m, int q0, int qstep, bool pp,
                          double *Iss_out, double *Ipp_out)
{
    const int nl = d.nt;
    const long long lo = d.lev_off;
    const double tv = vza_deg * OCRT_PI / 180.0, fp = (180.0 - raa_deg) * OCRT_PI / 180.0;
    const double sv = sin(tv), cv = cos(tv), cfp = cos(fp), sfp = sin(fp);
    const int use_w = have_aer && d.mom_off >= 0 && d.tau_a > 0.0;
    double PR = 1.0, PA = 1.0;
    if (use_w) {
        const double sn = sqrt(fmax(0.0, 1.0 - d.mu0 * d.mu0));
        const double ct = sn * sv * cfp - d.mu0 * cv;
        PR = 1.0 + (1.0 - OCRT_DEPOL) / (2.0 + OCRT_DEPOL) * 0.5 * (3.0 * ct * ct - 1.0);
        if (d.vk_n > 1 && vk_th) {
            // the value kernel's table, linear in the angle (rt_ipss.c:131-146)
            const double *th = vk_th + d.vk_off, *pv = vk_p11 + d.vk_off;
            const int n = d.vk_n;
            const double t = acos(fmax(-1.0, fmin(1.0, ct))) * 180.0 / OCRT_PI;
            if (t <= th[0]) {
                PA = pv[0];
            } else if (t >= th[n - 1]) {
                PA = pv[n - 1];
            } else {
                int lo = 0, hi = n - 1;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (th[mid] <= t) lo = mid; else hi = mid;
                }
                PA = pv[lo] + (t - th[lo]) / (th[hi] - th[lo]) * (pv[hi] - pv[lo]);
            }
        } else {
            // Legendre sum of the aerosol moments: one thread, then broadcast
            // (a serial FP64 recurrence; every thread would queue on the same pipe)
            if (threadIdx.x == 0) {
                double p0 = 1.0, p1 = ct, s = mb[d.mom_off];
                if (d.L_aer >= 1) s += mb[d.mom_off + 1] * p1;
                for (int l = 2; l <= d.L_aer; ++l) {
                    const double p2 = ((2.0 * l - 1.0) * ct * p1 - (l - 1.0) * p0) / l;
                    s += mb[d.mom_off + l] * p2; p0 = p1; p1 = p2;
                }
                m.red[36] = s > 0.0 ? s : 0.0;
            }
            __syncthreads();
            PA = m.red[36];
        }
    }
    // line of sight, pixel anchored (rt_ipss.c:495-521): radius decreases
    // monotonically from the TOA crossing to the pixel, one crossing per shell
    const double u0 = sv * cfp, u1 = sv * sfp, u2 = cv;
    const double Rt = m.R[nl], H = Rt - IPSS_RE;
    const double bq = IPSS_RE * u2;
    const double disc = bq * bq + Rt * Rt - IPSS_RE * IPSS_RE;
    const double smax = -bq + sqrt(disc);
    const double rA[3] = {smax * u0, smax * u1, IPSS_RE + smax * u2};
    const double bl = -(rA[0] * u0 + rA[1] * u1 + rA[2] * u2);
    const double c0l = rA[0] * rA[0] + rA[1] * rA[1] + rA[2] * rA[2];
    // crossing i (0 = TOA at s = 0, nl = pixel at s = smax) at shell edge
    // nl - i; interval i lies in shell nl - 1 - i
    for (int i = threadIdx.x; i <= nl; i += blockDim.x) {
        if (i == 0) m.lt[i] = 0.0;
        else if (i == nl) m.lt[i] = smax;
        else {
            const double R = m.R[nl - i];
            m.lt[i] = -bl - sqrt(bl * bl - (c0l - R * R));
        }
    }
    for (int j = threadIdx.x; j < nl; j += blockDim.x) {
        const int k = nl - 1 - j;
        double w;
        if (use_w) {
            const double wr = yd[lo + k + 1] > 0.0 ? yd[lo + k + 1] : 0.0;
            const double wa = xd[lo + k + 1] > 0.0 ? xd[lo + k + 1] : 0.0;
            w = wr * PR + wa * PA;
        } else if (tabs && d.gas) {
            // the layer's scattering fraction of its extinction (rt_ipss.c:64-70)
            const double dtau = h[lo + k + 1] - h[lo + k];
            const double ta = fmin(fmax(tabs[lo + k], 0.0), dtau);
            w = dtau > 0.0 ? (dtau - ta) / dtau : 0.0;
        } else {
            w = m.beta[j] > 0.0 ? 1.0 : 0.0;
        }
        m.wsrc[j] = w;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nl; i += blockDim.x) m.ltau[i] = (m.lt[i + 1] - m.lt[i]) * m.beta[nl - 1 - i];
    __syncthreads();
    block_prefix(m.ltau, nl, m.red);                 // ltau[i]: depth along the view up to crossing i + 1
    const double xq = 1.0 / sqrt(3.0);
    double Iss = 0.0, Ipp = 0.0;
    for (int q = q0; q < 2 * nl; q += qstep) {
        const int i = q >> 1;
        const int j = nl - 1 - i;
        if (!(m.beta[j] > 0.0)) continue;
        const double sa = m.lt[i], sb = m.lt[i + 1];
        const double hw = 0.5 * (sb - sa), mid = 0.5 * (sa + sb);
        const double sq = mid + hw * ((q & 1) ? xq : -xq);
        const double rB[3] = {rA[0] - sq * u0, rA[1] - sq * u1, rA[2] - sq * u2};
        const double hB = sqrt(rB[0] * rB[0] + rB[1] * rB[1] + rB[2] * rB[2]) - IPSS_RE;
        if (hB < 0.0 || hB > H) continue;
        const double tview = (i ? m.ltau[i - 1] : 0.0) + (sq - sa) * m.beta[j];
        const double tsun = ipss_tau_sun(m.R, m.beta, nl, d.mu0, rB, j);
        if (!isfinite(tsun)) continue;
        Iss += hw * m.beta[j] * m.wsrc[j] * exp(-tview - tsun);
    }
    if (pp && cv > 0.0) {
        const double C = 1.0 / cv + 1.0 / d.mu0;
        for (int j = threadIdx.x; j < nl; j += blockDim.x) {
            if (!(m.beta[j] > 0.0)) continue;
            // depths above the layer's upper (j + 1) and lower (j) edges
            const double up = j + 1 < nl ? m.above[nl - 2 - j] : 0.0, dn = m.above[nl - 1 - j];
            Ipp += m.wsrc[j] / (cv * C) * (exp(-C * up) - exp(-C * dn));
        }
    }
    *Iss_out = block_sum_d(Iss, m.red);
    if (pp) *Ipp_out = block_sum_d(Ipp, m.red);
    __syncthreads();
}

__device__ inline double ipss_ratio(double Iss, double Ipp)
{
    return (!(Ipp > 1.0e-300) || !isfinite(Iss)) ? 1.0 : Iss / Ipp;
}

// Grid (IPSS_SPLIT, P): block s takes the nodes s * blockDim + tid, + IPSS_SPLIT *
// blockDim, ... of the pixel's own view; part[p][s] its sum, and block 0 the
// plane-parallel sum at part[p][IPSS_SPLIT] and the slant depth.  k_finalize
// adds the parts in order.
__global__ void k_ipss(const PixDev *px, int P, const double *h, const double *z,
                       const double *xd, const double *yd, const double *tabs,
                       const double *mb, const double *vk_th, const double *vk_p11, double *part, double *tau_dir)
{
    extern __shared__ double sm[];
    const int p = blockIdx.y;
    if (p >= P) return;
    const PixDev &d = px[p];
    double *dst = part + (size_t)p * (IPSS_SPLIT + 1);
    if (!d.pssa || (int)(blockIdx.x * blockDim.x) >= 2 * d.nt) {
        if (threadIdx.x == 0) {
            dst[blockIdx.x] = 0.0;
            if (blockIdx.x == 0) tau_dir[p] = -1.0;
        }
        return;
    }
    const IpssMem m = ipss_mem(sm, d.nt);
    const int have = ipss_pixel(d, h, z, xd, m);
    double Iss = 0.0, Ipp = 0.0;
    ipss_view(d, have, d.vza_deg, d.raa_deg, h, xd, yd, tabs, mb, vk_th, vk_p11, m, blockIdx.x * blockDim.x + threadIdx.x,
              IPSS_SPLIT * blockDim.x, blockIdx.x == 0, &Iss, &Ipp);
    if (threadIdx.x == 0) {
        dst[blockIdx.x] = Iss;
        if (blockIdx.x == 0) {
            dst[IPSS_SPLIT] = Ipp;
            const double r0[3] = {0.0, 0.0, IPSS_RE};
            const double td = ipss_tau_sun(m.R, m.beta, d.nt, d.mu0, r0, 0);
            tau_dir[p] = isfinite(td) ? td : -1.0;
        }
    }
}

// The correction is even about the principal plane, so an azimuth r and its mirror
// image 360 - r share one evaluation; this key (exact: r is at least 180 where it is
// subtracted) is equal for exactly those.
__device__ __forceinline__ double ipss_azimuth_key(double r) { return r > 180.0 ? 360.0 - r : r; }

// IPSS kappa at every (vza, raa) of each pixel's LUT grid: blocks stride over
// the directions of a pixel.  The first azimuth of a key, in whatever order the grid
// lists them, is evaluated and written to every entry with that key, so each entry
// has one writer.
__global__ void k_ipss_lut(const PixDev *px, int P, const double *h, const double *z, const double *xd,
                           const double *yd, const double *tabs, const double *mb, const double *vk_th,
                           const double *vk_p11, const double *lut_vza, const double *lut_raa, double *lut_kappa)
{
    extern __shared__ double sm[];
    const int p = blockIdx.y;
    if (p >= P) return;
    const PixDev &d = px[p];
    const int npts = d.lut_nv * d.lut_nr;
    double *out = lut_kappa + d.lut_oo;
    if (!d.pssa) {
        for (int pt = blockIdx.x * blockDim.x + threadIdx.x; pt < npts; pt += gridDim.x * blockDim.x) out[pt] = 1.0;
        return;
    }
    const IpssMem m = ipss_mem(sm, d.nt);
    const double *raa = lut_raa + d.lut_ro;
    int have = -1;
    for (int pt = blockIdx.x; pt < npts; pt += gridDim.x) {
        const int iv = pt / d.lut_nr, ir = pt - iv * d.lut_nr;
        const double r = raa[ir], key = ipss_azimuth_key(r);
        int before = 0;
        for (int k = threadIdx.x; k < ir; k += blockDim.x) before |= ipss_azimuth_key(raa[k]) == key;
        if (__syncthreads_or(before)) continue;
        if (have < 0) have = ipss_pixel(d, h, z, xd, m);
        double Iss = 0.0, Ipp = 0.0;
        ipss_view(d, have, lut_vza[d.lut_vo + iv], r, h, xd, yd, tabs, mb, vk_th, vk_p11, m, threadIdx.x, blockDim.x,
                  true, &Iss, &Ipp);
        const double kap = ipss_ratio(Iss, Ipp);
        for (int k = ir + threadIdx.x; k < d.lut_nr; k += blockDim.x)
            if (ipss_azimuth_key(raa[k]) == key) out[iv * d.lut_nr + k] = kap;
    }
}

// A block of three warps per pixel, whose FP64 chains run side by side: the Fourier
// sums (lane l takes the modes l, l + 32, ...; the IPSS parts, kpart, nullptr
// without IPSS, are added in order), the direct sunglint, the transmittances.  One
// pixel: 32 us, 40 with one warp.
__global__ void __launch_bounds__(96) k_finalize(const PixDev *px, int P, const TaskState *state, const TaskOut *tout,
                           const double *gmu, const double *gw, const double *h,
                           const double *kpart, const double *tau_dir, ocrt_result *res)
{
    __shared__ double sg[3], sT[2];
    const int p = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (p >= P) return;
    const PixDev &d = px[p];
    const int M = d.M;
    const double mu0 = d.mu0, tau = d.tau_total;
    const double td = d.pssa ? tau_dir[p] : -1.0;
    double I = 0, Q = 0, U = 0, Dn = 0;
    int max_orders = 0, conv = 1, om = 0;
    if (warp == 1) {
        if (lane == 0 && d.surface == 2) {
            const double phi_v = (d.raa_deg - 180.0) * OCRT_PI / 180.0;
            const double mv = d.vza_deg > 0.0 ? d.mu_view : 1.0;
            double g[3];
            sunglint(d, mv, phi_v, tau, g);
            const double cg = td >= 0.0 ? exp(-(td - tau / mu0)) : 1.0;
            for (int i = 0; i < 3; ++i) sg[i] = g[i] * cg;
        }
    } else if (warp == 2) {
        if (lane < 2) sT[lane] = lane == 0 ? (td >= 0.0 ? exp(-td) : exp(-tau / mu0))
                                           : exp(-tau / (d.mu_view > 0.0 ? d.mu_view : 1.0));
    } else {
        const double phi = d.raa_deg * OCRT_PI / 180.0 + OCRT_PI;
        for (int m = lane; m <= M; m += 32) {
            const TaskOut &o = tout[d.task0 + m];
            const TaskState &st = state[d.task0 + m];
            double cm, sm;
            sincos((double)m * phi, &sm, &cm);
            cm = m == 0 ? 1.0 : 2.0 * cm;
            sm = m == 0 ? 0.0 : 2.0 * sm;
            I += cm * o.vI; Q += cm * o.vQ; U += sm * o.vU;
            Dn += cm * o.dn_view;
            if (st.orders > max_orders) max_orders = st.orders;
            if (!st.converged) conv = 0;
            om += st.orders;
        }
        for (int o = 16; o > 0; o >>= 1) {
            I += __shfl_xor_sync(0xffffffffu, I, o);
            Q += __shfl_xor_sync(0xffffffffu, Q, o);
            U += __shfl_xor_sync(0xffffffffu, U, o);
            Dn += __shfl_xor_sync(0xffffffffu, Dn, o);
        }
        max_orders = __reduce_max_sync(0xffffffffu, max_orders);
        conv = __reduce_min_sync(0xffffffffu, conv);
        om = __reduce_add_sync(0xffffffffu, om);
    }
    __syncthreads();
    if (threadIdx.x) return;
    ocrt_result r;
    memset(&r, 0, sizeof(r));
    r.I_TOA = I; r.Q_TOA = Q; r.U_TOA = U;
    r.rho_I = I / mu0; r.rho_Q = Q / mu0; r.rho_U = U / mu0;
    r.tau_R_total = d.tau_r;
    r.kappa_ipss = 1.0;
    if (d.pssa) {
        const double *kp = kpart + (size_t)p * (IPSS_SPLIT + 1);
        double Iss = 0.0;
        for (int s = 0; s < IPSS_SPLIT; ++s) Iss += kp[s];
        const double k = ipss_ratio(Iss, kp[IPSS_SPLIT]);
        r.kappa_ipss = k;
        r.rho_I *= k; r.rho_Q *= k; r.rho_U *= k;
        r.I_TOA *= k; r.Q_TOA *= k; r.U_TOA *= k;
    }
    if (d.surface == 2) {
        const double g[3] = {sg[0], sg[1], sg[2]};
        if (!d.decouple) { r.rho_I += g[0]; r.rho_Q += g[1]; r.rho_U += -g[2]; }
        if (d.wind > 0.0) {
            r.T_sg_up_dir = g[0] * mu0;
            r.rho_glint_direct_I = g[0]; r.rho_glint_direct_Q = g[1]; r.rho_glint_direct_U = g[2];
        }
    }
    r.n_orders_used = max_orders;
    r.converged = conv;
    r.order_modes = om;
    r.T_dir_dn = sT[0];
    r.T_diff_dn_hemi = 2.0 * OCRT_PI * tout[d.task0].fdn / (OCRT_PI * mu0);
    r.T_total_dn_hemi = r.T_dir_dn + r.T_diff_dn_hemi;
    r.T_diff_dn_dir = 2.0 * OCRT_PI * d.mu_view * Dn / (OCRT_PI * mu0);
    r.T_total_up_dir = r.rho_I * mu0;
    r.T_dir_up_view = sT[1];
    res[p] = r;
}
