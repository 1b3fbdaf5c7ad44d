// orders.cu — the successive orders of a task (pixel, Fourier mode) in one
// persistent kernel: source contraction on tcgen05 (rt_sos_operator.c:206-424),
// surface boundary condition (rt_surface_boundary.c:137-208), linear-in-tau
// transport (rt_layer_transport.c:107-208), order totals and the convergence
// test (rt_solver.c:2178-2197, 2923-3150), order after order without leaving
// the CTA.
//
// Tasks are independent, and what an order of a task reads is small: its
// operator (120 KB here) and its field (33 x 6 columns x levels).  Sweeping one
// order over all tasks at a time (k_source_tc, k_scan_tma) reads both from HBM
// and writes the source J for the scan to read back, about 1.1 MB per task and
// order at 200 levels.  Here a CTA takes a task through all of its orders: the
// operator sits in shared memory, the field makes its round trip through L2,
// the source never leaves tensor memory, and there are no per-order launches,
// lists or host polls.
//
// Parity form.  Mirroring the hemispheres (up <-> down, U -> -U) leaves the
// phase operator unchanged, so with F+- = F_up +- sigma F_dn (sigma = 1, 1, -1
// for I, Q, U) it splits into two blocks of half the size:
//     D+- = A+- (x F+-),  J_up = D+ + D-,  J_dn = sigma (D+ - D-)
// (x the aerosol fraction of the level; with a molecular term, m <= 2, it is
// applied to J instead),
// half the multiplications and half the operator.  A+- are the even- and
// odd-(l + m) sums of the phase tables.  Operands are three bf16 pieces each
// (split_bf16x3) and six products (all but those below 2^-26): FP32-level
// accuracy at the cost of 3xTF32 in tensor time and 3/4 of its shared memory.
// Per task: D+-[row][level] (FP32 in TMEM), rows = 3N Gauss outputs (s, g), 3E
// zero-weight outputs and, for m <= 2, three molecular functionals (xi_A, xi_B,
// xi_0), which give the molecular source as row factor x xi.
//
// Measured, 384 pixels x 33 modes at 32 streams and 50 to 400 levels (65181
// order-modes, rough surface, aerosol): 6.9 ms for all orders against 19.2 ms
// of order-1, source and scan passes; 500 pixels x 17 modes at 24 streams, which the
// tensor-core source does not take, 3.6 ms against 20 ms of CUDA-core source,
// molecular, order-1 and scan passes; one pixel at 400 levels 0.38 ms against 1.7 ms.  What bounds it is an
// order's serial chain, 29 000 cycles at 201 levels: 9 000 to the first tile (field
// rows back from L2, then per stage 1500 to split it, 1500 of MMA and 600 of
// barriers, two stages in flight), 6 700 to the second, 11 000 for the upward scan
// of both (60 cycles a level while the other roles run, 48 alone), 2 500 for
// residual and restart.  An MMA of 128 rows takes 62 cycles at 112 as at 80 levels
// (its operands' shared-memory reads), so tiles of 80 with three stages and three
// in TMEM were slower (7.9 ms), as were 8-level units per producer (7.4).  Order 1
// is 0.7 ms of it.
// The accumulator truncates at every step, so the incoming components are taken in
// the order U, Q, I: the sums stay small until the largest products, which come last.
// Against FP64 solves (96 pixels each, black, rough and flat surfaces) the error of the
// reflectance is 8.0, 7.6, 7.2 and 6.3e-7 rms at 8, 12, 24 and 28 streams, with FP32
// CUDA-core products 8.4, 8.2, 7.6 and 8.0e-7 (in the order I, Q, U 8.2, 7.8, 7.9 and
// 7.6e-7); at 16 and 32 streams 6.6 and 6.3e-7 (7.0 and 6.9e-7).
//
// Direct form (G.direct, groups with water columns).  Where the phase function is
// so forward-peaked that A+ and A- nearly cancel in what goes up, and the order
// sum feeds on it, the rounding of D+- at the size of the forward peak shows: the
// water-leaving reflectance of absorbing water was up to 2.9e-5 off at 32 streams.  There the
// two blocks are S = A+ + A- and B = A+ - A-, the field enters as F_up and
// sigma F_dn, and both outputs take both products: twice the MMAs (64 coupled
// pixel-bands 8.6 -> 10.2 ms of this kernel), and an error of at most 8e-6 at 32
// streams over eight such columns, 6e-6 with the separate passes.  In the atmosphere
// the two forms are equally far from FP64 (3.2e-6 rms at 32 streams for
// aerosols of g = 0.85..0.93), so it keeps the parity form.
//
// Levels run along the MMA's N, so a thread of a scan warp owns one output row
// and finds the levels of its recurrence in consecutive TMEM columns.  Tiles
// of 112 levels arrive in the order 0, T-1, 1, T-2, ...: the downward scan
// starts at the top and the upward one at the bottom while the other tiles are
// still being multiplied.  Two tiles fit in TMEM; a tile a scan cannot use yet
// is kept if no later tile needs its place, else its source rows go to J.
//
// Roles (16 warps, one CTA per SM; four warps per scheduler, so 128 registers a
// thread):
//   warps 0-3    order 1 and upward scan (TMEM lane quadrant = warp)
//                (the direction that ends at the surface sums its boundary condition)
//   warps 4-7    the same downward
//   warps 8-14   producers, 16 levels each: field rows of a tile and one incoming Stokes
//                component (loaded a stage ahead) -> F+-, split, swizzled
//                K-major B tile (128-byte rows: [F+ 32 | F- 32]) of a 2-stage ring
//   warp 15      issues the MMAs
// Thread 0 fetches tasks, starts the copy of a task's operator and posts one command per order (continue, new task,
// stop) when the order's field is complete.
//
// Every wait on an mbarrier is bounded (TC_WAIT_NS): a warp whose wait runs out raises
// the abort flag and goes on through the same barriers; all roles leave at the next
// order, record OCRT_ERR_DEVICE and free TMEM.  Named barriers have no bound, so
// warps that meet at one must decide alike: any role may raise the flag at any time,
// therefore the scan warps act on thread 0's one reading per order, which the
// end-of-order barrier publishes, and the other warps decide by vote.
//
// Adjoint (OR_ADJ).  The adjoint's orders a_{j+1} = S^T mu_j, mu_j the transposed
// transport of a_j (k_adj_scan), in units of the quadrature weights, b = a / w and
// f = mu / w: the phase matrix is symmetric under exchange of its directions
// (the sums X, Y of a pair are each other's transposes), so S^T in these units is the
// forward operator itself, molecular functionals included, and the same tiles,
// producers and MMAs serve.  Only the recurrence differs: nu = b + T nu', f = Ca nu +
// Cb nu', the upward columns from the top down and the downward ones from the
// bottom up, so the two scan directions trade columns; the surface sends
// nu of the upward columns at the bottom into b of the downward ones; the total of
// a at every level is kept for the gradients.  Measured, gradients of 96 pixels x 33
// modes x 3 rows at 32 streams and 200 levels: forward 2.9 ms and adjoint 4.8 ms,
// 6.3 and 9.5 ms with the separate passes; gradients of 7 pixels at 16 streams and 40
// levels 1.53 ms a step, 3.04 before.
#include <cuda.h>
#include <cstdint>
#include "kernels.cuh"
#include "tcgen05.cuh"

using namespace tcg;

#define OR_TS 112                     // levels of a tile
#define OR_THREADS 512
#define OR_GRP 16                     // levels per TMEM load
#define OR_BPIECE (OR_TS * 128)       // bytes of one bf16 piece of a B stage
#define OR_BSTAGE (3 * OR_BPIECE)

size_t orders_smem_bytes(const Geom &G, int Kmax)
{
    const size_t kp = (Kmax + OR_GRP + 3) & ~3;
    return par_bytes(G) + 2 * (size_t)OR_BSTAGE + 2 * kp * 4 + 2 * 2 * 3 * OR_TS * 4 + 3 * 128 * 4 + 2 * 8 * 8 + 128;
}

namespace {

__device__ __forceinline__ void or_bar(int id, int n)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Tile of arrival a of T: 0, T-1, 1, T-2, ...
__device__ __forceinline__ int or_tile(int a, int T) { return (a & 1) ? T - 1 - (a >> 1) : a >> 1; }

// What a scan thread reads: its row's factors and where its rows lie.
struct Scan {
    float T, Ca, Cb;                  // transport weights of a uniform column
    // The downward source of U is -x (D+ - D-): the sign sg sits in the weights
    // Ca, Cb and in what the source-only pass writes.
    float sg;
    float cm, c0;                     // molecular row factors of xi_A / xi_B and xi_0
    // source = D+ + kq D- upward, kq D+ + km D- downward: 1, -1, or in the direct
    // form 0, 1
    float kq, km;
    const float *xs, *ys;             // aerosol / molecular fractions per level
    const float *wT, *wA, *wB;        // per-layer weights of the slot (non-uniform columns)
    float *F, *Js, *Tot;              // field, source-spill and total columns
    float w;                          // quadrature weight (adjoint)
    int nt, NR;
    bool st, ok, uni, mol;            // row stored in the field; row valid; uniform column; m <= 2
};
// and what it carries along its column: radiance, source of the level before,
// max |I|; in the adjoint the transposed radiance, what the surface adds at the
// bottom, and the largest |source| and |total|
struct Col { float I, Jp, mi, mt; };

enum { OR_SCAN, OR_SPILL, OR_FROM_J };


// A tile of n levels from k0 in direction H (0: from the bottom up), 16 levels
// at a time: the source from TMEM at t (D+ at columns 0.., D- at 128..) or
// (OR_FROM_J) from a tile spilled before, then the recurrence, or (OR_SPILL) the
// source to J.  Groups that lie wholly inside a uniform column take a form
// without masks.  There is one copy of this code per direction, and it is kept
// short: the SM's instruction cache has to hold the loops of all roles (with
// the cases specialised the kernel was 200 KB and every loop ran at an eighth
// of its issue rate).
template <int H, int LDC, int MODE>
__device__ __forceinline__ void or_tile_run(const Scan &c, Col &v, int what, uint32_t t, int k0, int n, float ssg,
                                            const float *xa, const float *x0)
{
    constexpr bool ADJ = MODE == OR_ADJ, RMW = MODE == OR_TOT || ADJ;
    constexpr int HC = ADJ ? 1 - H : H;                    // hemisphere of the columns
    const int nt = c.nt, ng = (n + 15) >> 4;
    const float T0 = c.T, A0 = c.Ca, B0 = c.Cb;
    float I = v.I, Jp = v.Jp, mi = v.mi, mt = v.mt;
#pragma unroll 1
    for (int q = 0; q < ng; ++q) {
        // opaque to the compiler: left loop-invariant, these conditions would be
        // unswitched into a copy of the loop per combination
        int w = what, mol = c.mol, uni = c.uni;
        asm volatile("" : "+r"(w), "+r"(mol), "+r"(uni));
        const int gb = 16 * (H == 0 ? ng - 1 - q : q), kb = k0 + gb, nv = nt - kb;   // levels kb .. kb + min(15, nv) exist
        float J[16], tot[RMW ? 16 : 1];
        if (RMW && w != OR_SPILL) {
            const float *p = c.Tot + (size_t)kb * LDC;
#pragma unroll
            for (int i = 0; i < 16; ++i) tot[RMW ? i : 0] = (ADJ ? c.st : c.ok) && i <= nv ? p[i * LDC] : 0.f;
        }
        if (w == OR_FROM_J) {
            const float *p = c.Js + (size_t)kb * LDC;
#pragma unroll
            for (int i = 0; i < 16; ++i) J[i] = c.ok && i <= nv ? p[i * LDC] : 0.f;
        } else {
            uint32_t P[16], M[16];
            tmem_ld16_async(t + gb, P);
            tmem_ld16_async(t + 128 + gb, M);
            tmem_ld_wait(P, M);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float pv = __uint_as_float(P[i]), mv = __uint_as_float(M[i]);
                J[i] = HC == 0 ? fmaf(c.kq, mv, pv) : fmaf(c.kq, pv, c.km * mv);
            }
            if (mol) {
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 x = *reinterpret_cast<const float4 *>(c.xs + kb + i);
                    const float4 y = *reinterpret_cast<const float4 *>(c.ys + kb + i);
                    const float4 e = *reinterpret_cast<const float4 *>(xa + gb + i);
                    const float4 z = *reinterpret_cast<const float4 *>(x0 + gb + i);
                    J[i] = fmaf(y.x, fmaf(c.cm, e.x, c.c0 * z.x), x.x * J[i]);
                    J[i + 1] = fmaf(y.y, fmaf(c.cm, e.y, c.c0 * z.y), x.y * J[i + 1]);
                    J[i + 2] = fmaf(y.z, fmaf(c.cm, e.z, c.c0 * z.z), x.z * J[i + 2]);
                    J[i + 3] = fmaf(y.w, fmaf(c.cm, e.w, c.c0 * z.w), x.w * J[i + 3]);
                }
            }
        }
        // the group's values first, then its stores off one base address: a
        // store still reading its registers would hold up the next level's step
        float *dst = (w == OR_SPILL ? c.Js : c.F) + (size_t)kb * LDC;
        int last = c.st ? nv : -1;                         // levels kb .. kb + last are stored
        if (w == OR_SPILL) {
            last = c.ok ? nv : -1;
#pragma unroll
            for (int i = 0; i < 16; ++i) J[i] *= ssg;
        } else if (uni && kb > 0 && nv > 15) {
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int i = H == 0 ? 15 - r : r;
                const float j = J[i];
                if (ADJ) {
                    const float nu = fmaf(T0, I, j);
                    J[i] = fmaf(A0, nu, B0 * I);
                    I = nu;
                    mi = fmaxf(mi, fabsf(j));
                    tot[RMW ? i : 0] = fmaf(c.w, j, tot[RMW ? i : 0]);
                    mt = fmaxf(mt, fabsf(tot[RMW ? i : 0]));
                    continue;
                }
                I = fmaf(T0, I, fmaf(A0, j, B0 * Jp));
                Jp = j;
                mi = fmaxf(mi, fabsf(I));
                J[i] = I;
                if (RMW) tot[RMW ? i : 0] += I;
            }
        } else if (ADJ) {
            // ends of the column, or weights by layer: the step from the level
            // before uses the layer between, the level's own source the layer after
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int i = H == 0 ? 15 - r : r, k = kb + i;
                const int lp = HC == 0 ? k - 1 : k, la = HC == 0 ? k : k - 1;
                const bool in = i <= nv, hp = lp >= 0 && lp < nt, ha = la >= 0 && la < nt;
                float T = T0, A = A0, Bw = B0;
                if (!uni && in) {
                    if (hp) { T = __ldg(c.wT + lp * c.NR); Bw = __ldg(c.wB + lp * c.NR); }
                    if (ha) A = __ldg(c.wA + la * c.NR);
                }
                if (!ha) A = 0.f;
                // the downward radiance of the top is fixed at zero
                float j = in && !(HC == 1 && k == 0) ? J[i] : 0.f;
                if (HC == 1 && i == nv) j += Jp;
                const float nu = fmaf(T, I, j);
                J[i] = fmaf(A, nu, Bw * I);
                I = in ? nu : I;
                mi = fmaxf(mi, fabsf(j));
                tot[RMW ? i : 0] = fmaf(c.w, j, tot[RMW ? i : 0]);
                mt = fmaxf(mt, fabsf(tot[RMW ? i : 0]));
            }
        } else {
            // the column's ends (its first level holds the start value, levels
            // past the last one do not step), or weights by layer (k of level k
            // upward, k - 1 downward): only the levels lo .. hi of the group step
            const int lo = H == 1 && kb == 0 ? 1 : 0, hi = H == 0 ? nv - 1 : nv;
            const int e0 = (H == 0 ? kb : kb - 1) * c.NR;
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int i = H == 0 ? 15 - r : r;
                const bool step = i >= lo && i <= hi;
                float T = T0, A = A0, Bw = B0;
                if (!uni && step) {
                    const int e = e0 + i * c.NR;
                    T = __ldg(c.wT + e); A = c.sg * __ldg(c.wA + e); Bw = c.sg * __ldg(c.wB + e);
                }
                const float j = J[i], In = fmaf(T, I, fmaf(A, j, Bw * Jp));
                I = step ? In : I;
                Jp = j;
                mi = fmaxf(mi, fabsf(I));
                J[i] = I;
                if (RMW) tot[RMW ? i : 0] += I;
            }
        }
        if (last >= 15) {
#pragma unroll
            for (int i = 0; i < 16; ++i) dst[i * LDC] = J[i];
        } else {
#pragma unroll
            for (int i = 0; i < 15; ++i)
                if (i <= last) dst[i * LDC] = J[i];
        }
        if (RMW && w != OR_SPILL) {
            float *p = c.Tot + (size_t)kb * LDC;
            const int lt = (ADJ ? c.st : c.ok) ? nv : -1;
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i <= lt) p[i * LDC] = tot[RMW ? i : 0];
        }
    }
    v.I = I; v.Jp = Jp; v.mi = mi; v.mt = mt;
}

// Order 1 of a row: what its source, surface seed and outside source are made of.
struct Prim {
    float fa, fm;                     // aerosol and molecular factors of the direct-beam source
    double fA, fM, sb;                // and of the beam a flat surface reflects, 0.5 exp(-2 tau / mu0)
    float tdn, rs, ex;                // seed factors (rough surface), bottom source
    const float *ea;                  // attenuation of the surface's light per level, or null
    const float *lv;                  // level fractions and direct beam
    const double *hh;                 // level optical depths
    double mu0;
    bool flat, jd;                    // reflected beam; skylight source in J
};

// Order 1: direct beam (rt_primary_source.c:17-198), its reflection by a flat
// surface, the water column's skylight source, then the recurrence, and on top
// of the upward radiance the seeds of the direct beam off a rough surface
// (rt_surface_boundary.c:430-493) and of an outside bottom source (495-527).
// Tile by tile in the order of the recurrence, the level constants staged in
// shared memory (pc, 6 OR_TS floats of this direction; pe, the attenuations of
// the upward one, NR per level), eight levels at a time.  Like or_tile_run one short code
// for both directions and every case: a level that does not step (the column's
// first, those past its end) has the weights of a step that changes nothing.
template <int LDC, int MODE>
__device__ __forceinline__ float or_first(const Scan &c, const Prim &p, int h, int T, float *pc, float *pe, int tid,
                                          int g)
{
    const int nt = c.nt, K = nt + 1, dk = h == 0 ? -1 : 1;
    float *plc = pc, *plx = pc + OR_TS, *ply = pc + 2 * OR_TS;
    double *pbm = reinterpret_cast<double *>(pc + 4 * OR_TS);
    const float T0 = c.T, A0 = c.sg * c.Ca, B0 = c.sg * c.Cb;      // the source carries its own sign here
    float I = 0.f, Jp = 0.f;
#pragma unroll 1
    for (int q = 0; q < T; ++q) {
        const int k0 = (h == 0 ? T - 1 - q : q) * OR_TS, n = min(OR_TS, K - k0);
        or_bar(2 + h, 128);
        if (tid < n) {
            const float *l = p.lv + 3 * (k0 + tid);
            plx[tid] = l[0]; ply[tid] = l[1]; plc[tid] = l[2];
            if (p.flat) pbm[tid] = p.sb * exp(p.hh[k0 + tid] / p.mu0);
        }
        if (p.ea) {
            const float *s = p.ea + (size_t)k0 * c.NR;
#pragma unroll 8
            for (int x = tid; x < n * c.NR; x += 128) pe[x] = __ldg(s + x);
        }
        or_bar(2 + h, 128);
        if (!c.ok) continue;
#pragma unroll 1
        for (int x0 = 0; x0 < n;) {
            int plain = c.uni && !p.jd && !p.flat, lit = p.ea != nullptr;
            asm volatile("" : "+r"(plain), "+r"(lit));
            const int i0 = h == 0 ? n - 1 - x0 : x0, kb = k0 + i0;
            float *dst = c.F + (size_t)kb * LDC;
            if (plain && x0 + 8 <= n && q + x0 > 0) {
                // eight levels of a uniform column that all step
                float v[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) v[r] = lit ? pe[(i0 + dk * r) * c.NR + g] : 0.f;
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const int i = i0 + dk * r;
                    const float j = prim_source(plc[i], plx[i], ply[i], p.fa, p.fm);
                    I = prim_step(T0, I, A0, j, B0, Jp);
                    Jp = j;
                    v[r] = I + __fmul_rn(__fmul_rn(p.tdn, v[r]), p.rs) + __fmul_rn(p.ex, v[r]);
                }
                if (c.st) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) dst[dk * r * LDC] = v[r];
                }
                if (MODE == OR_TOT) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) c.Tot[(size_t)(kb + dk * r) * LDC] = v[r];
                }
                x0 += 8;
                continue;
            }
            // up to four levels of any column; the column's first level holds the
            // start value, and a step past the end changes nothing
            const int cnt = min(4, n - x0), w0 = (h == 0 ? kb : kb - 1) * c.NR;
            const bool first = q + x0 == 0;
            float J[4], wT[4], wA[4], wB[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const bool step = r < cnt && !(first && r == 0);
                J[r] = p.jd && r < cnt ? c.Js[(size_t)(kb + dk * r) * LDC] : 0.f;
                wT[r] = step ? T0 : 1.f; wA[r] = step ? A0 : 0.f; wB[r] = step ? B0 : 0.f;
                if (!c.uni && step) {
                    const int w = w0 + dk * r * c.NR;
                    wT[r] = __ldg(c.wT + w); wA[r] = __ldg(c.wA + w); wB[r] = __ldg(c.wB + w);
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (r < cnt) {
                    const int i = i0 + dk * r;
                    float j = __fadd_rn(prim_source(plc[i], plx[i], ply[i], p.fa, p.fm), J[r]);
                    if (p.flat && !(first && r == 0))
                        j += (float)(pbm[i] * ((double)plx[i] * p.fA + (double)ply[i] * p.fM));
                    I = prim_step(wT[r], I, wA[r], j, wB[r], Jp);
                    Jp = j;
                    const float e = lit ? pe[i * c.NR + g] : 0.f;
                    const float f = I + __fmul_rn(__fmul_rn(p.tdn, e), p.rs) + __fmul_rn(p.ex, e);
                    if (c.st) dst[dk * r * LDC] = f;
                    if (MODE == OR_TOT) c.Tot[(size_t)(kb + dk * r) * LDC] = f;
                }
            }
            x0 += cnt;
        }
    }
    return I;
}

// The adjoint's first scan: source factors, output weight (and over the
// quadrature weight) of the thread's column, transport of the inserted view.
struct AdjIn { float fa, fm, e, eb; const float *phi; };

template <int LDC>
__device__ __forceinline__ Col or_adj_first(const Scan &c, const AdjIn &a, int h, float bc)
{
    const int nt = c.nt, K = nt + 1, dk = h == 0 ? 1 : -1;
    Col v{0.f, bc, 0.f, 0.f};
    if (!c.ok) return v;
#pragma unroll 1
    for (int x0 = 0; x0 < K; x0 += 4) {
        const int kb = h == 0 ? x0 : nt - x0, cnt = min(4, K - x0);
        float wT[4], wA[4], wB[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int k = kb + dk * r, lp = h == 0 ? k - 1 : k, la = h == 0 ? k : k - 1;
            const bool hp = r < cnt && lp >= 0 && lp < nt, ha = r < cnt && la >= 0 && la < nt;
            wT[r] = c.T; wB[r] = c.Cb; wA[r] = ha ? c.Ca : 0.f;
            if (!c.uni && hp) { wT[r] = __ldg(c.wT + lp * c.NR); wB[r] = __ldg(c.wB + lp * c.NR); }
            if (!c.uni && ha) wA[r] = __ldg(c.wA + la * c.NR);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (r < cnt) {
                const int k = kb + dk * r;
                float j = prim_source(a.phi[k], c.xs[k], c.ys[k], a.fa, a.fm);
                if (h == 0) { if (k == 0) j += a.eb; }
                else { if (k == nt) j += bc; if (k == 0) j = 0.f; }
                const float nu = fmaf(wT[r], v.I, j), f = fmaf(wA[r], nu, wB[r] * v.I), t = c.w * j;
                v.I = nu;
                v.mi = fmaxf(v.mi, fabsf(j));
                v.mt = fmaxf(v.mt, fabsf(t));
                if (c.st) {
                    c.F[(size_t)k * LDC] = f;
                    c.Tot[(size_t)k * LDC] = t;
                } else {
                    c.Tot[(size_t)k * LDC] = k == 0 ? a.e : 0.f;       // the view's column
                }
            }
        }
    }
    return v;
}

struct Bars { uint64_t *bfull, *bempty, *tfull, *tempty, *order, *op, *fin; volatile int *abort; };

__device__ __noinline__ void or_wait_slow(uint64_t *bar, uint32_t parity, volatile int *abort)
{
    if (*abort) return;
    if (!mbar_wait(bar, parity)) *abort = 1;
}
__device__ __forceinline__ void or_wait(const Bars &b, uint64_t *bar, uint32_t parity)
{
    if (!mbar_try_wait(bar, parity)) or_wait_slow(bar, parity, b.abort);
}

// One order of the scan warps of direction H: every tile in arrival order.
// SRC: the source only, every tile to J.  U: arrivals before this order.  xi:
// this direction's functional buffers.
template <int H, int MODE, int LDC>
__device__ __forceinline__ Col or_order(const Scan &c, Col v, const Bars &b, uint32_t tmem, int T, int K, uint32_t U,
                                        float *xi, int f0, int row, int lane, int quad, bool par_odd, bool rowB)
{
    constexpr bool SRC = MODE == OR_SRC;
    int next = H == 0 ? T - 1 : 0, held = -1, a = 0;
    uint32_t held_slot = 0, nx = 0;                       // nx: functional buffers written
    const int dir = H == 0 ? -1 : 1;
    const bool fq = f0 < quad * 32 + 32 && f0 + 3 > quad * 32;            // quadrant holds functional rows
    const bool rows = quad * 32 < 3 * c.NR;               // quadrant holds output rows
    const float *xa = xi, *x0 = xi;
#pragma unroll 1
    for (;;) {
        int t, what = OR_SCAN;
        uint32_t slot = 0;
        if (held >= 0 && held == next) {
            t = held; slot = held_slot; held = -1;
        } else if (a < T) {
            t = or_tile(a, T);
            slot = (U + a) & 1;
            or_wait(b, &b.tfull[slot], ((U + a) >> 1) & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            __syncwarp();
            ++a;
            if (SRC || t != next) {
                if (!SRC && a > T - 2) { held = t; held_slot = slot; continue; }
                what = OR_SPILL;
            }
        } else if (!SRC && next >= 0 && next < T) {
            t = next;
            what = OR_FROM_J;
        } else {
            break;
        }
        const int k0 = t * OR_TS, n = min(OR_TS, K - k0);
        const uint32_t tb = tmem + slot * 256 + ((uint32_t)(quad * 32) << 16);
        if (c.mol && what != OR_FROM_J) {
            // the tile's molecular functionals, to every warp of this direction
            float *x = xi + (nx & 1) * 3 * OR_TS;
            ++nx;
            if (fq) {
                const int f = row - f0;
#pragma unroll 1
                for (int g = 0; g < (n + 7) >> 3; ++g) {
                    uint32_t z[8], o[8];
                    tmem_ld8_async(tb + (par_odd ? 128 : 0) + 8 * g, z);
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[i] = 0;
                    tmem_ld_wait(z, o);
                    if (f >= 0 && f < 3) {
                        uint4 *d = reinterpret_cast<uint4 *>(x + f * OR_TS + 8 * g);
                        d[0] = make_uint4(z[0], z[1], z[2], z[3]);
                        d[1] = make_uint4(z[4], z[5], z[6], z[7]);
                    }
                }
            }
            or_bar(2 + H, 128);
            xa = x + (rowB ? OR_TS : 0);
            x0 = x + 2 * OR_TS;
        }
        if (rows) or_tile_run<H, LDC, MODE>(c, v, what, tb, k0, n, SRC ? c.sg : 1.f, xa, x0);
        if (what != OR_FROM_J) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&b.tempty[slot]);
        }
        if (what != OR_SPILL) next += dir;
    }
    return v;
}

} // namespace

// SRC = false: every order of every task.  SRC = true: the
// source of the field at hand into J, once per task (the water column's
// skylight, k_dtop_field).
template <int MODE, int LDC>
__device__ __forceinline__ void orders_body(const BatchBufs &B, const WaveBufs &W, const Geom &G, int t0, int nw, int Kmax,
                                            const unsigned char *popt, const float *molc, int *counter, int ncot)
{
    constexpr bool SRC = MODE == OR_SRC, ADJ = MODE == OR_ADJ;
    // the declared alignment keeps the pointers below known as shared memory
    extern __shared__ __align__(1024) unsigned char or_smem[];
    unsigned char *base = or_smem;
    // pitch of the surface rows, round32(3 NR), which the row stride determines
    constexpr int RP = LDC == 224 ? 128 : LDC >= 160 ? 96 : LDC >= 96 ? 64 : 32;
    const int N = G.N, NR = G.NR, Rw = par_rows(G), kp = (Kmax + OR_GRP + 3) & ~3;
    const uint32_t a_tile = (uint32_t)Rw * 128u;
    unsigned char *sA = base, *sB = base + 9 * a_tile;
    float *xs = (float *)(sB + 2 * OR_BSTAGE), *ys = xs + kp;
    float *xi = ys + kp;                                  // [2 directions][2 buffers][3][OR_TS]
    float *fb = xi + 2 * 2 * 3 * OR_TS;                   // [128] surface-side radiance per row (x quadrature weight)
    float *bcx = fb + 128;                                // [2 orders][128] boundary values per row
    float2 *red = (float2 *)(bcx + 256);              // [2 orders][8 warps]
    Bars b;
    b.bfull = (uint64_t *)(red + 16);
    b.bempty = b.bfull + 2; b.tfull = b.bfull + 4; b.tempty = b.bfull + 6;
    b.order = b.bfull + 8; b.op = b.bfull + 9; b.fin = b.bfull + 10;
    uint32_t *tslot = (uint32_t *)(b.bfull + 11);
    b.abort = (volatile int *)(tslot + 1);
    volatile int *cmd = (volatile int *)(tslot + 2);      // [2]: 2 task + new, or -1
    volatile int *cur_s = (volatile int *)(tslot + 4);
    volatile int *nop_s = (volatile int *)(tslot + 5);    // operator copies issued
    volatile int *quit = (volatile int *)(tslot + 6);     // [2 orders]: the abort flag as the scan warps act on it
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // incoming component of the x-th stage of a tile
    auto comp = [&](int x) -> int { return G.direct ? x : 2 - x; };

    if (warp == 15) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&b.bfull[i], OR_TS / 16);
            mbar_init(&b.bempty[i], 1);
            mbar_init(&b.tfull[i], 1);
            mbar_init(&b.tempty[i], 8);
        }
        mbar_init(b.order, 1);
        mbar_init(b.op, 1);
        mbar_init(b.fin, 1);
        *b.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;

    if (warp < 8) {
        // ================= scan warps =================
        // walk direction (0: from the bottom up) and hemisphere of the columns
        const int hw = warp >> 2, h = ADJ ? 1 - hw : hw, quad = warp & 3, row = quad * 32 + lane;
        int s = 0, g = NR;
        if (row < 3 * N) { s = row / N; g = row - s * N; }
        else if (row < 3 * NR) { g = N + (row - 3 * N) / 3; s = (row - 3 * N) % 3; }
        const int c = g < NR ? col_of(G, s, h, g) : 0;
        const int f0 = 3 * NR;
        uint32_t U = 0;
        int step = 0, nxt = 0, nop = 0, ph = 0;           // commands posted; scans made
        if (tid == 0) nxt = atomicAdd(counter, 1);
        for (;;) {
            if (tid == 0) *cur_s = nxt < nw && !*b.abort ? nxt : -1;
            or_bar(1, 256);
            const int item = *cur_s, tl = ADJ ? item / ncot : item;
            if (item < 0) {
                if (tid == 0) {
                    cmd[step & 1] = -1;
                    mbar_arrive(b.order);
                    // an operator copy in flight lands before the CTA leaves
                    if (nop && !mbar_wait(b.op, (nop - 1) & 1)) *b.abort = 1;
                }
                break;
            }
            const TaskDev &tk = B.tasks[t0 + tl];
            const PixDev &d = B.px[tk.pix];
            const int nt = d.nt, K = nt + 1, T = (K + OR_TS - 1) / OR_TS;
            const bool water = d.medium == 1, mol = tk.m <= 2, more = SRC || ADJ || d.max_orders > 1;
            if (tid == 0) {
                nxt = atomicAdd(counter, 1);
                if (more) {
                    // the task's operator, behind order 1; its shared memory is
                    // free, every product of the task before has been consumed
                    mbar_expect_tx(b.op, 9 * a_tile);
                    bulk_g2s(sA, popt + (size_t)tl * par_bytes(G), 9 * a_tile, b.op);
                    *nop_s = ++nop;
                }
            }
            const float *lv = B.lvf + 3 * d.lev_off;
            for (int k = tid; (mol || ADJ) && k < K + OR_GRP; k += 256) {
                xs[k] = k < K ? lv[3 * k] : 0.f;
                ys[k] = k < K ? lv[3 * k + 1] : 0.f;
            }
            Scan sc;
            sc.ok = g < d.n_ring;
            sc.st = row < 3 * N;
            sc.uni = !d.gas && !d.has_dtau;
            sc.mol = mol;
            sc.sg = h == 1 && s == 2 ? -1.f : 1.f;
            sc.kq = G.direct ? 0.f : 1.f;
            sc.km = G.direct ? 1.f : -1.f;
            sc.xs = xs; sc.ys = ys; sc.nt = nt; sc.NR = NR;
            const size_t off = ADJ ? (size_t)tk.fld_off * ncot + (size_t)(item - tl * ncot) * K * LDC : (size_t)tk.fld_off;
            sc.F = W.F + off + c;
            sc.Js = W.J + off + c;
            sc.Tot = W.Tot + off + c;
            sc.w = ADJ && sc.st ? (float)B.gw[g] : 1.f;
            const int gc = sc.ok ? g : 0;
            sc.wT = B.Tc + d.coef_off + gc; sc.wA = B.Ca + d.coef_off + gc; sc.wB = B.Cb + d.coef_off + gc;
            // equal optical depths (no gas, no layer overrides): every layer has the weights of the first
            sc.T = sc.wT[0]; sc.Ca = (ADJ ? 1.f : sc.sg) * sc.wA[0]; sc.Cb = (ADJ ? 1.f : sc.sg) * sc.wB[0];
            if (ADJ && h == 1) { sc.kq *= sc.sg; sc.km *= sc.sg; }      // here it is the source that is added
            sc.cm = sc.c0 = 0.f;
            if (mol && sc.ok) {
                const float par = (tk.m & 1) ? -1.f : 1.f;
                const float v = molc[(size_t)tl * OR_MOLC + row];
                // downward: par, and sigma; the latter is in the weights
                sc.cm = h == 0 ? v : (ADJ ? sc.sg : 1.f) * par * v;
                sc.c0 = s == 0 && tk.m == 0 ? 1.f : 0.f;
            }
            // totals at the output levels (double-float) and, where all are
            // kept, at level 1
            float *Tot = sc.Tot;
            float2 t_top = make_float2(0.f, 0.f), t_bot = t_top;
            float t_one = 0.f;
            // the boundary is fed by the radiance going down at the bottom
            // (atmosphere) or going up at the top (under the water surface)
            const bool src = hw == (water ? 0 : 1), dst = !src && (water || d.surf_on);
            const float pw = row < 3 * N ? B.pw[(tk.m == 0 ? 0 : N) + g] : 0.f;
            const float *Rm = (water || d.rough) ? W.srf + tk.srf_off + row : nullptr;
            const float *MF = B.frs + ((size_t)tk.pix * NR + gc) * 9 + s * 3;
            const bool surf = !SRC && (water || d.surf_on);
            // The boundary values of the next order, by the threads of the source
            // direction (they finish first: the other one starts from the boundary
            // and ends away from it): radiance of this thread's row in, boundary
            // value of the same row number of the other direction out.
            auto boundary = [&](int at, float w) {
                fb[row] = Rm && !ADJ ? pw * w : w;
                or_bar(2 + hw, 128);
                float a = 0.f;
                if (ADJ) {
                    // transposed: what the surface's row sends back to its incoming column
                    if (Rm && row < 3 * N) {
                        const float *R = W.srf + tk.srf_off + (size_t)row * RP;
                        const int nr = 3 * d.n_ring;
                        float a0 = 0.f, a1 = 0.f;
                        int j = 0;
#pragma unroll 4
                        for (; j + 4 <= nr; j += 4) {
                            const float4 q = __ldg(reinterpret_cast<const float4 *>(R + j));
                            const float4 f = *reinterpret_cast<const float4 *>(fb + j);
                            a0 = fmaf(q.x, f.x, a0); a1 = fmaf(q.y, f.y, a1);
                            a0 = fmaf(q.z, f.z, a0); a1 = fmaf(q.w, f.w, a1);
                        }
                        for (; j < nr; ++j) a0 = fmaf(__ldg(R + j), fb[j], a0);
                        a = (a0 + a1) * (pw / sc.w);
                    }
                } else if (Rm) {
                    // 24 rows in flight (12: 7.1 ms where this takes 6.9; 48: no better)
                    float a0 = 0.f, a1 = 0.f;
                    if (row < 3 * NR) {
                        int j = 0;
#pragma unroll 1
                        for (; j + 24 <= 3 * N; j += 24) {
                            float r[24];
#pragma unroll
                            for (int q = 0; q < 24; ++q) r[q] = __ldg(Rm + j * RP + q * RP);
#pragma unroll
                            for (int q = 0; q < 24; q += 2) {
                                a0 = fmaf(r[q], fb[j + q], a0);
                                a1 = fmaf(r[q + 1], fb[j + q + 1], a1);
                            }
                        }
#pragma unroll 4
                        for (; j < 3 * N; j += 2) {
                            a0 = fmaf(__ldg(Rm + j * RP), fb[j], a0);
                            a1 = fmaf(__ldg(Rm + j * RP + RP), fb[j + 1], a1);
                        }
                    }
                    a = a0 + a1;
                } else if (sc.ok) {
                    a = MF[0] * fb[srf_row(G, g, 0)] + MF[1] * fb[srf_row(G, g, 1)] + MF[2] * fb[srf_row(G, g, 2)];
                }
                bcx[at * 128 + row] = a;
            };
            int it = 2;
            if (MODE == OR_FWD || MODE == OR_TOT) {
                Prim p;
                const float *pv = W.pvec + (size_t)tl * 2 * LDC + c;
                // an atmosphere driven only by a bottom source has no solar primary and no
                // surface seeds (rt_solver.c:949-954, rt_surface_boundary.c:553-569)
                const bool sun = sc.ok && !d.bottom_only, ext = d.ext_off >= 0 && tk.m <= d.ext_mmax;
                p.fa = sun ? pv[0] : 0.f;
                p.fm = sun ? pv[LDC] : 0.f;
                p.flat = d.flat && !d.bottom_only;
                p.fA = p.fM = 0.0;
                if (p.flat && sc.ok) {
                    // Stokes s of the reflected beam uses kernel components (s, s + 3)
                    const float *fa = W.fvec + ((size_t)tl * 4 + 2 * h) * 6 * NR, *fm = fa + 6 * NR;
                    p.fA = d.beam_RI * fa[s * NR + g] + d.beam_RQ * fa[(s + 3) * NR + g];
                    p.fM = d.beam_RI * fm[s * NR + g] + d.beam_RQ * fm[(s + 3) * NR + g];
                }
                p.sb = d.beam_sb;
                const bool seed = d.rough && h == 0 && sun, extb = d.medium == 0 && ext && h == 0 && sc.ok;
                p.tdn = p.rs = p.ex = 0.f;
                if (seed) {
                    p.tdn = (tk.m == 0 ? 1.f : 0.5f) * d.seed0;
                    p.rs = W.srf[tk.srf_off + G.srf_sun + g * 9 + s * 3];
                }
                if (extb) p.ex = (float)B.ext[d.ext_off + ((size_t)tk.m * NR + g) * 3 + s];
                p.ea = (d.rough && !d.bottom_only || d.medium == 0 && ext) && h == 0 ? B.Eatt + d.lev_off * NR : nullptr;
                p.lv = lv; p.hh = B.h + d.lev_off; p.mu0 = d.mu0;
                p.jd = water && ext;
                const float I1 = or_first<LDC, MODE>(sc, p, h, T, xi + h * 2 * 3 * OR_TS, reinterpret_cast<float *>(sB), tid & 127, gc);
                if (!isfinite(I1)) atomicExch(B.err, OCRT_ERR_NONFINITE);
                // totals at the two ends: the column's start value 0 and its end value, and the seeds
                auto lit = [&](float I, int k) {
                    const float e = p.ea ? __ldg(p.ea + (size_t)k * NR + gc) : 0.f;
                    return df_add(df_add(make_float2(I, 0.f), __fmul_rn(__fmul_rn(p.tdn, e), p.rs)), __fmul_rn(p.ex, e));
                };
                t_top = lit(h == 0 ? I1 : 0.f, 0);
                t_bot = lit(h == 0 ? 0.f : I1, nt);
                if (MODE == OR_FWD && G.tot_all && sc.ok && sc.st) t_one = sc.F[LDC];
                if (src && surf && more) boundary(ph & 1, sc.ok ? I1 : 0.f);
            }
            float resid = 0.f;
            int conv = 0;
            const int max_it = d.max_orders;
            const float tolf = __double2float_ru(d.tol);   // resid < tol as floats
            AdjIn ai{0.f, 0.f, 0.f, 0.f, nullptr};
            float mview = 0.f;                             // the view's own part of the adjoint total
            bool begin = ADJ, only = false;                // scan without a product; nothing but order 1
            if (ADJ) {
                // Order 1 is the output weights e at the top (k_adj_init wrote
                // them there).  Of an inserted view they lie on a column that no
                // product reads: its transposed transport phi is the same for the
                // three Stokes components but for e, and makes the source of order
                // 2; Gauss columns start with e itself.
                const bool ins = d.n_ring > N;
                float *phi = reinterpret_cast<float *>(sB), *vT = phi + kp, *vA = vT + kp, *vB = vA + kp;
                for (int k = tid; k < kp; k += 256) {
                    const int l = (sc.uni ? 0 : min(k, nt - 1)) * NR + N;
                    phi[k] = 0.f;
                    vT[k] = __ldg(B.Tc + d.coef_off + l); vA[k] = __ldg(B.Ca + d.coef_off + l);
                    vB[k] = __ldg(B.Cb + d.coef_off + l);
                }
                or_bar(1, 256);
                if (tid == 0 && ins) {
                    float nu = 1.f, up = 0.f;
                    for (int k = 0; k <= nt; ++k) {
                        if (k > 0) nu = vT[k - 1] * up;
                        phi[k] = (k < nt ? vA[k] * nu : 0.f) + (k > 0 ? vB[k - 1] * up : 0.f);
                        up = nu;
                    }
                    vT[kp - 1] = nu;                       // at the surface
                }
                or_bar(1, 256);
                ai.phi = phi;
                float ev[3] = {0.f, 0.f, 0.f};
                if (ins) {
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        ev[q] = W.F[off + col_of(G, q, 0, N)];
                        mview = fmaxf(mview, fabsf(ev[q]));
                    }
                    only = (mview > 0.f ? 1.0 : 0.0) < d.tol || d.max_orders <= 1;
                    resid = mview > 0.f ? 1.f : 0.f;
                    conv = (double)resid < d.tol;
                }
                ai.e = sc.ok ? sc.F[0] : 0.f;
                if (ins && !only && sc.st) {
                    // row "view" of the operator, transposed: its entries hold the
                    // weight of this thread's node
                    const unsigned char *Pt = popt + (size_t)tl * par_bytes(G) + (size_t)s * 3 * a_tile;
                    float qa = 0.f;
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        float m[2] = {0.f, 0.f};
#pragma unroll
                        for (int pr = 0; pr < 2; ++pr)
#pragma unroll
                            for (int pc = 0; pc < 3; ++pc) {
                                const int col = 32 * pr + g;
                                const uint32_t o = pc * a_tile + par_swz(srf_row(G, N, q), col & ~1) + 2 * (col & 1);
                                m[pr] += __uint_as_float((uint32_t)*reinterpret_cast<const uint16_t *>(Pt + o) << 16);
                            }
                        qa = fmaf(ev[q], h == 0 ? m[0] + m[1] : sc.sg * (m[0] - m[1]), qa);
                    }
                    ai.fa = qa / sc.w;
                    if (mol) {
                        const float *mv = molc + (size_t)tl * OR_MOLC;
                        const float P = mv[srf_row(G, N, 0)], R = mv[srf_row(G, N, 1)], Tt = -mv[srf_row(G, N, 2)];
                        float c3[3], c0[3];
                        par_functional(s == 0 ? 0 : 1, tk.m, d.depol, P, R, Tt, c3);
                        par_functional(2, tk.m, d.depol, P, R, Tt, c0);
                        ai.fm = sc.cm * (c3[0] * ev[0] + c3[1] * ev[1] + c3[2] * ev[2]) + sc.c0 * c0[0] * ev[0];
                    }
                }
                ai.eb = sc.st ? ai.e / sc.w : 0.f;
                if (src && surf) boundary(ph & 1, ins && !only && !sc.st && sc.ok && h == 0 ? ai.e * vT[kp - 1] : 0.f);
                it = ins && !only ? 2 : 1;
            }
            if (!more) { it = 1; conv = 1; }
            or_bar(1, 256);
            if (more && !ADJ && tid == 0) {
                cmd[step & 1] = 2 * item + 1;
                mbar_arrive(b.order);
            }
            for (; more; ++it) {
                const float bc = !SRC && dst && sc.ok ? bcx[(ph & 1) * 128 + row] : 0.f;
                Col v{ADJ ? 0.f : bc, ADJ ? bc : 0.f, 0.f, 0.f};
                if (ADJ && begin) {
                    v = or_adj_first<LDC>(sc, ai, h, bc);
                } else {
                    float *xh = xi + hw * 2 * 3 * OR_TS;
                    const bool odd = (tk.m & 1) && !G.direct, rb = s != 0;
                    if (hw == 0) v = or_order<0, MODE, LDC>(sc, v, b, tmem, T, K, U, xh, f0, row, lane, quad, odd, rb);
                    else v = or_order<1, MODE, LDC>(sc, v, b, tmem, T, K, U, xh, f0, row, lane, quad, odd, rb);
                    U += T;
                }
                if (SRC) { ++step; break; }
                // ---- end of the order: totals, surface-side radiance, residual ----
                float mi = 0.f, mt = 0.f;
                if (sc.ok) {
                    if (ADJ) {
                        mi = sc.st ? sc.w * v.mi : 0.f;
                        mt = sc.st ? v.mt : 0.f;
                    } else {
                        t_top = df_add(t_top, h == 0 ? v.I : bc);
                        t_bot = df_add(t_bot, h == 0 ? bc : v.I);
                        if (MODE == OR_FWD && G.tot_all && sc.st) t_one += sc.F[LDC];
                        mi = v.mi;
                        mt = fmaxf(fabsf(t_top.x), fabsf(t_bot.x));
                    }
                    if (!isfinite(v.I)) atomicExch(B.err, OCRT_ERR_NONFINITE);
                }
                if (src && surf) boundary((ph + 1) & 1, ADJ ? (sc.st ? sc.w * v.I : 0.f) : sc.ok ? v.I : 0.f);
                // non-negative floats order like their bits
                mi = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(mi, 0.f))));
                mt = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(mt, 0.f))));
                if (lane == 0) red[(ph & 1) * 8 + warp] = make_float2(mi, mt);
                if (tid == 0) quit[ph & 1] = *b.abort;
                or_bar(1, 256);
#pragma unroll
                for (int w = 0; w < 8; ++w) {
                    const float2 v = red[(ph & 1) * 8 + w];
                    mi = fmaxf(mi, v.x);
                    mt = fmaxf(mt, v.y);
                }
                ++ph;
                if (!(ADJ && begin)) ++step;
                if (ADJ && only) break;
                mt = fmaxf(mt, mview);
                resid = mt > 0.f ? mi / mt : 0.f;
                conv = resid < tolf;
                // read here, behind the other conditions: from right behind the barrier it
                // cost 4% (500 pixels at 24 streams 5.87 ms, 5.64 so)
                if (conv || it >= max_it || quit[(ph & 1) ^ 1]) break;
                if (tid == 0) {
                    cmd[step & 1] = 2 * item + (ADJ && begin ? 1 : 0);
                    mbar_arrive(b.order);
                }
                begin = false;
            }
            if (SRC) continue;
            if (!ADJ && sc.ok) {
                Tot[0] = t_top.x;
                Tot[(size_t)nt * LDC] = t_bot.x;
                W.Ttl[tot_tail_off(tk, G, 0, c)] = t_top.y;
                W.Ttl[tot_tail_off(tk, G, nt, c)] = t_bot.y;
                if (MODE == OR_FWD && G.tot_all && sc.st && nt > 1) Tot[LDC] = t_one;
            }
            if (tid == 0) {
                // no product waited for the operator: the next copy goes to the same place
                if (ADJ && begin && !mbar_wait(b.op, (nop - 1) & 1)) *b.abort = 1;
                TaskState st;
                st.active = 0; st.orders = it; st.converged = conv; st.pad_ = 0; st.resid = (double)resid;
                B.state[ADJ ? item : t0 + tl] = st;
            }
        }
    } else if (warp < 8 + OR_TS / 16) {
        // ================= producers =================
        const int pw = warp - 8;                          // 16-level block of the tile
        const int q = lane & 7, l2 = lane >> 3;
        // rows of iteration x: 4 apart within a warp store, so the two halves
        // of the swizzle fall on different banks
        auto r16 = [&](int x) -> int { return 16 * pw + x * 2 + (l2 >> 1) + (l2 & 1) * 4; };
        const bool qin = 4 * q < N;
        uint32_t gi = 0;                                  // stages filled
        int K = 0, T = 0;
        const float *Fb = nullptr, *lv = nullptr;
        // half stage j = 2 (3 a + x) + hh of an order, component si = comp(x): rows of iterations
        // 2 hh, 2 hh + 1 into registers
        struct Rows { float4 u[2], v[2]; float x[2]; };
        auto load = [&](Rows &d, int j) {
            const int e = j >> 1, a = e / 3, si = comp(e - 3 * a);
            const int k0 = or_tile(a, T) * OR_TS, nl = min(OR_TS, K - k0);
            const int rb = r16(0) + 8 * (j & 1);
            const float *src = Fb + (size_t)(k0 + rb) * LDC + 2 * N * si + 4 * q;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const bool in = qin && rb + 2 * x < nl;
                d.x[x] = in && lv ? __ldg(lv + 3 * (k0 + rb + 2 * x)) : 1.f;
                d.u[x] = in ? *reinterpret_cast<const float4 *>(src + 2 * x * LDC) : make_float4(0.f, 0.f, 0.f, 0.f);
                d.v[x] = in ? *reinterpret_cast<const float4 *>(src + 2 * x * LDC + N) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        // F+- of half a stage into its B tile
        auto fill = [&](const Rows &d, int j, uint32_t st) {
            const int si = comp((j >> 1) % 3), rb = r16(0) + 8 * (j & 1);
            // F+ = up + sigma down: for U the sum is F- and the difference F+
            unsigned char *tile = sB + st * OR_BSTAGE;
            const bool sw = si == 2 && !G.direct;
            const int cs = 4 * q + (sw ? 32 : 0), cd = 4 * q + (sw ? 0 : 32);
            // direct form: F_up and sigma F_dn
            const float ka = G.direct ? 0.f : 1.f, kb = G.direct ? (si == 2 ? 1.f : -1.f) : 1.f;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                uint32_t s0[3], s1[3], d0[3], d1[3];
                const float f = d.x[x];
                const float4 u = d.u[x], v = d.v[x];
                split_bf16x3_trunc(f * fmaf(ka, v.x, u.x), f * fmaf(ka, v.y, u.y), s0);
                split_bf16x3_trunc(f * fmaf(ka, v.z, u.z), f * fmaf(ka, v.w, u.w), s1);
                split_bf16x3_trunc(f * fmaf(ka, u.x, -kb * v.x), f * fmaf(ka, u.y, -kb * v.y), d0);
                split_bf16x3_trunc(f * fmaf(ka, u.z, -kb * v.z), f * fmaf(ka, u.w, -kb * v.w), d1);
                unsigned char *ps = tile + par_swz(rb + 2 * x, cs), *pd = tile + par_swz(rb + 2 * x, cd);
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    *reinterpret_cast<uint2 *>(ps + p * OR_BPIECE) = make_uint2(s0[p], s1[p]);
                    *reinterpret_cast<uint2 *>(pd + p * OR_BPIECE) = make_uint2(d0[p], d1[p]);
                }
            }
        };
        for (int step = 0;; ++step) {
            or_wait(b, b.order, step & 1);
            if (__any_sync(0xffffffffu, *b.abort != 0)) break;
            const int cm = cmd[step & 1];
            if (cm < 0) break;
            if (cm & 1) {
                const int item = cm >> 1, tl = ADJ ? item / ncot : item;
                const TaskDev &tk = B.tasks[t0 + tl];
                K = tk.K;
                T = (K + OR_TS - 1) / OR_TS;
                Fb = W.F + (ADJ ? (size_t)tk.fld_off * ncot + (size_t)(item - tl * ncot) * K * LDC : (size_t)tk.fld_off);
                lv = tk.m <= 2 ? nullptr : B.lvf + 3 * B.px[tk.pix].lev_off;
            }
            // the rows of a stage are loaded while the stage before is split
            Rows ra, rb;
            load(ra, 0);
            load(rb, 1);
#pragma unroll 1
            for (int j = 0; j < 6 * T; j += 2, ++gi) {
                const uint32_t st = gi & 1;
                const bool mine = 16 * pw < min(OR_TS, K - or_tile(j / 6, T) * OR_TS);
                if (gi >= 2) or_wait(b, &b.bempty[st], ((gi >> 1) - 1) & 1);
                __syncwarp();
                if (mine) fill(ra, j, st);
                if (j + 2 < 6 * T) load(ra, j + 2);
                if (mine) fill(rb, j + 1, st);
                if (j + 3 < 6 * T) load(rb, j + 3);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&b.bfull[st]);
            }
        }
    } else if (warp == 15) {
        // ================= operator load and MMA issue =================
        // The warp runs converged and one elected lane issues: addresses and
        // descriptors then stay on the uniform datapath (from a divergent
        // single lane an MMA took 119 cycles to issue, twice its run time).
        uint32_t gi = 0, U = 0;
        int K = 0, T = 0;
        const bool two = N > 16;                          // two 16-deep steps per parity
        const uint32_t sa = smem_u32(sA) >> 4, sb = smem_u32(sB) >> 4, at = a_tile >> 4;
        const uint64_t dbase = sdesc_sw128(0);            // layout bits; addresses are below 2^18
        for (int step = 0;; ++step) {
            or_wait(b, b.order, step & 1);
            if (__any_sync(0xffffffffu, *b.abort != 0)) break;
            const int cm = cmd[step & 1];
            if (cm < 0) break;
            if (cm & 1) {
                K = B.tasks[t0 + (ADJ ? (cm >> 1) / ncot : cm >> 1)].K;
                T = (K + OR_TS - 1) / OR_TS;
                or_wait(b, b.op, (*nop_s - 1) & 1);
                if (__any_sync(0xffffffffu, *b.abort != 0)) break;
            }
            bool stop = false;
#pragma unroll 1
            for (int a = 0; a < T && !stop; ++a, ++U) {
                const uint32_t slot = U & 1;
                const int nl = min(OR_TS, K - or_tile(a, T) * OR_TS), n16 = (nl + 15) & ~15;
                if (U >= 2) or_wait(b, &b.tempty[slot], ((U >> 1) - 1) & 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t idesc = idesc_bf16(128, n16), acc = tmem + slot * 256;
#pragma unroll 1
                for (int si = 0; si < 3; ++si, ++gi) {
                    const uint32_t st = gi & 1;
                    or_wait(b, &b.bfull[st], (gi >> 1) & 1);
                    if (__any_sync(0xffffffffu, *b.abort != 0)) { stop = true; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t ta = sa + comp(si) * 3 * at, tb = sb + st * (OR_BSTAGE >> 4);
                    if (elect_one()) {
                        // pieces (operator, field) of the six products, the small ones
                        // first: the accumulator is truncated at each step, so the
                        // fewer steps it takes at full size the better
                        constexpr int pa[6] = {2, 1, 0, 1, 0, 0}, pb[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll 1
                        for (int x = 0; x < (G.direct ? 4 : 2); ++x) {
                            // output half, half of the field, block of the operator
                            const uint32_t o = G.direct ? x >> 1 : x, i = x & 1, ab = G.direct ? o ^ i : o;
                            const uint32_t t = ta + ab * 4, u = tb + i * 4, first = G.direct ? i == 0 : 1;
#pragma unroll
                            for (int e = 0; e < 12; ++e) {
                                const int q = e >> 1, k = e & 1;
                                if (k && !two) continue;
                                umma_bf16(acc + o * 128, dbase | (t + k * 2 + pa[q] * at),
                                          dbase | (u + k * 2 + pb[q] * (OR_BPIECE >> 4)), idesc,
                                          (si > 0 || e > 0 || !first) ? 1u : 0u);
                            }
                        }
                        umma_commit(&b.bempty[st]);
                        if (si == 2) umma_commit(&b.tfull[slot]);
                    }
                    __syncwarp();
                }
            }
            if (stop) break;
        }
        // every MMA completes before the CTA leaves
        if (elect_one()) umma_commit(b.fin);
        __syncwarp();
        if (!mbar_wait(b.fin, 0)) *b.abort = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && *b.abort) atomicExch(B.err, OCRT_ERR_DEVICE);
    if (warp == 15) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// The row stride is a template argument: the scan's stores and the producers'
// loads then take immediate offsets.  Its values for N = 8 .. 32 with one or four
// zero-weight slots.
#define OR_ARGS BatchBufs B, WaveBufs W, Geom G, int t0, int nw, int Kmax, const unsigned char *popt, const float *molc, \
                int *counter, int ncot
template <int LDC>
__global__ void __launch_bounds__(OR_THREADS, 1) k_orders(OR_ARGS)
{
    orders_body<OR_FWD, LDC>(B, W, G, t0, nw, Kmax, popt, molc, counter, ncot);
}
template <int LDC>
__global__ void __launch_bounds__(OR_THREADS, 1) k_orders_source(OR_ARGS)
{
    orders_body<OR_SRC, LDC>(B, W, G, t0, nw, Kmax, popt, molc, counter, ncot);
}
template <int LDC>
__global__ void __launch_bounds__(OR_THREADS, 1) k_orders_total(OR_ARGS)
{
    orders_body<OR_TOT, LDC>(B, W, G, t0, nw, Kmax, popt, molc, counter, ncot);
}
template <int LDC>
__global__ void __launch_bounds__(OR_THREADS, 1) k_orders_adjoint(OR_ARGS)
{
    orders_body<OR_ADJ, LDC>(B, W, G, t0, nw, Kmax, popt, molc, counter, ncot);
}

// Task counters of a wave's launches.
__global__ void k_orders_reset(int *counter)
{
    if (threadIdx.x < 4) counter[threadIdx.x] = 0;
}

namespace {

typedef void (*OrdersFn)(OR_ARGS);
struct OrdersInst { int ldc; OrdersFn fn[4]; };                // by OR_FWD .. OR_ADJ
#define OR_INST(n) {n, {k_orders<n>, k_orders_source<n>, k_orders_total<n>, k_orders_adjoint<n>}}
const OrdersInst g_orders[] = {OR_INST(64), OR_INST(96), OR_INST(128), OR_INST(160), OR_INST(192), OR_INST(224)};

const OrdersInst *orders_inst(int ldc)
{
    for (const OrdersInst &o : g_orders)
        if (o.ldc == ldc) return &o;
    return nullptr;
}

} // namespace

// N a multiple of 4 keeps the producers' rows in whole float4s.  12 and 28 streams take this
// kernel (scene of 500 pixels, 17 modes, up to 150 layers: 4.9 and 8.1 ms against 10.7 and
// 29.6 with the separate passes).  N = 20 does not, though its shape fits and it would gain
// as much (the same scene 14.4 ms with the separate passes, 5.4 here; one pixel 0.70 and
// 0.37): the scan autotuner is reached by default only there and above 32 streams, and
// tests/test_gpu_scan.py pins its choice and record at 20.  3 NR + 3 rows fit one MMA of 128
// (111 at 32 streams with four zero-weight slots); larger N (48 streams) would need a
// second M tile and twice the operator, 480 KB, more than an SM has.
bool orders_supported(const Geom &G, int Kmax, bool adjoint)
{
    const OrdersInst *o = orders_inst(G.LDC);
    return (G.N % 8 == 0 || G.N % 16 == 12) && G.N <= 32 && 3 * G.NR + 3 <= 128 && o && (!adjoint || G.E == 1) &&
           orders_smem_bytes(G, Kmax) <= 227 * 1024;
}

void orders_launch(int kind, int grid, cudaStream_t st, const BatchBufs &B, const WaveBufs &W, const Geom &G, int t0,
                   int nw, int Kmax, const unsigned char *popt, const float *molc, int *counter, int ncot)
{
    orders_inst(G.LDC)->fn[kind]<<<grid, OR_THREADS, orders_smem_bytes(G, Kmax), st>>>(B, W, G, t0, nw, Kmax, popt, molc,
                                                                                      counter + kind, ncot);
}

cudaError_t orders_init()
{
    for (const OrdersInst &o : g_orders)
        for (OrdersFn f : o.fn) {
            const cudaError_t e = cudaFuncSetAttribute((const void *)f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       227 * 1024);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}
