// xstep.cuh -- the fused x pass of a step for power-of-two FP32 lines, in the forms
// of a step with uniform parameters (k_xstep), of the general step (k_xgstep), of a
// packed ensemble's size class (k_xens) and of a Runge-Kutta stage (k_xrk).  One
// translation unit per line length (xstep_32.cu and so on), which compile side by side.
#pragma once
#include "device.cuh"
#include "fftreg.cuh"
#include "fused.cuh"
#include "kparams.h"
#include "launch.h"
#include "terms.cuh"
#include "xreg.cuh"

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

// ------------------------------------------------------------------ fused x pass of a step
// One CTA owns ROWS consecutive rows r = z ny + y (the flattened (z, y) row
// index, r0 .. r0 + ROWS - 1), all three components, and runs on them, in
// shared memory:
//   1. the inverse x transform of the (y,z)-pass output (two rows per
//      complex line, Hermitian completion) -> the dipole field of the rows,
//      written to its slot;
//   2. the fused field terms + LLG update of the rows' sites with that field
//      as the addend -> the new spins (exchange neighbours read from the
//      current spin arrays, which no CTA writes);
//   3. (fwd) the forward x transform of the new spins (two rows per complex
//      line, split) -> the spectrum rows of the next step.
// The spectrum rows a CTA reads in 1 and writes in 3 are its own.  Every
// arithmetic step repeats k_ix_fast, fused_site and k_fx_fast operation for
// operation, so the result is bitwise that of the three separate kernels.
// SZ: the CTA's share.  0: 2048 sites (512-point lines 4096) on 512 threads
// (384 for the shared-memory Stockham lines of 512 points), two CTAs per SM at
// 64 registers, for lattices that fill the chip with such CTAs; 1: 512 sites on
// 256 threads, 2: 128 sites on 128 threads (two rows at least), for smaller
// ones (xs_size): a lattice of 128 x 128 x 4 is 32 CTAs of share 0, and the
// step is one CTA's chain; 3 (TIGHT): lines for 192 lanes on 256 threads, where
// many CTAs share an SM (packed replicas).  Lines are transformed alike at every
// share, so results do not depend on it.
// TIGHT keeps one buffer, exchanged, replaced by the new spins and transformed
// back in place, so that four CTAs fit an SM, and walks the sites alone rather
// than the padded line (open replicas are half padding).  A periodic film has no
// padding and its trip count is then known to the compiler: 256x256x8 takes
// 21.05 us a step in the form of share 0 and 21.9 in this one.
template <int PX, bool TH = false, int SZ = 0>
struct XSCfg {
    static constexpr int NT = SZ == 0 ? (XReg<PX>::OK ? 512 : 384) : (SZ == 2 ? 128 : 256);
    static constexpr int TPL = fr::Tpl<PX>::V;
    static constexpr int SMALL = (SZ == 1 ? 512 : 128) / PX;
    static constexpr int ROWS = SZ == 0 ? 2 * (384 / TPL) / 3 : (SZ == 3 ? 128 / XReg<PX>::T : (SMALL < 2 ? 2 : SMALL));
    static constexpr int L = 3 * ROWS / 2;              // complex lines
    static constexpr int R2 = ROWS / 2;
    static constexpr int KX = PX / 2 + 1;
    static constexpr bool TIGHT = SZ == 3;
    // line stride in shared memory, odd: the same k of consecutive lines
    // falls in different banks
    static constexpr int LS = (TIGHT && XReg<PX>::EX > PX ? XReg<PX>::EX : PX) | 1;
    static constexpr int LINE = L * LS;
    static constexpr int SPEC = 3 * ROWS * KX;
    static constexpr int BUF = !TIGHT && SPEC > LINE ? SPEC : LINE;
    static constexpr int NBUF = TIGHT ? 1 : 2;
    // thermal: the rows' normals, drawn while the spectrum loads are in
    // flight, [3][R2][PX] pairs (where the CTAs of OCC still fit)
    static constexpr bool PRE = TH && PX <= 256 && !TIGHT;
    static constexpr int NOISE = PRE ? 3 * R2 * PX : 0;
    // 32- to 256-point lines: register four-step transforms, one exchange buffer per line
    static constexpr int EX = XReg<PX>::OK && !TIGHT ? L * XReg<PX>::EX : 0;
    static constexpr int SMEM = (PX + NBUF * BUF + EX + NOISE) * 8;
    static_assert(ROWS % 2 == 0, "line layout");
    static_assert(XReg<PX>::OK ? L * XReg<PX>::T <= NT : L * TPL <= NT, "lines per CTA");
    // CTAs per SM: 64 registers per thread; the general form's 96 or so
    static constexpr int OCC = SZ == 0 ? 2 : (SZ == 2 ? 8 : 4);
    static constexpr int GOCC = SZ == 0 ? 1 : (SZ == 2 ? 4 : 2);
};

// The body of the fused x pass: begin() runs once the previous kernel's
// writes are visible; pre(p, x, i, both) is called for every row pair p and x
// of the CTA (sites i and, if both, i + nx) while the spectrum loads are in
// flight; site(i, row, x, y, z, A..., r...) gives the new spin of site i in the
// dipole field A, or with PAIR site(i, p, ...) those of i and i + nx.
template <int PX, bool TH, int SZ, bool PAIR, bool HZ, class Begin, class Pre, class Site>
__device__ __forceinline__ void xstep_body(const ConvK& c, const DevStep* adv_cur, DevStep* adv_next, int fwd,
                                           const float2* __restrict__ tw, float2* __restrict__ spec,
                                           const float* __restrict__ sx, const float* __restrict__ sy,
                                           const float* __restrict__ sz, float* __restrict__ hx,
                                           float* __restrict__ hy, float* __restrict__ hz, float* __restrict__ ox,
                                           float* __restrict__ oy, float* __restrict__ oz, Begin&& begin, Pre&& pre,
                                           Site&& site)
{
    using X = XSCfg<PX, TH, SZ>;
    constexpr int KX = X::KX, NT = X::NT, ROWS = X::ROWS, R2 = X::R2, LS = X::LS;
    extern __shared__ float2 sm[];
    float2* twl = sm;               // [PX]
    float2* A = twl + PX;                       // [L][LS] lines
    float2* B = X::TIGHT ? A : A + X::BUF;      // [L][LS] scratch
    float2* EXB = B + X::BUF;                   // [L][XReg<PX>::EX] exchange buffers (XReg<PX>::OK)
    const int nx = c.nx, ny = c.ny, nz = c.nz;
    const int nr = nz * ny;                     // rows (z, y), flattened
    const int row0 = blockIdx.x * ROWS;
    const int rows_here = min(ROWS, nr - row0);
    // items of the site step: (row pair, x) of the padded lines, or of the
    // sites alone (TIGHT), then divided by multiplication
    constexpr int XW = HZ ? PX / 2 : PX;
    constexpr int IP = (R2 * XW + NT - 1) / NT;
    const int npair = R2 * nx;
    const unsigned mnx = nx > 1 ? 0xffffffffu / (unsigned)nx + 1u : 0u;
    const auto items = [&](auto&& f) {
        if constexpr (X::TIGHT) {
#pragma unroll 1
            for (int idx = threadIdx.x; idx < npair; idx += NT) {
                const int p = mnx ? (int)__umulhi((unsigned)idx, mnx) : idx;
                f(p, idx - p * nx, true);
            }
        } else {
#pragma unroll 1
            for (int it = 0; it < IP; it++) {
                const int idx = threadIdx.x + it * NT;
                if (idx >= R2 * XW) break;
                const int p = idx / XW, x = idx % XW;
                f(p, x, x < nx);
            }
        }
    };
    for (int k = threadIdx.x; k < PX; k += NT) twl[k] = tw[k];
    pdl_trigger();
    pdl_wait();
    unsigned long long* tls = c.tl ? c.tl + 2 : nullptr;
    tl_start(tls);
    // captured steps: the next step's block (the other of the pair; no
    // kernel of this step reads it)
    if (adv_next && blockIdx.x == 0 && threadIdx.x == 0) {
        const DevStep* cu = adv_cur;
        DevStep* nx_ = adv_next;
        nx_->th_counter = cu->th_counter + 1ull;
        for (int a = 0; a < 3; a++) {
            nx_->B[a] = cu->B[a] + cu->dB[a];
            nx_->dB[a] = cu->dB[a];
        }
    }
    if (c.run_if && *c.run_if == 0) return;
    // the rows' spins and their z-neighbour rows, into L2 while the inverse
    // transform runs (the step reads them after it)
    if (threadIdx.x < 9) {
        const int comp = threadIdx.x % 3, which = threadIdx.x / 3;
        const int r = which == 0 ? row0 : (which == 1 ? row0 - ny : row0 + ny);
        const float* base = comp == 0 ? sx : (comp == 1 ? sy : sz);
        if (r >= 0 && r + rows_here <= nr) {
            const float* p = base + (size_t)r * nx;
            const unsigned bytes = (unsigned)(rows_here * nx * sizeof(float));
            if ((((uintptr_t)p) & 15) == 0 && (bytes & 15) == 0)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
        }
    }
    begin();
    // 1. line l = comp R2 + p: Z[k] = S_row(2p)[k] + i S_row(2p+1)[k] for
    // k < KX, Hermitian completion Z[PX - k] from the conjugates; one item
    // per (kx, comp, p), the row pair's two spectrum values (adjacent in
    // SPEC[kx][comp][row]) loaded together when the pair is 16-byte aligned
    constexpr int NPI = KX * 3 * R2;
    constexpr int IS = (NPI + NT - 1) / NT;
    {
        float4 v[IS];
        const bool pair_ld = (nr & 1) == 0;   // row0 is even: (kx 3 + comp) nr + row0 + 2p is even
#pragma unroll
        for (int it = 0; it < IS; it++) {
            const int idx = threadIdx.x + it * NT;
            const int kx = idx / (3 * R2), rem = idx % (3 * R2);
            const int comp = rem / R2, p = rem % R2;
            v[it] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (idx < NPI && 2 * p < rows_here) {
                const float2* src = spec + ((size_t)kx * 3 + comp) * nr + row0 + 2 * p;
                if (pair_ld && 2 * p + 1 < rows_here) {
                    v[it] = *reinterpret_cast<const float4*>(src);
                } else {
                    const float2 a = src[0];
                    const float2 b = 2 * p + 1 < rows_here ? src[1] : make_float2(0.f, 0.f);
                    v[it] = make_float4(a.x, a.y, b.x, b.y);
                }
            }
        }
        // the normals of this thread's sites in the step below, while the
        // loads are in flight
        if (X::PRE)
            items([&](int p, int x, bool in) {
                if (2 * p < rows_here && in) pre(p, x, (row0 + 2 * p) * nx + x, 2 * p + 1 < rows_here);
            });
#pragma unroll
        for (int it = 0; it < IS; it++) {
            const int idx = threadIdx.x + it * NT;
            if (idx >= NPI) continue;
            const int kx = idx / (3 * R2), l = idx % (3 * R2);   // l = comp R2 + p
            float2* Zl = A + l * LS;
            float2 a = make_float2(v[it].x, v[it].y), b = make_float2(v[it].z, v[it].w);
            Zl[kx] = make_float2(a.x - b.y, a.y + b.x);
            if (kx > 0 && kx < PX - KX + 1) {
                a = cconj(a); b = cconj(b);
                Zl[PX - kx] = make_float2(a.x - b.y, a.y + b.x);
            }
        }
    }
    __syncthreads();
    const int l = threadIdx.x / X::TPL, tl = threadIdx.x % X::TPL;
    const float2* R;
    if constexpr (XReg<PX>::OK) {
        xreg_lines<PX, +1, X::TIGHT, HZ>(A, LS, X::L, EXB, twl);
        R = A;
    } else {
        R = fr::sm_fft<PX, +1, X::TPL, float2, LS>(A, B, l, tl, twl, l < X::L);
    }
    // the new spins' lines (FWD): the free buffer, or (TIGHT) each where its
    // item read the field
    float2* W = (R == A) ? B : A;
    // 2. field of the rows to the slot (unless a later step of the same launch
    // overwrites it: hx null), then the step of every site: one (row pair, x)
    // per item, the pair's two rows the real and imaginary parts of one line
    // element
    // (z, y) of the CTA's first row; a later row's by counting forward (no
    // division per site)
    const int zr0 = row0 / ny, yr0 = row0 - zr0 * ny;
    if (X::TIGHT && fwd && nx < XW) {   // zero padding of the new lines
        for (int idx = threadIdx.x; idx < 3 * R2 * (XW - nx); idx += NT) {
            const int l = idx % (3 * R2);
            W[l * LS + nx + idx / (3 * R2)] = make_float2(0.f, 0.f);
        }
    }
    items([&](int p, int x, bool in) {
        const float2 Ax2 = R[(0 * R2 + p) * LS + x], Ay2 = R[(1 * R2 + p) * LS + x], Az2 = R[(2 * R2 + p) * LS + x];
        float2 o0 = make_float2(0.f, 0.f), o1 = o0, o2 = o0;
        int zz = zr0, y = yr0 + 2 * p;
        while (y >= ny) { y -= ny; zz++; }
        if constexpr (PAIR) {
            // ny is even: the pair lies in one layer, and both rows exist
            if (2 * p < rows_here && in) {
                const int i = (row0 + 2 * p) * nx + x;
                if (hx) {
                    hx[i] = Ax2.x; hy[i] = Ay2.x; hz[i] = Az2.x;
                    hx[i + nx] = Ax2.y; hy[i + nx] = Ay2.y; hz[i + nx] = Az2.y;
                }
                site(i, p, x, y, zz, Ax2, Ay2, Az2, o0, o1, o2);
                ox[i] = o0.x; oy[i] = o1.x; oz[i] = o2.x;
                ox[i + nx] = o0.y; oy[i + nx] = o1.y; oz[i + nx] = o2.y;
            }
        } else {
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                const int row = 2 * p + h;
                if (h && ++y >= ny) { y -= ny; zz++; }
                if (row < rows_here && in) {
                    const float Ax = h ? Ax2.y : Ax2.x, Ay = h ? Ay2.y : Ay2.x, Az = h ? Az2.y : Az2.x;
                    const size_t i = (size_t)(row0 + row) * nx + x;
                    if (hx) { hx[i] = Ax; hy[i] = Ay; hz[i] = Az; }
                    float rx, ry, rz;
                    site((int)i, row, x, y, zz, Ax, Ay, Az, rx, ry, rz);
                    ox[i] = rx; oy[i] = ry; oz[i] = rz;
                    if (h) { o0.y = rx; o1.y = ry; o2.y = rz; }
                    else { o0.x = rx; o1.x = ry; o2.x = rz; }
                }
            }
        }
        if (fwd) { W[(0 * R2 + p) * LS + x] = o0; W[(1 * R2 + p) * LS + x] = o1; W[(2 * R2 + p) * LS + x] = o2; }
    });
    if (!fwd) {
        tl_end(tls);
        return;
    }
    __syncthreads();
    // 3. forward transform of the new spins' lines, split into the two rows
    const float2* Q;
    if constexpr (XReg<PX>::OK) {
        xreg_lines<PX, -1, X::TIGHT, HZ>(W, LS, X::L, EXB, twl);
        Q = W;
    } else {
        Q = fr::sm_fft<PX, -1, X::TPL, float2, LS>(W, const_cast<float2*>(R), l, tl, twl, l < X::L);
    }
    constexpr int IQ = (X::SPEC + NT - 1) / NT;
#pragma unroll
    for (int it = 0; it < IQ; it++) {
        const int idx = threadIdx.x + it * NT;
        const int kx = idx / (3 * ROWS), rem = idx % (3 * ROWS);
        const int comp = rem / ROWS, row = rem % ROWS;
        if (idx >= X::SPEC || row >= rows_here) continue;
        const float2* Z = Q + (comp * R2 + (row >> 1)) * LS;
        const float2 zk = Z[kx], zn = Z[(PX - kx) & (PX - 1)];
        float2 o;
        if ((row & 1) == 0) o = make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y - zn.y));
        else o = make_float2(0.5f * (zk.y + zn.y), 0.5f * (zn.x - zk.x));
        spec[((size_t)kx * 3 + comp) * nr + row0 + row] = o;
    }
    tl_end(tls);
}

// PAIR: two sites at a time (fused_pair), for an even number of rows per layer
// and at most 2^30 sites.
template <int PX, int LT, bool ANI, bool TH, int SZ, bool PAIR, bool HZ>
__global__ void __launch_bounds__(XSCfg<PX, TH, SZ>::NT, XSCfg<PX, TH, SZ>::OCC) k_xstep(ConvK c, FastK F0,
                                                  int fwd, const float2* __restrict__ tw,
                                                  float2* __restrict__ spec, const float* __restrict__ sx,
                                                  const float* __restrict__ sy, const float* __restrict__ sz,
                                                  float* __restrict__ hx, float* __restrict__ hy,
                                                  float* __restrict__ hz, float* __restrict__ ox,
                                                  float* __restrict__ oy, float* __restrict__ oz)
{
    using X = XSCfg<PX, TH, SZ>;
    constexpr int NP = X::R2 * PX;
    extern __shared__ float2 sm[];
    float2* noise = sm + PX + X::NBUF * X::BUF + X::EX;   // [3][R2][PX] row pairs (X::PRE)
    // the step block's values are the previous kernel's: resolved after the wait
    FastK F;
    const auto begin = [&] { F = fastk_resolved(F0); };
    const auto pre = [&](int p, int x, int i, bool both) {
        const float3 g = thermal_normal3(F, i);
        float3 k = make_float3(0.f, 0.f, 0.f);
        if (PAIR || both) k = thermal_normal3(F, i + c.nx);
        float2* q = noise + p * PX + x;
        q[0] = make_float2(g.x, k.x); q[NP] = make_float2(g.y, k.y); q[2 * NP] = make_float2(g.z, k.z);
    };
    if constexpr (PAIR) {
        xstep_body<PX, TH, SZ, true, HZ>(
            c, F0.adv_cur, F0.adv_next, fwd, tw, spec, sx, sy, sz, hx, hy, hz, ox, oy, oz, begin, pre,
            [&](int i, int p, int x, int y, int z, float2 Ax, float2 Ay, float2 Az, float2& rx, float2& ry, float2& rz) {
                const p2 A[3] = {pk(Ax.x, Ax.y), pk(Ay.x, Ay.y), pk(Az.x, Az.y)};
                p2 n[3] = {pk(0.f, 0.f), pk(0.f, 0.f), pk(0.f, 0.f)}, r[3];
                if (X::PRE) {
                    const float2* q = noise + p * PX + x;
                    n[0] = pk(q[0].x, q[0].y); n[1] = pk(q[NP].x, q[NP].y); n[2] = pk(q[2 * NP].x, q[2 * NP].y);
                } else if (TH) {
                    const float3 g = thermal_normal3(F, i), k = thermal_normal3(F, i + c.nx);
                    n[0] = pk(g.x, k.x); n[1] = pk(g.y, k.y); n[2] = pk(g.z, k.z);
                }
                fused_pair<LT, ANI, TH>(F, c.nx, c.ny, c.nz, x, y, z, i, sx, sy, sz, A, n, r);
                rx = up(r[0]); ry = up(r[1]); rz = up(r[2]);
            });
    } else {
        xstep_body<PX, TH, SZ, false, HZ>(
            c, F0.adv_cur, F0.adv_next, fwd, tw, spec, sx, sy, sz, hx, hy, hz, ox, oy, oz, begin, pre,
            [&](int i, int row, int x, int y, int z, float Ax, float Ay, float Az, float& rx, float& ry, float& rz) {
                float3 g;
                if (X::PRE) {
                    const float* q = reinterpret_cast<const float*>(noise + (row >> 1) * PX + x) + (row & 1);
                    g = make_float3(q[0], q[2 * NP], q[4 * NP]);
                }
                fused_site_v<LT, true, ANI, TH, true>(F, c.nx, c.ny, c.nz, x, y, z, i, sx, sy, sz, Ax, Ay, Az, rx, ry,
                                                      rz, X::PRE ? &g : nullptr);
            });
    }
}

// The same pass for per-site parameters, pathway lists and further addends
// (FusedK): P.terms without the dipole addend, whose weight is addw.  Every
// site step repeats k_fused_step's arithmetic, so fused and separate steps
// agree bit for bit.
template <int PX, int SZ>
__global__ void __launch_bounds__(XSCfg<PX, false, SZ>::NT, XSCfg<PX, false, SZ>::GOCC) k_xgstep(ConvK c, const __grid_constant__ FusedK P, double addw,
                                                            double dt_sys, const DevStep* cur, DevStep* next,
                                                            const float2* __restrict__ tw, float2* __restrict__ spec,
                                                            float* __restrict__ hx, float* __restrict__ hy,
                                                            float* __restrict__ hz)
{
    xstep_body<PX, false, SZ, false, false>(
        c, cur, next, 1, tw, spec, static_cast<const float*>(P.sys.x), static_cast<const float*>(P.sys.y),
        static_cast<const float*>(P.sys.z), hx, hy, hz, static_cast<float*>(P.ox), static_cast<float*>(P.oy),
        static_cast<float*>(P.oz), [] {}, [](int, int, int, bool) {},
        [&](int i, int, int, int, int, float Ax, float Ay, float Az, float& rx, float& ry, float& rz) {
            const float ms = ms_at<float>(P.sys, i);
            Fields<float> F;
            if (ms > 0.f) {
                F = eval_terms<float>(P.terms, P.sys, (float)dt_sys, i);
                F.H = fma3((float)addw, v3<float>(Ax, Ay, Az), F.H);
            }
            const V3<float> o = step_site<float>(P, F, spin_at<float>(P.sys, i), ms, i);
            rx = o.x; ry = o.y; rz = o.z;
        });
}

// The fused x pass of one size class of a packed ensemble: blockIdx.y the
// replica of the class, packed replica E.rep0 + blockIdx.y, its sites from
// E.base + blockIdx.y n on; each with its own applied field and thermal
// deviation (the CTA of its first rows writes the next step's field).  Noise is
// drawn by packed site, as in k_fused_ens.
// Bound by issue and the barriers between its phases.  It replaces the inverse
// x pass, the field slot, the fused step and the next step's forward x pass:
// 512 open replicas of 16x16x16 to 64x64x4 (3.6 M sites), thermal,
// 382 -> 308 us a step (301 -> 296 by the padded ends left out, HZ).
template <int PX, int LT, bool ANI, bool TH, int SZ, bool HZ>
__global__ void __launch_bounds__(XSCfg<PX, TH, SZ>::NT, XSCfg<PX, TH, SZ>::OCC)
    k_xens(ConvK c, FastK F0, XEns E, const float2* __restrict__ tw, float2* __restrict__ spec,
           const float* __restrict__ sx, const float* __restrict__ sy, const float* __restrict__ sz,
           float* __restrict__ ox, float* __restrict__ oy, float* __restrict__ oz)
{
    using X = XSCfg<PX, TH, SZ>;
    constexpr int NP = X::R2 * PX;
    extern __shared__ float2 sm[];
    float2* noise = sm + PX + X::NBUF * X::BUF + X::EX;   // [3][R2][PX] row pairs (X::PRE)
    const int n = c.nx * c.ny * c.nz, rep = E.rep0 + blockIdx.y, off = E.base + blockIdx.y * n;
    FastK F;
    const auto begin = [&] {
        F = fastk_resolved(F0);
        F.B[0] = (float)E.rB[3 * rep]; F.B[1] = (float)E.rB[3 * rep + 1]; F.B[2] = (float)E.rB[3 * rep + 2];
        if (TH) F.sigma = E.rsig[rep];
        if (blockIdx.x == 0 && threadIdx.x < 3)
            E.rBn[3 * rep + threadIdx.x] = E.rB[3 * rep + threadIdx.x] + E.rdB[3 * rep + threadIdx.x];
    };
    const float *s0 = sx + off, *s1 = sy + off, *s2 = sz + off;
    xstep_body<PX, TH, SZ, true, HZ>(
        c, nullptr, nullptr, 1, tw, spec + (size_t)blockIdx.y * c.Kx * 3 * c.nz * c.ny, s0, s1, s2, nullptr, nullptr,
        nullptr, ox + off, oy + off, oz + off, begin,
        [&](int p, int x, int i, bool) {
            const float3 g = thermal_normal3(F, off + i), k = thermal_normal3(F, off + i + c.nx);
            float2* q = noise + p * PX + x;
            q[0] = make_float2(g.x, k.x); q[NP] = make_float2(g.y, k.y); q[2 * NP] = make_float2(g.z, k.z);
        },
        [&](int i, int p, int x, int y, int z, float2 Ax, float2 Ay, float2 Az, float2& rx, float2& ry, float2& rz) {
            const p2 A[3] = {pk(Ax.x, Ax.y), pk(Ay.x, Ay.y), pk(Az.x, Az.y)};
            p2 nn[3] = {pk(0.f, 0.f), pk(0.f, 0.f), pk(0.f, 0.f)}, r[3];
            if (TH && !X::PRE) {
                const float3 g = thermal_normal3(F, off + i), k = thermal_normal3(F, off + i + c.nx);
                nn[0] = pk(g.x, k.x); nn[1] = pk(g.y, k.y); nn[2] = pk(g.z, k.z);
            } else if (TH) {
                const float2* q = noise + p * PX + x;
                nn[0] = pk(q[0].x, q[0].y); nn[1] = pk(q[NP].x, q[NP].y); nn[2] = pk(q[2 * NP].x, q[2 * NP].y);
            }
            fused_pair<LT, ANI, TH>(F, c.nx, c.ny, c.nz, x, y, z, i, s0, s1, s2, A, nn, r);
            rx = up(r[0]); ry = up(r[1]); rz = up(r[2]);
        });
}

// A stage of a Runge-Kutta scheme: the inverse x pass of the stage's field, its
// local terms and the rows it contributes to, two sites at a time; forward x
// pass of row 0, the next stage's spins (fwd).  Bound like k_xstep by the
// instructions of its sites; CTAs of 512 sites (two per SM at 128 registers).
// An RK4 step with a thermal kick of 256x256x8 as 10 kernels in place of 29
// (fields evaluated to slots and one pass per row and stage): alone 300 -> 169
// us, among others 211 -> 122.
template <int PX, int LT, bool ANI, int SZ>
__global__ void __launch_bounds__(XSCfg<PX, false, SZ>::NT, XSCfg<PX, false, SZ>::GOCC)
    k_xrk(ConvK c, const __grid_constant__ FastK F, const __grid_constant__ RkRows<float> rows, int fwd,
          const float2* __restrict__ tw, float2* __restrict__ spec, const float* sx, const float* sy, const float* sz,
          float* hx, float* hy, float* hz, float* ox, float* oy, float* oz)
{
    xstep_body<PX, false, SZ, true, false>(
        c, nullptr, nullptr, fwd, tw, spec, sx, sy, sz, hx, hy, hz, ox, oy, oz, [] {}, [](int, int, int, bool) {},
        [&](int i, int, int x, int y, int z, float2 Ax, float2 Ay, float2 Az, float2& rx, float2& ry, float2& rz) {
            p2 M[3], H[3], g[3], o[3];
            const p2 n = pk(0.f, 0.f);
            pair_near(F, c.nx, c.ny, c.nz, x, y, z, i, sx, sy, sz, M, H);
            fused_field<ANI, false, true, float, p2>(F, M[0], M[1], M[2], H[0], H[1], H[2], n, n, n, pk(Ax.x, Ax.y),
                                                     pk(Ay.x, Ay.y), pk(Az.x, Az.y), g[0], g[1], g[2]);
            rk_rows<LT, float, p2>(
                F, rows, M, H, [&](const float* b) { return pk(b[i], b[i + c.nx]); },
                [&](float* d, p2 v) {
                    const float2 u = up(v);
                    d[i] = u.x;
                    d[i + c.nx] = u.y;
                },
                o);
            rx = up(o[0]); ry = up(o[1]); rz = up(o[2]);
        });
}

// ------------------------------------------------------------------ launches
namespace mlb {

// Share of a CTA (XSCfg): the largest that gives at least about as many CTAs as
// SMs.  A step alone, share 0 / the one taken: 32x32x1 13.3 / 9.0 us, 64x64x2
// 15.0 / 9.0, 128x128x4 19.3 / 13.0, 256x256x1 22.9 / 17.1, 64x512x4 25.7 / 20.2,
// 512x512x1 60.6 / 41.2; 256x256x4 (128 CTAs of share 0) 26.1 at either.
template <int PX>
static int xs_size(const ConvK& c)
{
    const int nr = c.nz * c.ny;
    if (nr >= 120 * XSCfg<PX>::ROWS) return 0;
    if (PX > 128 || nr >= 120 * XSCfg<PX, false, 1>::ROWS) return 1;
    return 2;
}

template <int PX, int LT, bool ANI, bool TH, int SZ, bool PAIR, bool HZ>
static cudaError_t xstep_sz(const ConvK& c, const FastK& F, int fwd, const float2* tw, float2* spec,
                            const float* s[3], float* h[3], float* o[3], cudaStream_t st)
{
    using X = XSCfg<PX, TH, SZ>;
    dim3 grid((c.nz * c.ny + X::ROWS - 1) / X::ROWS, 1, 1);
    return launch_pdl_carved(k_xstep<PX, LT, ANI, TH, SZ, PAIR, HZ>, grid, dim3(X::NT), (size_t)X::SMEM, st, c, F, fwd, tw, spec,
                      s[0], s[1], s[2], h[0], h[1], h[2], o[0], o[1], o[2]);
}
template <int PX, int LT, bool ANI, bool TH, bool HZ>
static cudaError_t xstep_z(const ConvK& c, const FastK& F, int fwd, const float2* tw, float2* spec,
                           const float* s[3], float* h[3], float* o[3], cudaStream_t st)
{
    const int sz = xs_size<PX>(c);
    if (sz == 0) return xstep_sz<PX, LT, ANI, TH, 0, true, HZ>(c, F, fwd, tw, spec, s, h, o, st);
    if constexpr (PX <= 128)
        if (sz == 2) return xstep_sz<PX, LT, ANI, TH, 2, true, HZ>(c, F, fwd, tw, spec, s, h, o, st);
    return xstep_sz<PX, LT, ANI, TH, 1, true, HZ>(c, F, fwd, tw, spec, s, h, o, st);
}
// Rows that end in the first half of their lines (an open x) take HZ: half of
// the site loop's items and of the transforms' padded ends are never there.
// k_xstep of 128^3 open 102 -> 90 us.
template <int PX, int LT, bool ANI, bool TH>
static cudaError_t xstep_t(const ConvK& c, const FastK& F, int fwd, const float2* tw, float2* spec,
                           const float* s[3], float* h[3], float* o[3], cudaStream_t st)
{
    if (!xstep_pairs(c)) return xstep_sz<PX, LT, ANI, TH, 0, false, false>(c, F, fwd, tw, spec, s, h, o, st);
    if constexpr (XReg<PX>::OK)
        if (c.nx <= PX / 2) return xstep_z<PX, LT, ANI, TH, true>(c, F, fwd, tw, spec, s, h, o, st);
    return xstep_z<PX, LT, ANI, TH, false>(c, F, fwd, tw, spec, s, h, o, st);
}
template <int PX, int LT>
static cudaError_t xstep_lt(const ConvK& c, const FastK& F, int fwd, const float2* tw, float2* spec,
                            const float* s[3], float* h[3], float* o[3], cudaStream_t st)
{
    if (F.ani) {
        if (F.th) return xstep_t<PX, LT, true, true>(c, F, fwd, tw, spec, s, h, o, st);
        return xstep_t<PX, LT, true, false>(c, F, fwd, tw, spec, s, h, o, st);
    }
    if (F.th) return xstep_t<PX, LT, false, true>(c, F, fwd, tw, spec, s, h, o, st);
    return xstep_t<PX, LT, false, false>(c, F, fwd, tw, spec, s, h, o, st);
}
template <int PX>
static cudaError_t xstep_px(const ConvK& c, const FastK& F, int fwd, const float2* tw, float2* spec,
                            const float* s[3], float* h[3], float* o[3], cudaStream_t st)
{
    if (F.llg_type == LLG_CART) return xstep_lt<PX, LLG_CART>(c, F, fwd, tw, spec, s, h, o, st);
    return xstep_lt<PX, LLG_QUAT>(c, F, fwd, tw, spec, s, h, o, st);
}

template <int PX, int LT, bool ANI, bool TH>
static cudaError_t xens_t(const ConvK& c, const FastK& F, const XEns& E, const float2* tw, float2* spec,
                          const float* const s[3], float* const o[3], cudaStream_t st)
{
    constexpr int SZ = 3;
    using X = XSCfg<PX, TH, SZ>;
    return launch_pdl_carved(c.nx <= PX / 2 ? k_xens<PX, LT, ANI, TH, SZ, true> : k_xens<PX, LT, ANI, TH, SZ, false>,
                      dim3((c.nz * c.ny + X::ROWS - 1) / X::ROWS, c.nrep), dim3(X::NT), (size_t)X::SMEM, st, c, F, E, tw,
                      spec, s[0], s[1], s[2], o[0], o[1], o[2]);
}
template <int PX>
static cudaError_t xens_px(const ConvK& c, const FastK& F, const XEns& E, const float2* tw, float2* spec,
                           const float* const s[3], float* const o[3], cudaStream_t st)
{
    if (F.llg_type == LLG_CART) {
        if (F.ani) return F.th ? xens_t<PX, LLG_CART, true, true>(c, F, E, tw, spec, s, o, st)
                               : xens_t<PX, LLG_CART, true, false>(c, F, E, tw, spec, s, o, st);
        return F.th ? xens_t<PX, LLG_CART, false, true>(c, F, E, tw, spec, s, o, st)
                    : xens_t<PX, LLG_CART, false, false>(c, F, E, tw, spec, s, o, st);
    }
    if (F.ani) return F.th ? xens_t<PX, LLG_QUAT, true, true>(c, F, E, tw, spec, s, o, st)
                           : xens_t<PX, LLG_QUAT, true, false>(c, F, E, tw, spec, s, o, st);
    return F.th ? xens_t<PX, LLG_QUAT, false, true>(c, F, E, tw, spec, s, o, st)
                : xens_t<PX, LLG_QUAT, false, false>(c, F, E, tw, spec, s, o, st);
}

template <int PX, int LT, bool ANI, int SZ>
static cudaError_t xrk_sz(const ConvK& c, const FastK& F, const RkRows<float>& rows, int fwd, const float2* tw,
                          float2* spec, const float* const s[3], float* const h[3], float* const o[3], cudaStream_t st)
{
    using X = XSCfg<PX, false, SZ>;
    return launch_pdl(k_xrk<PX, LT, ANI, SZ>, dim3((c.nz * c.ny + X::ROWS - 1) / X::ROWS), dim3(X::NT), (size_t)X::SMEM,
                      st, c, F, rows, fwd, tw, spec, s[0], s[1], s[2], h[0], h[1], h[2], o[0], o[1], o[2]);
}
template <int PX, int LT, bool ANI>
static cudaError_t xrk_px(const ConvK& c, const FastK& F, const RkRows<float>& rows, int fwd, const float2* tw,
                          float2* spec, const float* const s[3], float* const h[3], float* const o[3], cudaStream_t st)
{
    const int sz = xs_size<PX>(c);
    if constexpr (PX <= 128)
        if (sz == 2) return xrk_sz<PX, LT, ANI, 2>(c, F, rows, fwd, tw, spec, s, h, o, st);
    return xrk_sz<PX, LT, ANI, 1>(c, F, rows, fwd, tw, spec, s, h, o, st);
}

template <int PX, int SZ>
static cudaError_t xgstep_sz(const ConvK& c, const FusedK& P, double addw, double dt_sys, const DevStep* cur,
                             DevStep* next, const float2* tw, float2* spec, float* const h[3], cudaStream_t st)
{
    using X = XSCfg<PX, false, SZ>;
    return launch_pdl(k_xgstep<PX, SZ>, dim3((c.nz * c.ny + X::ROWS - 1) / X::ROWS), dim3(X::NT), (size_t)X::SMEM, st, c,
                      P, addw, dt_sys, cur, next, tw, spec, h[0], h[1], h[2]);
}
template <int PX>
static cudaError_t xgstep_px(const ConvK& c, const FusedK& P, double addw, double dt_sys, const DevStep* cur,
                             DevStep* next, const float2* tw, float2* spec, float* const h[3], cudaStream_t st)
{
    const int sz = xs_size<PX>(c);
    if (sz == 0) return xgstep_sz<PX, 0>(c, P, addw, dt_sys, cur, next, tw, spec, h, st);
    if constexpr (PX <= 128)
        if (sz == 2) return xgstep_sz<PX, 2>(c, P, addw, dt_sys, cur, next, tw, spec, h, st);
    return xgstep_sz<PX, 1>(c, P, addw, dt_sys, cur, next, tw, spec, h, st);
}

template <int PX>
cudaError_t XUnit<PX>::init()
{
    return fr::fill_tables();
}
template <int PX>
cudaError_t XUnit<PX>::step(const ConvK& c, const FastK& F, int fwd, const float2* tw, float2* spec, const float* s[3],
                            float* h[3], float* o[3], cudaStream_t st)
{
    return xstep_px<PX>(c, F, fwd, tw, spec, s, h, o, st);
}
template <int PX>
cudaError_t XUnit<PX>::gstep(const ConvK& c, const FusedK& P, double addw, double dt_sys, const DevStep* cur,
                             DevStep* next, const float2* tw, float2* spec, float* const h[3], cudaStream_t st)
{
    return xgstep_px<PX>(c, P, addw, dt_sys, cur, next, tw, spec, h, st);
}
template <int PX>
cudaError_t XUnit<PX>::ens(const ConvK& c, const FastK& F, const XEns& E, const float2* tw, float2* spec,
                           const float* const s[3], float* const o[3], cudaStream_t st)
{
    // the normals of 512-point lines do not fit
    if constexpr (PX <= 256) return xens_px<PX>(c, F, E, tw, spec, s, o, st);
    return cudaErrorInvalidValue;
}
template <int PX>
cudaError_t XUnit<PX>::rk(const ConvK& c, const FastK& F, const RkRows<float>& rows, int fwd, const float2* tw,
                          float2* spec, const float* const s[3], float* const h[3], float* const o[3], cudaStream_t st)
{
    if (F.llg_type == LLG_CART)
        return F.ani ? xrk_px<PX, LLG_CART, true>(c, F, rows, fwd, tw, spec, s, h, o, st)
                     : xrk_px<PX, LLG_CART, false>(c, F, rows, fwd, tw, spec, s, h, o, st);
    return F.ani ? xrk_px<PX, LLG_QUAT, true>(c, F, rows, fwd, tw, spec, s, h, o, st)
                 : xrk_px<PX, LLG_QUAT, false>(c, F, rows, fwd, tw, spec, s, h, o, st);
}

} // namespace mlb
