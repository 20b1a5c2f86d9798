// mx.cu -- dipole convolution and fused step for lattice edges of any
// (31-smooth) length, FP32 and FP64 state, for tensors with the point-dipole
// parities (others, user tensors and sheared cells among them, keep the passes of
// kernels.cu).
//
//   k_mx_fx / k_mx_ix   x transforms of row pairs (two real rows per complex
//                       line) to and from SPEC[kx][c][z][y];
//   k_mx_yz             per kx: y transforms of the 3 nz data rows, the sum
//                       over source layers with the layer-pair tensor
//                       T(kx, ky, dz), inverse y transforms;
//   k_mx_step           inverse x transform, field terms + LLG, forward x
//                       transform of the new spins in one pass.
//
// Transforms.  A CTA's lines lie in shared memory and go through two or three
// stages of radix 2..31 butterflies, each held in one thread's registers and
// written back to the places it was read from: decimation in frequency
// forward (natural order in, digit-reversed out), decimation in time back.
// Nothing is reordered: the layer tensor is stored in the digit-reversed order
// of ky, and the x spectra are read and written through a table of kx places.
// So a line needs one buffer and a stage one barrier.  The stages a length
// takes are chosen on the host from the number of lines that share the CTA
// (mx_axis): few large butterflies leave threads idle, many small ones cost a
// barrier each; so is the padding of the lines against bank conflicts.  An
// inverse transform is the conjugate of the forward one of the conjugate.
//
// Layers.  The z direction is not transformed: with the point-dipole parities
// (checked on the FP64 tensor) T(kx, ky, dz) of XX, XY, YY, ZZ is real and
// even in dz, of XZ, YZ imaginary and odd, so nz^2 real multiplies per
// component pair replace the zero-padded transforms, nothing is padded, and
// the plane stays at 3 nz rows.
//
// What bounds them: at 100 to 300 CTAs of one wave each, a CTA's own chain of
// loads, stages and barriers (DRAM sees the tensor only); at a million sites
// instruction issue (400x500x5: 817 instructions per site in k_mx_step).
// Measured, one step alone, before (mixed-radix stages with runtime divisions,
// three components in turn, zero-padded z transforms, five kernels) and after:
// 200x150x5 FP32 122 -> 23 us, 128x128x4 FP64 37.5 -> 24 us, 32x95x3 FP64 173 ->
// 19 us, 128x58x3 with per-site anisotropy (prime factor 29) 381 -> 24 us,
// 32x32x1 FP64 25 -> 13 us.
#include "device.cuh"
#include "kparams.h"
#include "launch.h"
#include "mxradix.h"

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <vector>

// ------------------------------------------------------------------ host
namespace mlb {

static unsigned qmagic(int d) { return d <= 1 ? 0u : (unsigned)((1ull << 32) / (unsigned)d + 1ull); }

// Instructions of one radix-R butterfly, about: its arithmetic (real
// operations), and per point the accesses, addresses and twiddle
static double mx_ops(int R)
{
    if (R == 1) return 0;
    if (R == 2) return 4;
    if (R == 4) return 16;
    const int a = mx::first_factor(R);
    if (a == 0) {
        const double h = (R - 1) / 2;
        return 4 * h * h + 8 * h;
    }
    const int b = R / a;
    return b * mx_ops(a) + a * mx_ops(b) + 4.0 * (a - 1) * (b - 1);
}

static const int kRadix[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 15, 16, 17, 19, 23, 29, 31};

// Time of one stage of `items` radix-R butterflies on a CTA, in cycles: a
// chain of loads, arithmetic and stores, then the warps that share a
// scheduler one after the other.
static double mx_stage_cost(int R, int items, bool f64)
{
    const double instr = (f64 ? 2.0 : 1.0) * mx_ops(R) + 16.0 * R;
    return 150.0 + 4.0 * R + instr * std::max(1, (items + 127) / 128);
}

static double mx_best(int n, int total, bool f64, std::vector<int>& out)
{
    if (n == 1) {
        out.clear();
        return 0;
    }
    double best = 1e300;
    for (int R : kRadix) {
        if (n % R) continue;
        std::vector<int> rest;
        const double c = mx_stage_cost(R, total / R, f64) + mx_best(n / R, total, f64, rest);
        if (c < best) {
            best = c;
            out = rest;
            out.push_back(R);
        }
    }
    return best;
}

// Wavefronts of the axis' shared-memory accesses with padding shift sh: the
// first warps of every stage, elements of eb bytes; counted up to `limit`.
static int mx_conflicts(const MxAxis& ax, int sh, int nl, int eb, int limit)
{
    const int lanes = 128 / eb, LS = (ax.n + (ax.n >> sh)) | 1;
    int sum = 0, line[128], at[128];
    for (int i = 0; i < ax.nst; i++) {
        const MxStage& s = ax.s[i];
        const int total = std::min(nl * s.nb, 128);
        for (int t = 0; t < total; t++) {
            const int q = t % s.nb;
            line[t] = t / s.nb * LS;
            at[t] = (q / s.m) * s.m * s.R + q % s.m;
        }
        for (int w = 0; w < total; w += lanes)
            for (int r = 0, rm = 0; r < s.R; r++, rm += s.m) {
                int hit[16] = {0}, worst = 0;
                for (int t = w; t < std::min(w + lanes, total); t++) {
                    const int p = at[t] + rm;
                    worst = std::max(worst, ++hit[(line[t] + p + (p >> sh)) & (lanes - 1)]);
                }
                sum += worst;
                if (sum >= limit) return limit;
            }
    }
    return sum;
}

// The stages of an axis of n points of which a CTA holds nl lines, their
// padding, and the place of each frequency after the forward transform (into
// *at); false when n has a prime factor above 31.  prev: the axis of the same
// length and type for prev_nl lines, taken over if the search would be the same.
static bool mx_axis(int n, int nl, bool f64, MxAxis& ax, std::vector<int>* at, const MxAxis* prev = nullptr,
                    int prev_nl = 0)
{
    std::vector<int> r;
    if (mx_best(n, nl * n, f64, r) >= 1e300 || (int)r.size() > MX_MAX_STAGES) return false;
    memset(&ax, 0, sizeof(ax));
    ax.n = n;
    ax.nst = (int)r.size();
    ax.sh = 4;
    ax.big = std::any_of(r.begin(), r.end(), [](int R) { return R > 16; });
    // order and padding with the fewest bank conflicts; a large prime comes
    // last, where its butterflies need no twiddles
    std::sort(r.begin(), r.end());
    int best = 1 << 30;
    MxAxis t = ax;
    bool same = prev && prev->nst == ax.nst;
    if (same) {
        std::vector<int> pr;
        for (int i = 0; i < prev->nst; i++) pr.push_back(prev->s[i].R);
        std::sort(pr.begin(), pr.end());
        same = pr == r && std::all_of(r.begin(), r.end(), [&](int R) {
            return std::min(nl * (n / R), 128) == std::min(prev_nl * (n / R), 128);
        });
    }
    if (same) ax = *prev;
    else do {
        if (ax.big && r.back() <= 16) continue;
        int len = n;   // points of a block
        for (int i = 0; i < t.nst; i++) {
            MxStage& s = t.s[i];
            s.R = r[i];
            s.nb = n / r[i];
            s.m = len / r[i];
            s.tws = n / len;
            s.mnb = qmagic(s.nb);
            s.mm = qmagic(s.m);
            len = s.m;
        }
        for (int sh : {3, 4, 5, 30}) {
            const int c = mx_conflicts(t, sh, nl, f64 ? 16 : 8, best);
            if (c < best) {
                best = c;
                ax = t;
                ax.sh = sh;
            }
        }
    } while (std::next_permutation(r.begin(), r.end()));
    ax.LS = (n + (n >> ax.sh)) | 1;   // odd: the same place of consecutive lines in different banks
    if (at) {
        at->resize(n);
        for (int k = 0; k < n; k++) {
            int q = k, p = 0;
            for (int i = 0; i < ax.nst; i++) {
                p += (q % ax.s[i].R) * ax.s[i].m;
                q /= ax.s[i].R;
            }
            (*at)[k] = p;
        }
    }
    return true;
}

static size_t mx_smem_x(const MxAxis& ax, int nl, int rb)
{
    const size_t cb = 2 * rb;
    return ((size_t)ax.n + ((size_t)(ax.n / 2 + 1) * sizeof(int) + cb - 1) / cb + (size_t)nl * ax.LS) * cb;
}
static size_t mx_smem_y(const MxAxis& ax, int nl, int rb) { return ((size_t)ax.n + (size_t)nl * ax.LS) * 2 * rb; }

constexpr size_t MX_SMEM = 227 * 1024;

// The x passes' plan.  Rows per CTA: the estimated time of the busiest SM,
// waves of the CTAs it holds (a chain of latencies each) plus its share of the
// work, in cycles; sizes near a multiple of 148 CTAs differ by a whole wave.
bool mx_plan_x(const ConvK& c, int rb, MxX& x, std::vector<int>& at)
{
    memset(&x, 0, sizeof(x));
    if (c.nrep != 1 || c.Px > 8192) return false;
    const bool f64 = rb == 8;
    const int nr = c.nz * c.ny;
    double best = 1e300;
    int rows = 0;
    MxAxis prev;
    for (int r = 2; r <= 32; r += 2) {
        MxAxis ax;
        if (!mx_axis(c.Px, 3 * r / 2, f64, ax, nullptr, r > 2 ? &prev : nullptr, 3 * (r - 2) / 2)) return false;
        prev = ax;
        const size_t sm = mx_smem_x(ax, 3 * r / 2, rb);
        if (sm > MX_SMEM) break;
        const int regs = f64 ? (ax.big ? 1 : 2) : (ax.big ? 2 : 3);
        const int occ = std::max(1, std::min(regs, (int)(MX_SMEM / (sm + 1024))));
        const int per_sm = ((nr + r - 1) / r + 147) / 148, sites = r * c.Px;
        const double t = (double)((per_sm + occ - 1) / occ) * (5000.0 + 6.0 * sites) + 10.0 * per_sm * sites;
        if (t < best) { best = t; rows = r; }
        if (r >= nr) break;
    }
    if (!rows) return false;
    mx_axis(c.Px, 3 * rows / 2, f64, x.ax, &at);
    for (int& p : at) p += p >> x.ax.sh;
    for (int k = 0; k <= c.Px / 2; k++) at[k] |= (k ? at[c.Px - k] : at[0]) << 16;
    x.nx = c.nx; x.ny = c.ny; x.nz = c.nz; x.nr = nr; x.Kx = c.Kx;
    x.rows = rows;
    x.m3r2 = qmagic(3 * rows / 2);
    x.mr2 = qmagic(rows / 2);
    x.mPx = qmagic(c.Px);
    x.mnx = qmagic(c.nx);
    return true;
}

bool mx_plan_yz(const ConvK& c, int rb, MxYZ& y, std::vector<int>& at)
{
    memset(&y, 0, sizeof(y));
    if (c.general || c.nrep != 1 || c.nz > 32 || c.Py > 8192) return false;
    const int nl = 3 * c.nz, pts = nl * c.Py;
    if (!mx_axis(c.Py, nl, rb == 8, y.ax, &at) || mx_smem_y(y.ax, nl, rb) > MX_SMEM) return false;
    y.ny = c.ny; y.nz = c.nz;
    y.mPy = qmagic(c.Py);
    y.mny = qmagic(c.ny);
    y.threads = pts >= 4096 && !(rb == 8 && y.ax.big) ? 512 : (pts >= 1024 ? 256 : 128);
    y.mcols = qmagic(y.threads / (c.nz <= 8 ? 3 : nl));
    return true;
}

static size_t mx_smem_lr2d(const MxAxis& ax, int nl, int rb)
{
    return ((size_t)ax.n + 2 * (size_t)nl * ax.LS) * 2 * rb;
}

bool mx_plan_lr2d(const ConvK& c, int rb, MxYZ& y, std::vector<int>& at)
{
    memset(&y, 0, sizeof(y));
    if (c.ny > 8192) return false;
    const int nl = 3 * c.nz;
    if (!mx_axis(c.ny, nl, rb == 8, y.ax, &at) || mx_smem_lr2d(y.ax, nl, rb) > MX_SMEM - 1024) return false;
    y.ny = c.ny; y.nz = c.nz;
    y.mny = qmagic(c.ny);
    y.threads = rb == 8 && y.ax.big ? 256 : (nl * c.ny >= 512 ? 512 : 256);
    return true;
}

static size_t mx_smem(const MxX& x, int rb) { return mx_smem_x(x.ax, 3 * x.rows / 2, rb); }

// a call of the translation unit that has the axis' radices
#define MX_UNIT(R, AX, CALL) ((AX).big ? MxUnit<R, true>::CALL : MxUnit<R, false>::CALL)

cudaError_t launch_mx_yz(const ConvK& c, const MxYZ& plan, const FftLen L[3], const void* tw, void* spec, const void* tz,
                         int rb, cudaStream_t st)
{
    Prof pf("k_conv_yz", st);
    MxYZ y = plan;
    y.run_if = c.run_if;
    y.g = c.g;
    const size_t sm = mx_smem_y(y.ax, 3 * c.nz, rb);
    if (rb == 8)
        return MX_UNIT(double, y.ax, yz(y, c.Kx, sm, static_cast<const double2*>(tw) + L[1].tw_off,
                                        static_cast<double2*>(spec), static_cast<const double*>(tz), st));
    return MX_UNIT(float, y.ax, yz(y, c.Kx, sm, static_cast<const float2*>(tw) + L[1].tw_off, static_cast<float2*>(spec),
                                   static_cast<const float*>(tz), st));
}

cudaError_t launch_mx_lr2d(const ConvK& c, const MxYZ& y, const FftLen L[3], const void* tw, void* spec, const void* Q,
                           const LR2DScale& sc, int rb, cudaStream_t st)
{
    Prof pf("k_lr2d_yz", st);
    const size_t qb = (size_t)c.Kx * c.ny * c.nz * c.nz * 9 * 2 * rb, sm = mx_smem_lr2d(y.ax, 3 * c.nz, rb);
    const int stream = qb > ((size_t)64 << 20) ? 1 : 0;
    if (rb == 8)
        return MX_UNIT(double, y.ax, lr2d(y, c.Kx, sm, sc, stream, static_cast<const double2*>(tw) + L[1].tw_off,
                                          static_cast<double2*>(spec), static_cast<const double2*>(Q), st));
    return MX_UNIT(float, y.ax, lr2d(y, c.Kx, sm, sc, stream, static_cast<const float2*>(tw) + L[1].tw_off,
                                     static_cast<float2*>(spec), static_cast<const float2*>(Q), st));
}

cudaError_t launch_mx_fx(const MxX& plan, const FftLen L[3], const void* tw, const void* const s[3], void* spec,
                         const int* run_if, int rb, cudaStream_t st)
{
    Prof pf("k_conv_fx", st);
    MxX x = plan;
    x.run_if = run_if;
    if (rb == 8)
        return MX_UNIT(double, x.ax, fx(x, mx_smem(x, rb), static_cast<const double2*>(tw) + L[0].tw_off, s,
                                        static_cast<double2*>(spec), st));
    return MX_UNIT(float, x.ax, fx(x, mx_smem(x, rb), static_cast<const float2*>(tw) + L[0].tw_off, s,
                                   static_cast<float2*>(spec), st));
}

cudaError_t launch_mx_ix(const MxX& plan, const FftLen L[3], const void* tw, const void* spec, void* const h[3],
                         const int* run_if, int rb, cudaStream_t st)
{
    Prof pf("k_conv_ix", st);
    MxX x = plan;
    x.run_if = run_if;
    if (rb == 8)
        return MX_UNIT(double, x.ax, ix(x, mx_smem(x, rb), static_cast<const double2*>(tw) + L[0].tw_off,
                                        static_cast<const double2*>(spec), h, st));
    return MX_UNIT(float, x.ax, ix(x, mx_smem(x, rb), static_cast<const float2*>(tw) + L[0].tw_off,
                                   static_cast<const float2*>(spec), h, st));
}

template <typename R>
cudaError_t launch_mx_step(const MxX& x, const FftLen L[3], const void* tw, void* spec, const FastKT<R>& F,
                           const R* const s[3], R* const h[3], R* const o[3], cudaStream_t st)
{
    typedef typename CT<R>::T C;
    Prof pf("k_xstep", st);
    return MX_UNIT(R, x.ax, step(x, mx_smem(x, sizeof(R)), static_cast<const C*>(tw) + L[0].tw_off, static_cast<C*>(spec),
                                 F, s, h, o, st));
}
template cudaError_t launch_mx_step<float>(const MxX&, const FftLen[3], const void*, void*, const FastKT<float>&,
                                           const float* const[3], float* const[3], float* const[3], cudaStream_t);
template cudaError_t launch_mx_step<double>(const MxX&, const FftLen[3], const void*, void*, const FastKT<double>&,
                                            const double* const[3], double* const[3], double* const[3], cudaStream_t);

template <typename R>
cudaError_t launch_mx_rk(const MxX& x, const FftLen L[3], const void* tw, void* spec, const FastKT<R>& F,
                         const RkRows<R>& rows, const R* const s[3], R* const h[3], R* const o[3], cudaStream_t st)
{
    typedef typename CT<R>::T C;
    Prof pf("k_xrk", st);
    return MX_UNIT(R, x.ax, rk(x, mx_smem(x, sizeof(R)), static_cast<const C*>(tw) + L[0].tw_off, static_cast<C*>(spec), F,
                               rows, s, h, o, st));
}
template cudaError_t launch_mx_rk<float>(const MxX&, const FftLen[3], const void*, void*, const FastKT<float>&,
                                         const RkRows<float>&, const float* const[3], float* const[3], float* const[3],
                                         cudaStream_t);
template cudaError_t launch_mx_rk<double>(const MxX&, const FftLen[3], const void*, void*, const FastKT<double>&,
                                          const RkRows<double>&, const double* const[3], double* const[3],
                                          double* const[3], cudaStream_t);

cudaError_t launch_mx_gstep(const MxX& x, const FftLen L[3], const void* tw, void* spec, const FusedK& P, double addw,
                            double dt_sys, const DevStep* cur, DevStep* next, void* const h[3], int rb, cudaStream_t st)
{
    Prof pf("k_xstep", st);
    if (rb == 8)
        return MX_UNIT(double, x.ax, gstep(x, mx_smem(x, rb), static_cast<const double2*>(tw) + L[0].tw_off,
                                           static_cast<double2*>(spec), P, addw, dt_sys, cur, next, h, st));
    return MX_UNIT(float, x.ax, gstep(x, mx_smem(x, rb), static_cast<const float2*>(tw) + L[0].tw_off,
                                      static_cast<float2*>(spec), P, addw, dt_sys, cur, next, h, st));
}

cudaError_t mx_init()
{
    cudaError_t e;
    if ((e = MxUnit<float, false>::init()) || (e = MxUnit<float, true>::init()) || (e = MxUnit<double, false>::init())) return e;
    return MxUnit<double, true>::init();
}

} // namespace mlb
