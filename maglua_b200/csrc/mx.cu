// mx.cu -- dipole convolution and fused step for lattice edges of any
// (31-smooth) length, FP32 and FP64 state.
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
// instruction issue (400x500x5: 830 instructions per site in k_mx_step).
// Measured, one step alone, before (mixed-radix stages with runtime divisions,
// three components in turn, zero-padded z transforms, five kernels) and after:
// 200x150x5 FP32 122 -> 23 us, 128x128x4 FP64 37.5 -> 24 us, 32x95x3 FP64 173 ->
// 19 us, 128x58x3 with per-site anisotropy (prime factor 29) 381 -> 24 us,
// 32x32x1 FP64 25 -> 13 us.
#include "device.cuh"
#include "fused.cuh"
#include "kparams.h"
#include "launch.h"
#include "terms.cuh"

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <vector>

namespace mx {

constexpr int MAXR = 31;
// w_R^k = exp(-2 pi i k / R) at R (R - 1) / 2 + k
constexpr int NW = MAXR * (MAXR + 1) / 2;
static __constant__ float2 c_wf[NW];
static __constant__ double2 c_wd[NW];

template <typename C> __device__ __forceinline__ C cw(int R, int k);
template <> __device__ __forceinline__ float2 cw<float2>(int R, int k) { return c_wf[R * (R - 1) / 2 + k]; }
template <> __device__ __forceinline__ double2 cw<double2>(int R, int k) { return c_wd[R * (R - 1) / 2 + k]; }

// ------------------------------------------------------------------ DFTs in registers
// First factor of a composite radix (0: prime)
__host__ __device__ constexpr int first_factor(int R)
{
    if (R > 4 && R % 4 == 0) return 4;
    for (int p = 2; p * p <= R; p++)
        if (R % p == 0) return p;
    return 0;
}

// Odd prime R: the half sums and differences of (r, R - r); out(k, X_k) takes
// each output as it is formed, so that a long butterfly never holds inputs
// and outputs at once.
template <int R, typename C, class F>
__device__ __forceinline__ void dft_prime(const C* v, F&& out)
{
    typedef decltype(C().x) T;
    constexpr int H = (R - 1) / 2;
    C t[H], d[H];
    C s = v[0];
#pragma unroll
    for (int r = 0; r < H; r++) {
        t[r] = cadd(v[r + 1], v[R - 1 - r]);
        d[r] = csub(v[r + 1], v[R - 1 - r]);
        s = cadd(s, t[r]);
    }
    out(0, s);
#pragma unroll
    for (int k = 1; k <= H; k++) {
        T ax = v[0].x, ay = v[0].y, bx = 0, by = 0;
#pragma unroll
        for (int r = 1; r <= H; r++) {
            const C w = cw<C>(R, (r * k) % R);
            ax += w.x * t[r - 1].x; ay += w.x * t[r - 1].y;
            bx += w.y * d[r - 1].x; by += w.y * d[r - 1].y;
        }
        out(k, cmk<C>(ax - by, ay + bx));
        out(R - k, cmk<C>(ax + by, ay - bx));
    }
}

template <int R, typename C>
__device__ __forceinline__ void dft(C* v)
{
    constexpr int R1 = first_factor(R);
    if constexpr (R == 2) {
        const C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (R == 4) {
        const C a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
        const C b0 = cadd(v[1], v[3]), b1 = cmul_i(csub(v[1], v[3]), -1);
        v[0] = cadd(a0, b0);
        v[2] = csub(a0, b0);
        v[1] = cadd(a1, b1);
        v[3] = csub(a1, b1);
    } else if constexpr (R1 == 0) {
        C o[R];
        dft_prime<R>(v, [&](int k, C x) { o[k] = x; });
#pragma unroll
        for (int k = 0; k < R; k++) v[k] = o[k];
    } else {
        constexpr int R2 = R / R1;
        C u[R];
#pragma unroll
        for (int n2 = 0; n2 < R2; n2++) {
            C a[R1];
#pragma unroll
            for (int n1 = 0; n1 < R1; n1++) a[n1] = v[n1 * R2 + n2];
            dft<R1>(a);
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++)
                u[k1 * R2 + n2] = n2 * k1 == 0 ? a[k1] : cmul(a[k1], cw<C>(R, n2 * k1));
        }
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) {
            dft<R2>(u + k1 * R2);
#pragma unroll
            for (int k2 = 0; k2 < R2; k2++) v[k1 + R1 * k2] = u[k1 * R2 + k2];
        }
    }
}

// ------------------------------------------------------------------ lines in shared memory
// n / d by multiplication, m = floor(2^32 / d) + 1 (0: d = 1); exact while
// n d < 2^32
__device__ __forceinline__ int qdiv(int n, unsigned m) { return m ? (int)__umulhi((unsigned)n, m) : n; }

// place of element i of a line
__device__ __forceinline__ int pd(const MxAxis& ax, int i) { return i + (i >> ax.sh); }

extern __shared__ __align__(16) unsigned char mx_sm[];

// One radix-R stage of `total` butterflies (nb per line), in place on the
// lines at element A; the axis' twiddle table lies at element 0.  Butterfly j
// of a block of R m points takes its points j, j + m, ...
template <int R, typename C, bool DIT>
__device__ __noinline__ void stage(int A, int total, const MxStage s, int LS, int sh)
{
    C* sm = reinterpret_cast<C*>(mx_sm);
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int l = qdiv(idx, s.mnb), i = idx - l * s.nb;
        const int blk = qdiv(i, s.mm), j = i - blk * s.m;
        const int o = blk * s.m * R + j;
        C* a = sm + A + l * LS;
        C v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int p = o + r * s.m;
            v[r] = a[p + (p >> sh)];
        }
        const int e = j * s.tws;   // twiddles w^{j r} of the block length
        if (DIT && s.m > 1) {
            int t = e;
#pragma unroll
            for (int r = 1; r < R; r++, t += e) v[r] = cmul(v[r], sm[t]);
        }
        if constexpr (first_factor(R) == 0 && R > 7) {
            dft_prime<R>(v, [&](int k, C x) {
                if (!DIT && k > 0) x = cmul(x, sm[e * k]);
                const int p = o + k * s.m;
                a[p + (p >> sh)] = x;
            });
        } else {
            dft<R>(v);
            if (!DIT && s.m > 1) {
                int t = e;
#pragma unroll
                for (int r = 1; r < R; r++, t += e) v[r] = cmul(v[r], sm[t]);
            }
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int p = o + r * s.m;
                a[p + (p >> sh)] = v[r];
            }
        }
    }
}

// The same for a prime radix when there are few butterflies: H + 1 threads
// per butterfly, thread k forming the outputs k and R - k from all inputs, so
// that a stage is R long and not R^2 / 2 (R = 31, 18 butterflies: the chain of
// one thread takes 3.5 us).  A turn's inputs are read before its outputs are
// written; the points of other turns are not touched.
template <int R, typename C, bool DIT>
__device__ __noinline__ void stage_split(int A, int total, const MxStage s, int LS, int sh)
{
    typedef decltype(C().x) T;
    constexpr int H = (R - 1) / 2;
    C* sm = reinterpret_cast<C*>(mx_sm);
    const int per = blockDim.x / (H + 1);   // butterflies of a turn
    const int b = threadIdx.x / (H + 1), k = threadIdx.x - b * (H + 1);
    const int wst = s.nb;                   // n / R: w_R^1 in the axis' table
    for (int b0 = 0; b0 < total; b0 += per) {
        const int idx = b0 + b;
        const bool act = b < per && idx < total;
        C x0 = cmk<C>(0, 0), x1 = x0;
        C* a = sm;
        int o = 0, e = 0;
        if (act) {
            const int l = qdiv(idx, s.mnb), i = idx - l * s.nb;
            const int blk = qdiv(i, s.mm), j = i - blk * s.m;
            o = blk * s.m * R + j;
            e = j * s.tws;
            a = sm + A + l * LS;
            const C v0 = a[o + (o >> sh)];
            T ax = v0.x, ay = v0.y, bx = 0, by = 0;
            int q = 0;
#pragma unroll 5
            for (int r = 1; r <= H; r++) {
                const int p = o + r * s.m, u = o + (R - r) * s.m;
                C f = a[p + (p >> sh)], g = a[u + (u >> sh)];
                if (DIT && s.m > 1) {
                    f = cmul(f, sm[e * r]);
                    g = cmul(g, sm[e * (R - r)]);
                }
                q += k;
                if (q >= R) q -= R;
                const C w = sm[q * wst];   // w_R^{r k}
                ax += w.x * (f.x + g.x); ay += w.x * (f.y + g.y);
                bx += w.y * (f.x - g.x); by += w.y * (f.y - g.y);
            }
            x0 = cmk<C>(ax - by, ay + bx);
            x1 = cmk<C>(ax + by, ay - bx);
            if (!DIT && s.m > 1) {
                x0 = cmul(x0, sm[e * k]);
                if (k > 0) x1 = cmul(x1, sm[e * (R - k)]);
            }
        }
        __syncthreads();
        if (act) {
            const int p = o + k * s.m, u = o + (R - k) * s.m;
            a[p + (p >> sh)] = x0;
            if (k > 0) a[u + (u >> sh)] = x1;
        }
    }
}

template <int R, typename C, bool DIT>
__device__ __forceinline__ void stage_prime(int A, int total, const MxStage s, int LS, int sh)
{
    // the split butterfly does about three times the arithmetic: taken while
    // the CTA's threads hold all of it in two turns
    if (total * ((R + 1) / 2) <= 2 * (int)blockDim.x) stage_split<R, C, DIT>(A, total, s, LS, sh);
    else stage<R, C, DIT>(A, total, s, LS, sh);
}

// Forward transforms of the nl lines at element A, in place: natural order to
// digit-reversed (DIT: back).  Every thread of the CTA calls it, and the CTA is
// synchronised after each stage.  BIG: the axis has a prime radix above 13,
// whose butterflies take twice the registers of the others.
template <typename C, bool DIT, bool BIG>
__device__ __forceinline__ void fft(int A, int nl, const MxAxis& ax)
{
    for (int i = 0; i < ax.nst; i++) {
        const MxStage s = ax.s[DIT ? ax.nst - 1 - i : i];
        const int total = nl * s.nb;
        switch (s.R) {
        case 2: stage<2, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 3: stage<3, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 4: stage<4, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 5: stage<5, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 6: stage<6, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 7: stage<7, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 8: stage<8, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 9: stage<9, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 10: stage<10, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 11: stage_prime<11, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 12: stage<12, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 13: stage_prime<13, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 15: stage<15, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        case 16: stage<16, C, DIT>(A, total, s, ax.LS, ax.sh); break;
        default:
            if constexpr (BIG) {
                switch (s.R) {
                case 17: stage_prime<17, C, DIT>(A, total, s, ax.LS, ax.sh); break;
                case 19: stage_prime<19, C, DIT>(A, total, s, ax.LS, ax.sh); break;
                case 23: stage_prime<23, C, DIT>(A, total, s, ax.LS, ax.sh); break;
                case 29: stage_prime<29, C, DIT>(A, total, s, ax.LS, ax.sh); break;
                case 31: stage_prime<31, C, DIT>(A, total, s, ax.LS, ax.sh); break;
                }
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ x passes
// A CTA owns `rows` (even) consecutive rows r = z ny + y of all three
// components: 3 R2 complex lines (R2 = rows / 2), line comp R2 + p holding
// rows 2p and 2p + 1 as real and imaginary parts.  Shared memory: twiddles
// [n], the places of kx (low half) and n - kx (high half) [n / 2 + 1], lines.
struct RowCta {
    int row0, here;   // first row, rows that exist
};
__device__ __forceinline__ RowCta row_cta(const MxX& m)
{
    RowCta c;
    c.row0 = blockIdx.x * m.rows;
    c.here = min(m.rows, m.nr - c.row0);
    return c;
}
template <typename C> __device__ __forceinline__ int* places(const MxAxis& ax)
{
    return reinterpret_cast<int*>(reinterpret_cast<C*>(mx_sm) + ax.n);
}
// element where the lines start (the table of places before them)
template <typename C> __device__ __forceinline__ int lines_at(const MxAxis& ax)
{
    return ax.n + ((ax.n / 2 + 1) * (int)sizeof(int) + (int)sizeof(C) - 1) / (int)sizeof(C);
}

// SPEC rows -> the conjugates of Hermitian lines
template <typename C>
__device__ __forceinline__ void load_lines(const MxX& m, const RowCta& rc, const C* __restrict__ spec, int A)
{
    C* sm = reinterpret_cast<C*>(mx_sm);
    const int* at = places<C>(m.ax);
    const int R2 = m.rows >> 1, n3 = 3 * R2, total = m.Kx * n3;
    constexpr int U = 4;   // row pairs in flight per thread
    for (int i0 = threadIdx.x; i0 < total; i0 += U * blockDim.x) {
        C a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int idx = i0 + u * blockDim.x;
            a[u] = b[u] = cmk<C>(0, 0);
            if (idx < total) {
                const int kx = qdiv(idx, m.m3r2), rem = idx - kx * n3;
                const int comp = qdiv(rem, m.mr2), p = rem - comp * R2;
                const C* src = spec + ((size_t)kx * 3 + comp) * m.nr + rc.row0 + 2 * p;
                if (2 * p < rc.here) a[u] = src[0];
                if (2 * p + 1 < rc.here) b[u] = src[1];
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int idx = i0 + u * blockDim.x;
            if (idx >= total) break;
            const int kx = qdiv(idx, m.m3r2), l = idx - kx * n3;
            C* Z = sm + A + l * m.ax.LS;
            // conj of Z[k] = S_2p[k] + i S_2p+1[k]; Z[n - k] from the
            // conjugate spectra
            const int pp = at[kx];
            Z[pp & 0xffff] = cmk<C>(a[u].x - b[u].y, -(a[u].y + b[u].x));
            if (kx > 0 && 2 * kx < m.ax.n) Z[pp >> 16] = cmk<C>(a[u].x + b[u].y, a[u].y - b[u].x);
        }
    }
}

// Transformed lines -> the two rows' spectra to SPEC
template <typename C>
__device__ __forceinline__ void store_spec(const MxX& m, const RowCta& rc, int A, C* __restrict__ spec)
{
    typedef decltype(C().x) R;
    const C* sm = reinterpret_cast<const C*>(mx_sm);
    const int* at = places<C>(m.ax);
    const int R2 = m.rows >> 1, n3 = 3 * R2, total = m.Kx * n3;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int kx = qdiv(idx, m.m3r2), l = idx - kx * n3;
        const int comp = qdiv(l, m.mr2), p = l - comp * R2;
        const C* Z = sm + A + l * m.ax.LS;
        const int pp = at[kx];
        const C zk = Z[pp & 0xffff], zn = Z[pp >> 16];
        C* dst = spec + ((size_t)kx * 3 + comp) * m.nr + rc.row0 + 2 * p;
        if (2 * p < rc.here) dst[0] = cmk<C>((R)0.5 * (zk.x + zn.x), (R)0.5 * (zk.y - zn.y));
        if (2 * p + 1 < rc.here) dst[1] = cmk<C>((R)0.5 * (zk.y + zn.y), (R)0.5 * (zn.x - zk.x));
    }
}

// twiddles and (at: global) the places of an axis to shared memory
template <typename C>
__device__ __forceinline__ void load_tables(const MxAxis& ax, const C* __restrict__ tw, const int* __restrict__ at)
{
    C* sm = reinterpret_cast<C*>(mx_sm);
    for (int k = threadIdx.x; k < ax.n; k += blockDim.x) {
        sm[k] = tw[k];
        if (at && k <= ax.n / 2) places<C>(ax)[k] = at[k];
    }
}

} // namespace mx

// CTAs of 256 threads per SM the registers allow
// (x passes), and the threads of a (y,z) CTA
template <typename R, bool BIG> struct Occ {
    static constexpr int X = sizeof(R) == 4 ? (BIG ? 2 : 3) : (BIG ? 1 : 2);
    static constexpr int YZ = sizeof(R) == 8 && BIG ? 256 : 512;
};

// Forward x transform of the spins to SPEC.
template <typename R, bool BIG>
__global__ void __launch_bounds__(256, Occ<R, BIG>::X) k_mx_fx(const __grid_constant__ MxX m, const typename CT<R>::T* __restrict__ tw,
                                                  const R* __restrict__ sx, const R* __restrict__ sy,
                                                  const R* __restrict__ sz, typename CT<R>::T* __restrict__ spec)
{
    typedef typename CT<R>::T C;
    using namespace mx;
    load_tables<C>(m.ax, tw, m.at);
    pdl_trigger();
    pdl_wait();
    if (m.run_if && *m.run_if == 0) return;
    C* sm = reinterpret_cast<C*>(mx_sm);
    const RowCta rc = row_cta(m);
    const int R2 = m.rows >> 1, A = lines_at<C>(m.ax);
    const int total = m.rows * m.ax.n;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int row = qdiv(idx, m.mPx), x = idx - row * m.ax.n;
        R v[3] = {0, 0, 0};
        if (x < m.nx && row < rc.here) {
            const size_t i = (size_t)(rc.row0 + row) * m.nx + x;
            v[0] = __ldg(sx + i); v[1] = __ldg(sy + i); v[2] = __ldg(sz + i);
        }
#pragma unroll
        for (int c = 0; c < 3; c++)
            reinterpret_cast<R*>(sm + A + (c * R2 + (row >> 1)) * m.ax.LS + pd(m.ax, x))[row & 1] = v[c];
    }
    __syncthreads();
    fft<C, false, BIG>(A, 3 * R2, m.ax);
    store_spec<C>(m, rc, A, spec);
}

// Inverse x transform of SPEC to the field.
template <typename R, bool BIG>
__global__ void __launch_bounds__(256, Occ<R, BIG>::X) k_mx_ix(const __grid_constant__ MxX m, const typename CT<R>::T* __restrict__ tw,
                                                  const typename CT<R>::T* __restrict__ spec, R* __restrict__ hx,
                                                  R* __restrict__ hy, R* __restrict__ hz)
{
    typedef typename CT<R>::T C;
    using namespace mx;
    load_tables<C>(m.ax, tw, m.at);
    pdl_trigger();
    pdl_wait();
    if (m.run_if && *m.run_if == 0) return;
    const C* sm = reinterpret_cast<const C*>(mx_sm);
    const RowCta rc = row_cta(m);
    const int R2 = m.rows >> 1, A = lines_at<C>(m.ax);
    __syncthreads();
    load_lines<C>(m, rc, spec, A);
    __syncthreads();
    fft<C, true, BIG>(A, 3 * R2, m.ax);
    const int total = rc.here * m.nx, cs = 2 * R2 * m.ax.LS;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int row = qdiv(idx, m.mnx), x = idx - row * m.nx;
        const size_t i = (size_t)(rc.row0 + row) * m.nx + x;
        const R* z = reinterpret_cast<const R*>(sm + A + (row >> 1) * m.ax.LS + pd(m.ax, x)) + (row & 1);
        const R s = (row & 1) ? (R)-1 : (R)1;   // conjugate
        hx[i] = s * z[0]; hy[i] = s * z[cs]; hz[i] = s * z[2 * cs];
    }
}

// ------------------------------------------------------------------ fused x pass of a step
// The CTA's rows through the inverse x transform (-> their dipole field,
// written to its slot unless hx is null), the field terms and LLG update of their sites (-> the
// new spins; neighbours read from the current spin arrays, which no CTA
// writes) and the forward x transform of the new spins (-> the next step's
// spectrum rows, the ones the CTA itself read).  site(i, x, y, z, A) returns
// the new spin of site i in the dipole field A.
namespace mx {
// captured steps: the next step's block (the other of the pair; no kernel
// of this step reads it)
__device__ __forceinline__ void next_block(const DevStep* cu, DevStep* nx)
{
    if (nx && blockIdx.x == 0 && threadIdx.x == 0) {
        nx->th_counter = cu->th_counter + 1ull;
        for (int a = 0; a < 3; a++) {
            nx->B[a] = cu->B[a] + cu->dB[a];
            nx->dB[a] = cu->dB[a];
        }
    }
}

template <typename R, bool BIG, class F>
__device__ __forceinline__ void step_rows(const MxX& m, typename CT<R>::T* __restrict__ spec, R* __restrict__ hx,
                                          R* __restrict__ hy, R* __restrict__ hz, R* __restrict__ ox,
                                          R* __restrict__ oy, R* __restrict__ oz, F&& site)
{
    typedef typename CT<R>::T C;
    C* sm = reinterpret_cast<C*>(mx_sm);
    const RowCta rc = row_cta(m);
    const int R2 = m.rows >> 1, LS = m.ax.LS, A = lines_at<C>(m.ax);
    __syncthreads();
    load_lines<C>(m, rc, spec, A);
    __syncthreads();
    fft<C, true, BIG>(A, 3 * R2, m.ax);
    const int zr0 = rc.row0 / m.ny, yr0 = rc.row0 - zr0 * m.ny;
    const int total = m.rows * m.ax.n, cs = 2 * R2 * LS;
    // a thread reads the field of its row and x and puts the new spin in the
    // same places
#pragma unroll 1
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int row = qdiv(idx, m.mPx), x = idx - row * m.ax.n;
        R* q = reinterpret_cast<R*>(sm + A + (row >> 1) * LS + pd(m.ax, x)) + (row & 1);
        V3<R> o = v3<R>(0, 0, 0);
        if (x < m.nx && row < rc.here) {
            const R s = (row & 1) ? (R)-1 : (R)1;   // conjugate
            const V3<R> Ad = v3<R>(s * q[0], s * q[cs], s * q[2 * cs]);
            int z = zr0, y = yr0 + row;
            while (y >= m.ny) { y -= m.ny; z++; }
            const int i = (rc.row0 + row) * m.nx + x;
            if (hx) { hx[i] = Ad.x; hy[i] = Ad.y; hz[i] = Ad.z; }
            o = site(i, x, y, z, Ad);
            ox[i] = o.x; oy[i] = o.y; oz[i] = o.z;
        }
        q[0] = o.x; q[cs] = o.y; q[2 * cs] = o.z;
    }
    __syncthreads();
    fft<C, false, BIG>(A, 3 * R2, m.ax);
    store_spec<C>(m, rc, A, spec);
}
} // namespace mx

// Uniform parameters (FastKT).
template <typename R, int LT, bool ANI, bool TH, bool BIG>
__global__ void __launch_bounds__(256, Occ<R, BIG>::X) k_mx_step(const __grid_constant__ MxX m, const __grid_constant__ FastKT<R> F,
                                                    const typename CT<R>::T* __restrict__ tw,
                                                    typename CT<R>::T* __restrict__ spec, const R* __restrict__ sx,
                                                    const R* __restrict__ sy, const R* __restrict__ sz,
                                                    R* __restrict__ hx, R* __restrict__ hy, R* __restrict__ hz,
                                                    R* __restrict__ ox, R* __restrict__ oy, R* __restrict__ oz)
{
    mx::load_tables<typename CT<R>::T>(m.ax, tw, m.at);
    pdl_trigger();
    pdl_wait();
    mx::next_block(F.adv_cur, F.adv_next);
    mx::step_rows<R, BIG>(m, spec, hx, hy, hz, ox, oy, oz, [&](int i, int x, int y, int z, V3<R> A) {
        V3<R> o;
        fused_site_v<LT, true, ANI, TH, true, R>(F, m.nx, m.ny, m.nz, x, y, z, i, sx, sy, sz, A.x, A.y, A.z, o.x, o.y,
                                                 o.z);
        return o;
    });
}

// A stage of a Runge-Kutta scheme (rk_rows).
template <typename R, int LT, bool ANI, bool BIG>
__global__ void __launch_bounds__(256, Occ<R, BIG>::X)
    k_mx_rk(const __grid_constant__ MxX m, const __grid_constant__ FastKT<R> F, const __grid_constant__ RkRows<R> rows,
            const typename CT<R>::T* __restrict__ tw, typename CT<R>::T* __restrict__ spec, const R* sx, const R* sy,
            const R* sz, R* hx, R* hy, R* hz, R* ox, R* oy, R* oz)
{
    mx::load_tables<typename CT<R>::T>(m.ax, tw, m.at);
    pdl_trigger();
    pdl_wait();
    mx::step_rows<R, BIG>(m, spec, hx, hy, hz, ox, oy, oz, [&](int i, int x, int y, int z, V3<R> A) {
        const GlobalSpins<R> ld{{sx, sy, sz}};
        const R M[3] = {ld(0, i), ld(1, i), ld(2, i)};
        R H[3], g[3], o[3];
        fused_near<true, R>(F, m.nx, m.ny, m.nz, x, y, z, i, ld, H[0], H[1], H[2]);
        fused_field<ANI, false, true, R, R>(F, M[0], M[1], M[2], H[0], H[1], H[2], (R)0, (R)0, (R)0, A.x, A.y, A.z, g[0],
                                            g[1], g[2]);
        rk_rows<LT, R, R>(F, rows, M, H, [&](const R* b) { return b[i]; }, [&](R* d, R v) { d[i] = v; }, o);
        return v3<R>(o[0], o[1], o[2]);
    });
}

// Per-site parameters, pathway lists, further addends (FusedK): P.terms
// without the dipole addend, whose weight is addw.
template <typename R, bool BIG>
__global__ void __launch_bounds__(256, BIG && sizeof(R) == 8 ? 1 : 2) k_mx_gstep(const __grid_constant__ MxX m, const __grid_constant__ FusedK P,
                                                     double addw, double dt_sys, const DevStep* cur, DevStep* next,
                                                     const typename CT<R>::T* __restrict__ tw,
                                                     typename CT<R>::T* __restrict__ spec, R* __restrict__ hx,
                                                     R* __restrict__ hy, R* __restrict__ hz)
{
    mx::load_tables<typename CT<R>::T>(m.ax, tw, m.at);
    pdl_trigger();
    pdl_wait();
    mx::next_block(cur, next);
    mx::step_rows<R, BIG>(m, spec, hx, hy, hz, static_cast<R*>(P.ox), static_cast<R*>(P.oy), static_cast<R*>(P.oz),
                     [&](int i, int, int, int, V3<R> A) {
                         const R ms = ms_at<R>(P.sys, i);
                         Fields<R> F;
                         if (ms > (R)0) {
                             F = eval_terms<R>(P.terms, P.sys, (R)dt_sys, i);
                             F.H = fma3((R)addw, A, F.H);
                         }
                         return step_site<R>(P, F, spin_at<R>(P.sys, i), ms, i);
                     });
}

// ------------------------------------------------------------------ (y,z) pass
// One CTA per kx.  Layer sum of component a at column ky:
//   H_a[zt] = g sum_b sum_zs T_ab(zt - zs) M_b[zs],
// T_ab(dz) real and even in dz, or (exactly one of a, b is z) i times a real
// odd function.  tz: [kx][dz][6][ky].  One thread per (a, ky) keeps all NZ
// sums in registers (each spectrum value is read once per component, each
// tensor value once per thread); NZ = 0: one thread per (a, zt, ky).  ky: the
// digit-reversed places the transforms leave, in which tz is stored.
template <typename R, int NZ, bool BIG>
__global__ void __launch_bounds__(Occ<R, BIG>::YZ, 1) k_mx_yz(const __grid_constant__ MxYZ m, const typename CT<R>::T* __restrict__ tw,
                                                  typename CT<R>::T* __restrict__ spec, const R* __restrict__ tz)
{
    typedef typename CT<R>::T C;
    using namespace mx;
    const int kx = blockIdx.x, nz = NZ > 0 ? NZ : m.nz, ny = m.ny, Py = m.ax.n, LS = m.ax.LS;
    const int nl = 3 * nz;
    const R* T = tz + (size_t)kx * nz * 6 * Py;
    if (threadIdx.x == 0) {
        // this kx's tensor (constant between steps) starts towards L2
        const unsigned bytes = (unsigned)(nz * 6 * Py * sizeof(R));
        if ((((uintptr_t)T) & 15) == 0 && (bytes & 15) == 0)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(T), "r"(bytes) : "memory");
    }
    load_tables<C>(m.ax, tw, nullptr);
    pdl_trigger();
    pdl_wait();
    if (m.run_if && *m.run_if == 0) return;
    C* sm = reinterpret_cast<C*>(mx_sm);
    const int A = Py;
    C* sp = spec + (size_t)kx * nl * ny;
    constexpr int U = 4;
    {
        const int total = nl * Py;
        for (int i0 = threadIdx.x; i0 < total; i0 += U * blockDim.x) {
            C v[U];
            int at[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int idx = i0 + u * blockDim.x;
                const int l = qdiv(idx, m.mPy), y = idx - l * Py;
                v[u] = idx < total && y < ny ? sp[l * ny + y] : cmk<C>(0, 0);
                at[u] = A + l * LS + pd(m.ax, y);
            }
#pragma unroll
            for (int u = 0; u < U; u++)
                if (i0 + u * blockDim.x < total) sm[at[u]] = v[u];
        }
    }
    __syncthreads();
    fft<C, false, BIG>(A, nl, m.ax);
    // columns (places of the digit-reversed ky), as many at a time as the
    // CTA's threads cover whole: all of them are read before any is written
    const R g = (R)m.g;
    const int per = NZ > 0 ? 3 : nl, cols = blockDim.x / per;
    const int w = qdiv(threadIdx.x, m.mcols), c = threadIdx.x - w * cols;   // component (and layer), column
    for (int k0 = 0; k0 < Py; k0 += cols) {
        const int ky = k0 + c, kp = pd(m.ax, ky);
        const bool act = w < per && ky < Py;
        if constexpr (NZ > 0) {
            const int a = w;
            C acc[NZ];
#pragma unroll
            for (int z = 0; z < NZ; z++) acc[z] = cmk<C>(0, 0);
            if (act) {
#pragma unroll
                for (int b = 0; b < 3; b++) {
                    const int lo = min(a, b), hi = max(a, b);
                    const int q = lo == 0 ? hi : lo + hi + 1;   // XX XY XZ YY YZ ZZ
                    const bool odd = (a == 2) != (b == 2);
                    R t[NZ], tn[NZ];
#pragma unroll
                    for (int d = 0; d < NZ; d++) {
                        t[d] = __ldg(T + (d * 6 + q) * Py + ky);
                        tn[d] = odd ? -t[d] : t[d];
                    }
#pragma unroll
                    for (int zs = 0; zs < NZ; zs++) {
                        const C v = sm[A + (b * NZ + zs) * LS + kp];
                        const C s = odd ? cmk<C>(-v.y, v.x) : v;
#pragma unroll
                        for (int zt = 0; zt < NZ; zt++) {
                            const R u = zt >= zs ? t[zt - zs] : tn[zs - zt];
                            acc[zt].x += u * s.x;
                            acc[zt].y += u * s.y;
                        }
                    }
                }
            }
            __syncthreads();
            if (act) {
#pragma unroll
                for (int z = 0; z < NZ; z++) sm[A + (a * NZ + z) * LS + kp] = cmk<C>(g * acc[z].x, -(g * acc[z].y));
            }
        } else {
            const int a = w / nz, zt = w - a * nz;
            C acc = cmk<C>(0, 0);
            if (act) {
                for (int b = 0; b < 3; b++) {
                    const int lo = min(a, b), hi = max(a, b);
                    const int q = lo == 0 ? hi : lo + hi + 1;
                    const bool odd = (a == 2) != (b == 2);
                    for (int zs = 0; zs < nz; zs++) {
                        const int dz = zt - zs;
                        R u = __ldg(T + (abs(dz) * 6 + q) * Py + ky);
                        if (odd && dz < 0) u = -u;
                        const C v = sm[A + (b * nz + zs) * LS + kp];
                        acc.x += u * (odd ? -v.y : v.x);
                        acc.y += u * (odd ? v.x : v.y);
                    }
                }
            }
            __syncthreads();
            if (act) sm[A + w * LS + kp] = cmk<C>(g * acc.x, -(g * acc.y));
        }
    }
    __syncthreads();
    fft<C, true, BIG>(A, nl, m.ax);
    for (int idx = threadIdx.x; idx < nl * ny; idx += blockDim.x) {
        const int l = qdiv(idx, m.mny), y = idx - l * ny;
        sp[idx] = cconj(sm[A + l * LS + pd(m.ax, y)]);
    }
}

// ------------------------------------------------------------------ LongRange2D
// One CTA per kx: y transforms of the 3 nz rows, for every column the layer
// mixing
//   H_a[d] = dst[d] sum_s src[s] sum_b Q[s][d][ab] M_b[s]
// into a second buffer (no column waits for another), inverse y transforms.
// Q: [kx][s][d][9][ky], read once, one thread per (a, d, ky): consecutive
// threads take consecutive ky, three tensor values per source layer each, U
// layers in flight.  stream: Q is larger than the L2 keeps; its lines are
// evicted first.  Bound by one CTA's chain up to some 10 MB of Q, by its
// stream above (256x256x8: 151 MB).  A step of a film with these layers alone,
// before (y transforms, mixing and inverse y transforms as three passes, x
// passes apart: seven kernels) and after: 128x128x4 28.0 -> 19.4 us, 100x60x3
// 68.3 -> 15.0, 58x62x3 1334 -> 17.4, 256x256x8 75.4 -> 67.6.
template <typename R, bool BIG>
__global__ void __launch_bounds__(Occ<R, BIG>::YZ, 1) k_mx_lr2d(const __grid_constant__ MxYZ m,
                                                                const __grid_constant__ LR2DScale sc, int stream,
                                                                const typename CT<R>::T* __restrict__ tw,
                                                                typename CT<R>::T* __restrict__ spec,
                                                                const typename CT<R>::T* __restrict__ Q)
{
    typedef typename CT<R>::T C;
    using namespace mx;
    const int kx = blockIdx.x, nz = m.nz, ny = m.ny, LS = m.ax.LS, nl = 3 * nz;
    __shared__ R src[MLB_LR2D_MAXZ], dst[MLB_LR2D_MAXZ];
    if (threadIdx.x < nz) {
        src[threadIdx.x] = (R)sc.src[threadIdx.x];
        dst[threadIdx.x] = (R)sc.dst[threadIdx.x];
    }
    load_tables<C>(m.ax, tw, nullptr);
    pdl_trigger();
    pdl_wait();
    C* sm = reinterpret_cast<C*>(mx_sm);
    const int A = ny, B = A + nl * LS;
    C* sp = spec + (size_t)kx * nl * ny;
    for (int idx = threadIdx.x; idx < nl * ny; idx += blockDim.x) {
        const int l = qdiv(idx, m.mny), y = idx - l * ny;
        sm[A + l * LS + pd(m.ax, y)] = sp[idx];
    }
    __syncthreads();
    fft<C, false, BIG>(A, nl, m.ax);
    const C* Qk = Q + (size_t)kx * nz * nz * 9 * ny;
    constexpr int U = 4;
    for (int idx = threadIdx.x; idx < nl * ny; idx += blockDim.x) {
        const int w = qdiv(idx, m.mny), ky = idx - w * ny, kp = pd(m.ax, ky);
        const int a = w / nz, d = w - a * nz;
        C acc = cmk<C>(0, 0);
        for (int s0 = 0; s0 < nz; s0 += U) {
            C q[U][3];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const C* p = Qk + (((size_t)min(s0 + u, nz - 1) * nz + d) * 9 + 3 * a) * ny + ky;
#pragma unroll
                for (int b = 0; b < 3; b++) q[u][b] = stream ? __ldcs(p + (size_t)b * ny) : __ldg(p + (size_t)b * ny);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (s0 + u >= nz) break;
                const R v = src[s0 + u];
#pragma unroll
                for (int b = 0; b < 3; b++) {
                    const C M = sm[A + (b * nz + s0 + u) * LS + kp];
                    acc = cadd(acc, cmul(cmk<C>(v * q[u][b].x, v * q[u][b].y), M));
                }
            }
        }
        const R g = dst[d];
        sm[B + w * LS + kp] = cmk<C>(g * acc.x, -(g * acc.y));   // conjugate, for the inverse transform
    }
    __syncthreads();
    fft<C, true, BIG>(B, nl, m.ax);
    for (int idx = threadIdx.x; idx < nl * ny; idx += blockDim.x) {
        const int l = qdiv(idx, m.mny), y = idx - l * ny;
        sp[idx] = cconj(sm[B + l * LS + pd(m.ax, y)]);
    }
}

// ------------------------------------------------------------------ tensor
// T(kx, ky, dz) of six components from their FP64 transforms over x and y,
// W[q][z][ky][kx] (z = dz mod Pz): tz[kx][dz][q][at[ky]], the real part or (XZ,
// YZ) the imaginary part, ky at its place after the y transform.  stat: bits of the largest |W| and of the largest
// deviation from the parities the layer sum relies on.
template <typename R>
__global__ void k_mx_pack(const double2* W, int Px, int Py, int Pz, int nz, int Kx, const int* at, R* tz,
                          unsigned long long* stat)
{
    const long long total = (long long)Kx * nz * 6 * Py;
    double big = 0, dev = 0;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        // kx fastest for the reads: the writes are Py apart
        const int kx = (int)(e % Kx);
        long long r = e / Kx;
        const int ky = (int)(r % Py);
        r /= Py;
        const int q = (int)(r % 6), dz = (int)(r / 6);
        const double2* Wq = W + (size_t)q * Px * Py * Pz;
        const double2 v = Wq[((size_t)dz * Py + ky) * Px + kx];
        const double2 u = Wq[((size_t)((Pz - dz) % Pz) * Py + ky) * Px + kx];
        const bool odd = q == 2 || q == 4;
        tz[(((size_t)kx * nz + dz) * 6 + q) * Py + at[ky]] = (R)(odd ? v.y : v.x);
        big = fmax(big, fmax(fabs(v.x), fabs(v.y)));
        dev = fmax(dev, odd ? fmax(fmax(fabs(v.x), fabs(u.x)), fabs(v.y + u.y))
                            : fmax(fmax(fabs(v.y), fabs(u.y)), fabs(v.x - u.x)));
    }
    unsigned long long s[2] = {(unsigned long long)__double_as_longlong(big), (unsigned long long)__double_as_longlong(dev)};
    for (int k = 0; k < 2; k++) {
        unsigned long long x = s[k];
        for (int o = 16; o > 0; o >>= 1) x = max(x, __shfl_xor_sync(0xffffffffu, x, o));
        if ((threadIdx.x & 31) == 0 && x) atomicMax(stat + k, x);
    }
}

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

size_t mx_tensor_bytes(const ConvK& c, int rb) { return (size_t)c.Kx * c.nz * 6 * c.Py * rb; }

cudaError_t launch_mx_pack(const double2* W, const ConvK& c, const int* at, void* tz, unsigned long long* stat2, int rb,
                           cudaStream_t st)
{
    const long long total = (long long)c.Kx * c.nz * 6 * c.Py;
    const unsigned nb = (unsigned)std::min<long long>((total + 255) / 256, 148 * 8);
    if (rb == 8)
        k_mx_pack<double><<<nb, 256, 0, st>>>(W, c.Px, c.Py, c.Pz, c.nz, c.Kx, at, static_cast<double*>(tz),
                                              stat2);
    else
        k_mx_pack<float><<<nb, 256, 0, st>>>(W, c.Px, c.Py, c.Pz, c.nz, c.Kx, at, static_cast<float*>(tz),
                                             stat2);
    return cudaGetLastError();
}

template <typename R>
static cudaError_t mx_fx(const MxX& x, const typename CT<R>::T* tw, const void* const s[3],
                         typename CT<R>::T* spec, cudaStream_t st)
{
    Prof pf("k_conv_fx", st);
    return launch_pdl(x.ax.big ? k_mx_fx<R, true> : k_mx_fx<R, false>, dim3((x.nr + x.rows - 1) / x.rows), dim3(256),
                      mx_smem_x(x.ax, 3 * x.rows / 2, sizeof(R)), st, x, tw, static_cast<const R*>(s[0]),
                      static_cast<const R*>(s[1]), static_cast<const R*>(s[2]), spec);
}

template <typename R>
static cudaError_t mx_ix(const MxX& x, const typename CT<R>::T* tw, const typename CT<R>::T* spec, void* const h[3],
                         cudaStream_t st)
{
    Prof pf("k_conv_ix", st);
    return launch_pdl(x.ax.big ? k_mx_ix<R, true> : k_mx_ix<R, false>, dim3((x.nr + x.rows - 1) / x.rows), dim3(256),
                      mx_smem_x(x.ax, 3 * x.rows / 2, sizeof(R)), st, x, tw, spec, static_cast<R*>(h[0]),
                      static_cast<R*>(h[1]), static_cast<R*>(h[2]));
}

template <typename R, bool BIG>
static void (*yz_kernel_b(int nz))(MxYZ, const typename CT<R>::T*, typename CT<R>::T*, const R*)
{
    switch (nz) {
    case 1: return k_mx_yz<R, 1, BIG>;
    case 2: return k_mx_yz<R, 2, BIG>;
    case 3: return k_mx_yz<R, 3, BIG>;
    case 4: return k_mx_yz<R, 4, BIG>;
    case 5: return k_mx_yz<R, 5, BIG>;
    case 6: return k_mx_yz<R, 6, BIG>;
    case 7: return k_mx_yz<R, 7, BIG>;
    case 8: return k_mx_yz<R, 8, BIG>;
    }
    return k_mx_yz<R, 0, BIG>;
}
template <typename R>
static auto yz_kernel(int nz, bool big) { return big ? yz_kernel_b<R, true>(nz) : yz_kernel_b<R, false>(nz); }

template <typename R>
static cudaError_t mx_yz(const ConvK& c, const MxYZ& y, const typename CT<R>::T* tw, typename CT<R>::T* spec,
                         const R* tz, cudaStream_t st)
{
    Prof pf("k_conv_yz", st);
    return launch_pdl(yz_kernel<R>(c.nz, y.ax.big), dim3(c.Kx), dim3(y.threads), mx_smem_y(y.ax, 3 * c.nz, sizeof(R)), st, y, tw,
                      spec, tz);
}

cudaError_t launch_mx_yz(const ConvK& c, const MxYZ& plan, const FftLen L[3], const void* tw, void* spec, const void* tz,
                         int rb, cudaStream_t st)
{
    MxYZ y = plan;
    y.run_if = c.run_if;
    y.g = c.g;
    if (rb == 8)
        return mx_yz<double>(c, y, static_cast<const double2*>(tw) + L[1].tw_off, static_cast<double2*>(spec),
                             static_cast<const double*>(tz), st);
    return mx_yz<float>(c, y, static_cast<const float2*>(tw) + L[1].tw_off, static_cast<float2*>(spec),
                        static_cast<const float*>(tz), st);
}

template <typename R>
static cudaError_t mx_lr2d_t(const ConvK& c, const MxYZ& y, const FftLen L[3], const void* tw, void* spec,
                             const void* Q, const LR2DScale& sc, cudaStream_t st)
{
    typedef typename CT<R>::T C;
    Prof pf("k_lr2d_yz", st);
    const size_t qb = (size_t)c.Kx * c.ny * c.nz * c.nz * 9 * sizeof(C);
    return launch_pdl(y.ax.big ? k_mx_lr2d<R, true> : k_mx_lr2d<R, false>, dim3(c.Kx), dim3(y.threads),
                      mx_smem_lr2d(y.ax, 3 * c.nz, sizeof(R)), st, y, sc, qb > ((size_t)64 << 20) ? 1 : 0,
                      static_cast<const C*>(tw) + L[1].tw_off, static_cast<C*>(spec), static_cast<const C*>(Q));
}

cudaError_t launch_mx_lr2d(const ConvK& c, const MxYZ& y, const FftLen L[3], const void* tw, void* spec, const void* Q,
                           const LR2DScale& sc, int rb, cudaStream_t st)
{
    if (rb == 8) return mx_lr2d_t<double>(c, y, L, tw, spec, Q, sc, st);
    return mx_lr2d_t<float>(c, y, L, tw, spec, Q, sc, st);
}

cudaError_t launch_mx_fx(const MxX& plan, const FftLen L[3], const void* tw, const void* const s[3], void* spec,
                         const int* run_if, int rb, cudaStream_t st)
{
    MxX x = plan;
    x.run_if = run_if;
    if (rb == 8) return mx_fx<double>(x, static_cast<const double2*>(tw) + L[0].tw_off, s, static_cast<double2*>(spec), st);
    return mx_fx<float>(x, static_cast<const float2*>(tw) + L[0].tw_off, s, static_cast<float2*>(spec), st);
}

template <typename R>
using StepKernel = void (*)(MxX, FastKT<R>, const typename CT<R>::T*, typename CT<R>::T*, const R*, const R*, const R*,
                            R*, R*, R*, R*, R*, R*);

template <typename R, bool BIG>
static StepKernel<R> step_kernel_b(int llg, bool ani, bool th)
{
    if (llg == LLG_CART) {
        if (ani) return th ? k_mx_step<R, LLG_CART, true, true, BIG> : k_mx_step<R, LLG_CART, true, false, BIG>;
        return th ? k_mx_step<R, LLG_CART, false, true, BIG> : k_mx_step<R, LLG_CART, false, false, BIG>;
    }
    if (ani) return th ? k_mx_step<R, LLG_QUAT, true, true, BIG> : k_mx_step<R, LLG_QUAT, true, false, BIG>;
    return th ? k_mx_step<R, LLG_QUAT, false, true, BIG> : k_mx_step<R, LLG_QUAT, false, false, BIG>;
}
template <typename R>
static StepKernel<R> step_kernel(int llg, bool ani, bool th, bool big)
{
    return big ? step_kernel_b<R, true>(llg, ani, th) : step_kernel_b<R, false>(llg, ani, th);
}

template <typename R>
cudaError_t launch_mx_step(const MxX& x, const FftLen L[3], const void* tw, void* spec, const FastKT<R>& F,
                           const R* const s[3], R* const h[3], R* const o[3], cudaStream_t st)
{
    typedef typename CT<R>::T C;
    Prof pf("k_xstep", st);
    return launch_pdl(step_kernel<R>(F.llg_type, F.ani != 0, F.th != 0, x.ax.big), dim3((x.nr + x.rows - 1) / x.rows), dim3(256),
                      mx_smem_x(x.ax, 3 * x.rows / 2, sizeof(R)), st, x, F, static_cast<const C*>(tw) + L[0].tw_off,
                      static_cast<C*>(spec), s[0], s[1], s[2], h[0], h[1], h[2], o[0], o[1], o[2]);
}
template cudaError_t launch_mx_step<float>(const MxX&, const FftLen[3], const void*, void*, const FastKT<float>&,
                                           const float* const[3], float* const[3], float* const[3], cudaStream_t);
template cudaError_t launch_mx_step<double>(const MxX&, const FftLen[3], const void*, void*, const FastKT<double>&,
                                            const double* const[3], double* const[3], double* const[3], cudaStream_t);

template <typename R>
using RkKernel = void (*)(MxX, FastKT<R>, RkRows<R>, const typename CT<R>::T*, typename CT<R>::T*, const R*, const R*,
                          const R*, R*, R*, R*, R*, R*, R*);
template <typename R, bool BIG>
static RkKernel<R> rk_kernel_b(int llg, bool ani)
{
    if (llg == LLG_CART) return ani ? k_mx_rk<R, LLG_CART, true, BIG> : k_mx_rk<R, LLG_CART, false, BIG>;
    return ani ? k_mx_rk<R, LLG_QUAT, true, BIG> : k_mx_rk<R, LLG_QUAT, false, BIG>;
}

template <typename R>
cudaError_t launch_mx_rk(const MxX& x, const FftLen L[3], const void* tw, void* spec, const FastKT<R>& F,
                         const RkRows<R>& rows, const R* const s[3], R* const h[3], R* const o[3], cudaStream_t st)
{
    typedef typename CT<R>::T C;
    Prof pf("k_xrk", st);
    const auto k = x.ax.big ? rk_kernel_b<R, true>(F.llg_type, F.ani != 0) : rk_kernel_b<R, false>(F.llg_type, F.ani != 0);
    return launch_pdl(k, dim3((x.nr + x.rows - 1) / x.rows), dim3(256), mx_smem_x(x.ax, 3 * x.rows / 2, sizeof(R)), st, x,
                      F, rows, static_cast<const C*>(tw) + L[0].tw_off, static_cast<C*>(spec), s[0], s[1], s[2], h[0],
                      h[1], h[2], o[0], o[1], o[2]);
}
template cudaError_t launch_mx_rk<float>(const MxX&, const FftLen[3], const void*, void*, const FastKT<float>&,
                                         const RkRows<float>&, const float* const[3], float* const[3], float* const[3],
                                         cudaStream_t);
template cudaError_t launch_mx_rk<double>(const MxX&, const FftLen[3], const void*, void*, const FastKT<double>&,
                                          const RkRows<double>&, const double* const[3], double* const[3],
                                          double* const[3], cudaStream_t);

template <typename R>
static cudaError_t mx_gstep_t(const MxX& x, const FftLen L[3], const void* tw, void* spec, const FusedK& P, double addw,
                              double dt_sys, const DevStep* cur, DevStep* next, void* const h[3], cudaStream_t st)
{
    typedef typename CT<R>::T C;
    Prof pf("k_xstep", st);
    return launch_pdl(x.ax.big ? k_mx_gstep<R, true> : k_mx_gstep<R, false>, dim3((x.nr + x.rows - 1) / x.rows), dim3(256),
                      mx_smem_x(x.ax, 3 * x.rows / 2, sizeof(R)), st, x, P, addw, dt_sys, cur, next,
                      static_cast<const C*>(tw) + L[0].tw_off, static_cast<C*>(spec), static_cast<R*>(h[0]),
                      static_cast<R*>(h[1]), static_cast<R*>(h[2]));
}

cudaError_t launch_mx_gstep(const MxX& x, const FftLen L[3], const void* tw, void* spec, const FusedK& P, double addw,
                            double dt_sys, const DevStep* cur, DevStep* next, void* const h[3], int rb, cudaStream_t st)
{
    if (rb == 8) return mx_gstep_t<double>(x, L, tw, spec, P, addw, dt_sys, cur, next, h, st);
    return mx_gstep_t<float>(x, L, tw, spec, P, addw, dt_sys, cur, next, h, st);
}

cudaError_t launch_mx_ix(const MxX& plan, const FftLen L[3], const void* tw, const void* spec, void* const h[3],
                         const int* run_if, int rb, cudaStream_t st)
{
    MxX x = plan;
    x.run_if = run_if;
    if (rb == 8)
        return mx_ix<double>(x, static_cast<const double2*>(tw) + L[0].tw_off, static_cast<const double2*>(spec), h, st);
    return mx_ix<float>(x, static_cast<const float2*>(tw) + L[0].tw_off, static_cast<const float2*>(spec), h, st);
}

template <typename K>
static cudaError_t mx_max_smem(K kern)
{
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, kern);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(MX_SMEM - a.sharedSizeBytes));
}

template <typename R, bool BIG>
static cudaError_t mx_configure_t()
{
    cudaError_t e;
    if ((e = mx_max_smem(k_mx_fx<R, BIG>)) != cudaSuccess || (e = mx_max_smem(k_mx_ix<R, BIG>)) != cudaSuccess) return e;
    for (int nz = 0; nz <= 8; nz++)
        if ((e = mx_max_smem(yz_kernel_b<R, BIG>(nz))) != cudaSuccess) return e;
    for (int q = 0; q < 8; q++)
        if ((e = mx_max_smem(step_kernel_b<R, BIG>(q & 1 ? LLG_CART : LLG_QUAT, q & 2, q & 4))) != cudaSuccess) return e;
    for (int q = 0; q < 4; q++)
        if ((e = mx_max_smem(rk_kernel_b<R, BIG>(q & 1 ? LLG_CART : LLG_QUAT, q & 2))) != cudaSuccess) return e;
    if ((e = mx_max_smem(k_mx_lr2d<R, BIG>)) != cudaSuccess) return e;
    return mx_max_smem(k_mx_gstep<R, BIG>);
}

cudaError_t mx_configure()
{
    static float2 hf[mx::NW];
    static double2 hd[mx::NW];
    for (int R = 1; R <= mx::MAXR; R++)
        for (int k = 0; k < R; k++) {
            const double a = 2.0 * M_PI * k / R;
            hd[R * (R - 1) / 2 + k] = make_double2(cos(a), -sin(a));
            hf[R * (R - 1) / 2 + k] = make_float2((float)cos(a), (float)-sin(a));
        }
    cudaError_t e;
    if ((e = cudaMemcpyToSymbol(mx::c_wf, hf, sizeof(hf))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(mx::c_wd, hd, sizeof(hd))) != cudaSuccess) return e;
    if ((e = mx_configure_t<float, false>()) != cudaSuccess || (e = mx_configure_t<float, true>()) != cudaSuccess) return e;
    if ((e = mx_configure_t<double, false>()) != cudaSuccess) return e;
    return mx_configure_t<double, true>();
}

} // namespace mlb
