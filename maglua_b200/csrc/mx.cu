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
// Stockham stages of radix 2..31 (one butterfly per thread and turn, in
// registers).  The stages a length takes are chosen on the host from the
// number of lines that share the CTA (mx_axis): few large butterflies leave
// threads idle, many small ones cost a barrier each.  Indices use
// multiply-shift division; lines are padded (one element per 128 bytes) so
// that stride-R stores spread over the banks.  An inverse transform is the
// forward one with real and imaginary parts swapped on the way in and out.
//
// Layers.  The z direction is not transformed: with the point-dipole parities
// (checked on the FP64 tensor) T(kx, ky, dz) of XX, XY, YY, ZZ is real and
// even in dz, of XZ, YZ imaginary and odd, so nz^2 real multiplies per
// component pair replace the zero-padded transforms, nothing is padded, and
// the plane stays at 3 nz rows.
//
// What bounds them: at 100 to 200 CTAs of one wave each, a CTA's own chain of
// loads, stages and barriers (DRAM sees the tensor only).  Measured, one step
// alone, before (mixed-radix stages with runtime divisions, three components
// in turn, zero-padded z transforms) and after: 200x150x5 FP32 122 -> 33 us,
// 128x128x4 FP64 37.5 -> 31 us, 32x95x3 FP64 173 -> 29 us, 128x58x3 (prime
// factor 29) 381 -> 29 us.
#include "device.cuh"
#include "fused.cuh"
#include "kparams.h"
#include "launch.h"

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

template <typename C> struct Pad { static constexpr int SH = sizeof(C) == 8 ? 4 : 3; };
template <typename C> __device__ __forceinline__ int pd(int i) { return i + (i >> Pad<C>::SH); }

extern __shared__ __align__(16) unsigned char mx_sm[];

// One radix-R stage of `total` butterflies (nb per line) from the lines at
// element src to those at dst; the axis' twiddle table lies at element 0.
template <int R, typename C>
__device__ __noinline__ void stage(int src, int dst, int total, const MxStage s, int LS)
{
    C* sm = reinterpret_cast<C*>(mx_sm);
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int l = qdiv(idx, s.mnb), j = idx - l * s.nb;
        const C* a = sm + src + l * LS;
        C v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = a[pd<C>(j + r * s.nb)];
        const int q = qdiv(j, s.mNs), jm = j - q * s.Ns;
        if (s.Ns > 1) {
            const int e = jm * s.tws;
            int t = e;
#pragma unroll
            for (int r = 1; r < R; r++, t += e) v[r] = cmul(v[r], sm[t]);
        }
        C* b = sm + dst + l * LS;
        const int o = q * s.Ns * R + jm;
        if constexpr (first_factor(R) == 0 && R > 7) {
            dft_prime<R>(v, [&](int k, C x) { b[pd<C>(o + k * s.Ns)] = x; });
        } else {
            dft<R>(v);
#pragma unroll
            for (int r = 0; r < R; r++) b[pd<C>(o + r * s.Ns)] = v[r];
        }
    }
}

// Forward transforms of the nl lines at element a (line stride ax.LS), b a
// buffer of the same size; every thread of the CTA calls it, and the CTA is
// synchronised after each stage.  Returns the element where the result lies.
template <typename C>
__device__ __forceinline__ int fft(int a, int b, int nl, const MxAxis& ax)
{
    for (int i = 0; i < ax.nst; i++) {
        const MxStage s = ax.s[i];
        const int total = nl * s.nb;
        switch (s.R) {
        case 2: stage<2, C>(a, b, total, s, ax.LS); break;
        case 3: stage<3, C>(a, b, total, s, ax.LS); break;
        case 4: stage<4, C>(a, b, total, s, ax.LS); break;
        case 5: stage<5, C>(a, b, total, s, ax.LS); break;
        case 6: stage<6, C>(a, b, total, s, ax.LS); break;
        case 7: stage<7, C>(a, b, total, s, ax.LS); break;
        case 8: stage<8, C>(a, b, total, s, ax.LS); break;
        case 9: stage<9, C>(a, b, total, s, ax.LS); break;
        case 10: stage<10, C>(a, b, total, s, ax.LS); break;
        case 11: stage<11, C>(a, b, total, s, ax.LS); break;
        case 12: stage<12, C>(a, b, total, s, ax.LS); break;
        case 13: stage<13, C>(a, b, total, s, ax.LS); break;
        case 15: stage<15, C>(a, b, total, s, ax.LS); break;
        case 16: stage<16, C>(a, b, total, s, ax.LS); break;
        case 17: stage<17, C>(a, b, total, s, ax.LS); break;
        case 19: stage<19, C>(a, b, total, s, ax.LS); break;
        case 23: stage<23, C>(a, b, total, s, ax.LS); break;
        case 29: stage<29, C>(a, b, total, s, ax.LS); break;
        case 31: stage<31, C>(a, b, total, s, ax.LS); break;
        }
        __syncthreads();
        const int t = a;
        a = b;
        b = t;
    }
    return a;
}

template <typename C>
__device__ __forceinline__ C swp(C a) { return cmk<C>(a.y, a.x); }

// ------------------------------------------------------------------ x passes
// A CTA owns `rows` (a power of two) consecutive rows r = z ny + y of all
// three components: 3 rows/2 complex lines, line comp R2 + p holding rows
// 2p and 2p + 1 as real and imaginary parts.
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

// SPEC rows -> Hermitian lines, parts swapped for the inverse transform
template <typename C>
__device__ __forceinline__ void load_lines(const MxX& m, const RowCta& rc, const C* __restrict__ spec, int A)
{
    C* sm = reinterpret_cast<C*>(mx_sm);
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
                const int comp = rem >> m.r2sh, p = rem & (R2 - 1);
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
            // Z[k] = S_2p[k] + i S_2p+1[k], Z[Px - k] from the conjugates
            Z[pd<C>(kx)] = cmk<C>(a[u].y + b[u].x, a[u].x - b[u].y);
            if (kx > 0 && 2 * kx < m.ax.n) Z[pd<C>(m.ax.n - kx)] = cmk<C>(b[u].x - a[u].y, a[u].x + b[u].y);
        }
    }
}

// Transformed lines -> the two rows' spectra to SPEC
template <typename C>
__device__ __forceinline__ void store_spec(const MxX& m, const RowCta& rc, int Q, C* __restrict__ spec)
{
    typedef decltype(C().x) R;
    const C* sm = reinterpret_cast<const C*>(mx_sm);
    const int R2 = m.rows >> 1, n3 = 3 * R2, total = m.Kx * n3;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int kx = qdiv(idx, m.m3r2), l = idx - kx * n3;
        const int comp = l >> m.r2sh, p = l & (R2 - 1);
        const C* Z = sm + Q + l * m.ax.LS;
        const C zk = Z[pd<C>(kx)], zn = Z[pd<C>(kx ? m.ax.n - kx : 0)];
        C* dst = spec + ((size_t)kx * 3 + comp) * m.nr + rc.row0 + 2 * p;
        if (2 * p < rc.here) dst[0] = cmk<C>((R)0.5 * (zk.x + zn.x), (R)0.5 * (zk.y - zn.y));
        if (2 * p + 1 < rc.here) dst[1] = cmk<C>((R)0.5 * (zk.y + zn.y), (R)0.5 * (zn.x - zk.x));
    }
}

template <typename C>
__device__ __forceinline__ void load_twiddles(const MxAxis& ax, const C* __restrict__ tw)
{
    C* sm = reinterpret_cast<C*>(mx_sm);
    for (int k = threadIdx.x; k < ax.n; k += blockDim.x) sm[k] = tw[k];
}

} // namespace mx

// Forward x transform of the spins to SPEC.
template <typename R>
__global__ void __launch_bounds__(256, 2) k_mx_fx(const __grid_constant__ MxX m, const typename CT<R>::T* __restrict__ tw,
                                                  const R* __restrict__ sx, const R* __restrict__ sy,
                                                  const R* __restrict__ sz, typename CT<R>::T* __restrict__ spec)
{
    typedef typename CT<R>::T C;
    using namespace mx;
    load_twiddles<C>(m.ax, tw);
    pdl_trigger();
    pdl_wait();
    if (m.run_if && *m.run_if == 0) return;
    C* sm = reinterpret_cast<C*>(mx_sm);
    const RowCta rc = row_cta(m);
    const int R2 = m.rows >> 1, A = m.ax.n, B = A + 3 * R2 * m.ax.LS;
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
            reinterpret_cast<R*>(sm + A + (c * R2 + (row >> 1)) * m.ax.LS + pd<C>(x))[row & 1] = v[c];
    }
    __syncthreads();
    const int Q = fft<C>(A, B, 3 * R2, m.ax);
    store_spec<C>(m, rc, Q, spec);
}

// Inverse x transform of SPEC to the field.
template <typename R>
__global__ void __launch_bounds__(256, 2) k_mx_ix(const __grid_constant__ MxX m, const typename CT<R>::T* __restrict__ tw,
                                                  const typename CT<R>::T* __restrict__ spec, R* __restrict__ hx,
                                                  R* __restrict__ hy, R* __restrict__ hz)
{
    typedef typename CT<R>::T C;
    using namespace mx;
    load_twiddles<C>(m.ax, tw);
    pdl_trigger();
    pdl_wait();
    if (m.run_if && *m.run_if == 0) return;
    const C* sm = reinterpret_cast<const C*>(mx_sm);
    const RowCta rc = row_cta(m);
    const int R2 = m.rows >> 1, A = m.ax.n, B = A + 3 * R2 * m.ax.LS;
    load_lines<C>(m, rc, spec, A);
    __syncthreads();
    const int Q = fft<C>(A, B, 3 * R2, m.ax);
    const int total = rc.here * m.nx;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int row = qdiv(idx, m.mnx), x = idx - row * m.nx;
        const size_t i = (size_t)(rc.row0 + row) * m.nx + x;
        const R* z = reinterpret_cast<const R*>(sm + Q + (row >> 1) * m.ax.LS + pd<C>(x)) + ((row & 1) ^ 1);
        const int cs = 2 * R2 * m.ax.LS;
        hx[i] = z[0]; hy[i] = z[cs]; hz[i] = z[2 * cs];
    }
}

// ------------------------------------------------------------------ (y,z) pass
// One CTA per kx.  Layer sum of component a at column ky:
//   H_a[zt] = g sum_b sum_zs T_ab(zt - zs) M_b[zs],
// T_ab(dz) real and even in dz, or (exactly one of a, b is z) i times a real
// odd function.  tz: [kx][dz][6][ky].  One thread per (a, ky) keeps all NZ
// sums in registers (each spectrum value is read once per component, each
// tensor value once per thread); NZ = 0: one thread per (a, zt, ky).
template <typename R, int NZ>
__global__ void __launch_bounds__(512, 1) k_mx_yz(const __grid_constant__ MxYZ m, const typename CT<R>::T* __restrict__ tw,
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
    load_twiddles<C>(m.ax, tw);
    pdl_trigger();
    pdl_wait();
    if (m.run_if && *m.run_if == 0) return;
    C* sm = reinterpret_cast<C*>(mx_sm);
    const int A = Py, B = A + nl * LS;
    C* sp = spec + (size_t)kx * nl * ny;
    constexpr int U = 4;
    {
        const int total = nl * Py;
        for (int i0 = threadIdx.x; i0 < total; i0 += U * blockDim.x) {
            C v[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int idx = i0 + u * blockDim.x;
                const int l = qdiv(idx, m.mPy), y = idx - l * Py;
                v[u] = idx < total && y < ny ? sp[l * ny + y] : cmk<C>(0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int idx = i0 + u * blockDim.x;
                const int l = qdiv(idx, m.mPy), y = idx - l * Py;
                if (idx < total) sm[A + l * LS + pd<C>(y)] = v[u];
            }
        }
    }
    __syncthreads();
    const int P = fft<C>(A, B, nl, m.ax);
    const int Hb = P == A ? B : A;
    const R g = (R)m.g;
    if constexpr (NZ > 0) {
        for (int idx = threadIdx.x; idx < 3 * Py; idx += blockDim.x) {
            const int a = idx >= 2 * Py ? 2 : (idx >= Py ? 1 : 0), ky = idx - a * Py, kp = pd<C>(ky);
            C acc[NZ];
#pragma unroll
            for (int z = 0; z < NZ; z++) acc[z] = cmk<C>(0, 0);
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
                    const C v = sm[P + (b * NZ + zs) * LS + kp];
                    const C s = odd ? cmk<C>(-v.y, v.x) : v;
#pragma unroll
                    for (int zt = 0; zt < NZ; zt++) {
                        const R w = zt >= zs ? t[zt - zs] : tn[zs - zt];
                        acc[zt].x += w * s.x;
                        acc[zt].y += w * s.y;
                    }
                }
            }
#pragma unroll
            for (int z = 0; z < NZ; z++) sm[Hb + (a * NZ + z) * LS + kp] = cmk<C>(g * acc[z].y, g * acc[z].x);
        }
    } else {
        for (int idx = threadIdx.x; idx < nl * Py; idx += blockDim.x) {
            const int l = qdiv(idx, m.mPy), ky = idx - l * Py, kp = pd<C>(ky);
            const int a = l / nz, zt = l - a * nz;
            C acc = cmk<C>(0, 0);
            for (int b = 0; b < 3; b++) {
                const int lo = min(a, b), hi = max(a, b);
                const int q = lo == 0 ? hi : lo + hi + 1;
                const bool odd = (a == 2) != (b == 2);
                for (int zs = 0; zs < nz; zs++) {
                    const int dz = zt - zs;
                    R w = __ldg(T + (abs(dz) * 6 + q) * Py + ky);
                    if (odd && dz < 0) w = -w;
                    const C v = sm[P + (b * nz + zs) * LS + kp];
                    acc.x += w * (odd ? -v.y : v.x);
                    acc.y += w * (odd ? v.x : v.y);
                }
            }
            sm[Hb + l * LS + kp] = cmk<C>(g * acc.y, g * acc.x);
        }
    }
    __syncthreads();
    const int Q = fft<C>(Hb, P, nl, m.ax);
    for (int idx = threadIdx.x; idx < nl * ny; idx += blockDim.x) {
        const int l = qdiv(idx, m.mny), y = idx - l * ny;
        sp[idx] = swp(sm[Q + l * LS + pd<C>(y)]);
    }
}

// ------------------------------------------------------------------ tensor
// T(kx, ky, dz) of six components from their FP64 transforms over x and y,
// W[q][z][ky][kx] (z = dz mod Pz): tz[kx][dz][q][ky], the real part or (XZ,
// YZ) the imaginary part.  stat: bits of the largest |W| and of the largest
// deviation from the parities the layer sum relies on.
template <typename R>
__global__ void k_mx_pack(const double2* W, int Px, int Py, int Pz, int nz, int Kx, R* tz, unsigned long long* stat)
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
        tz[(((size_t)kx * nz + dz) * 6 + q) * Py + ky] = (R)(odd ? v.y : v.x);
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

// The stages of an axis of n points of which a CTA holds nl lines; false when
// n has a prime factor above 31.
static bool mx_axis(int n, int nl, bool f64, MxAxis& ax)
{
    std::vector<int> r;
    if (mx_best(n, nl * n, f64, r) >= 1e300 || (int)r.size() > MX_MAX_STAGES) return false;
    ax.n = n;
    ax.nst = (int)r.size();
    const int sh = f64 ? 3 : 4;
    ax.LS = n + (n >> sh) + 1;
    int Ns = 1;
    for (int i = 0; i < ax.nst; i++) {
        MxStage& s = ax.s[i];
        s.R = r[i];
        s.nb = n / r[i];
        s.Ns = Ns;
        s.tws = n / (Ns * r[i]);
        s.mnb = qmagic(s.nb);
        s.mNs = qmagic(Ns);
        Ns *= r[i];
    }
    return true;
}

static size_t mx_smem(const MxAxis& ax, int nl, int rb) { return ((size_t)ax.n + 2 * (size_t)nl * ax.LS) * 2 * rb; }

constexpr size_t MX_SMEM = 227 * 1024;

// Rows per CTA of the x passes: as few as keep the 148 SMs supplied (more
// rows make longer contiguous runs of SPEC), within shared memory.
bool mx_plan(const ConvK& c, int rb, MxPlan& p)
{
    if (c.general || c.nrep != 1 || c.nz > 32) return false;
    const bool f64 = rb == 8;
    memset(&p, 0, sizeof(p));
    const int nr = c.nz * c.ny;
    if ((long long)c.Px * c.Py > (1 << 22) || c.Px > 8192 || c.Py > 8192) return false;
    MxX& x = p.x;
    if (!mx_axis(c.Py, 3 * c.nz, f64, p.yz.ax) || mx_smem(p.yz.ax, 3 * c.nz, rb) > MX_SMEM) return false;
    int rows = 2;
    while (rows < 16 && (nr + 2 * rows - 1) / (2 * rows) >= 148) rows *= 2;
    for (;; rows /= 2) {
        if (rows < 2) return false;
        if (!mx_axis(c.Px, 3 * rows / 2, f64, x.ax)) return false;
        if (mx_smem(x.ax, 3 * rows / 2, rb) <= MX_SMEM / (rows > 2 ? 2 : 1)) break;
    }
    x.nx = c.nx; x.ny = c.ny; x.nz = c.nz; x.nr = nr; x.Kx = c.Kx;
    x.rows = rows;
    x.r2sh = rows == 2 ? 0 : (rows == 4 ? 1 : (rows == 8 ? 2 : 3));
    x.m3r2 = qmagic(3 * rows / 2);
    x.mPx = qmagic(c.Px);
    x.mnx = qmagic(c.nx);
    MxYZ& y = p.yz;
    y.ny = c.ny; y.nz = c.nz;
    y.mPy = qmagic(c.Py);
    y.mny = qmagic(c.ny);
    const int pts = 3 * c.nz * c.Py;
    y.threads = pts >= 4096 ? 512 : (pts >= 1024 ? 256 : 128);
    return true;
}

size_t mx_tensor_bytes(const ConvK& c, int rb) { return (size_t)c.Kx * c.nz * 6 * c.Py * rb; }

cudaError_t launch_mx_pack(const double2* W, const ConvK& c, void* tz, unsigned long long* stat2, int rb,
                           cudaStream_t st)
{
    const long long total = (long long)c.Kx * c.nz * 6 * c.Py;
    const unsigned nb = (unsigned)std::min<long long>((total + 255) / 256, 148 * 8);
    if (rb == 8)
        k_mx_pack<double><<<nb, 256, 0, st>>>(W, c.Px, c.Py, c.Pz, c.nz, c.Kx, static_cast<double*>(tz), stat2);
    else
        k_mx_pack<float><<<nb, 256, 0, st>>>(W, c.Px, c.Py, c.Pz, c.nz, c.Kx, static_cast<float*>(tz), stat2);
    return cudaGetLastError();
}

template <typename R>
static cudaError_t mx_fx(const MxX& x, const MxPlan& p, const typename CT<R>::T* tw, const void* const s[3],
                         typename CT<R>::T* spec, cudaStream_t st)
{
    Prof pf("k_conv_fx", st);
    return launch_pdl(k_mx_fx<R>, dim3((x.nr + x.rows - 1) / x.rows), dim3(256),
                      mx_smem(x.ax, 3 * x.rows / 2, sizeof(R)), st, x, tw, static_cast<const R*>(s[0]),
                      static_cast<const R*>(s[1]), static_cast<const R*>(s[2]), spec);
}

template <typename R>
static cudaError_t mx_ix(const MxX& x, const typename CT<R>::T* tw, const typename CT<R>::T* spec, void* const h[3],
                         cudaStream_t st)
{
    Prof pf("k_conv_ix", st);
    return launch_pdl(k_mx_ix<R>, dim3((x.nr + x.rows - 1) / x.rows), dim3(256),
                      mx_smem(x.ax, 3 * x.rows / 2, sizeof(R)), st, x, tw, spec, static_cast<R*>(h[0]),
                      static_cast<R*>(h[1]), static_cast<R*>(h[2]));
}

template <typename R>
static void (*yz_kernel(int nz))(MxYZ, const typename CT<R>::T*, typename CT<R>::T*, const R*)
{
    switch (nz) {
    case 1: return k_mx_yz<R, 1>;
    case 2: return k_mx_yz<R, 2>;
    case 3: return k_mx_yz<R, 3>;
    case 4: return k_mx_yz<R, 4>;
    case 5: return k_mx_yz<R, 5>;
    case 6: return k_mx_yz<R, 6>;
    case 7: return k_mx_yz<R, 7>;
    case 8: return k_mx_yz<R, 8>;
    }
    return k_mx_yz<R, 0>;
}

template <typename R>
static cudaError_t mx_yz(const ConvK& c, const MxYZ& y, const typename CT<R>::T* tw, typename CT<R>::T* spec,
                         const R* tz, cudaStream_t st)
{
    Prof pf("k_conv_yz", st);
    return launch_pdl(yz_kernel<R>(c.nz), dim3(c.Kx), dim3(y.threads), mx_smem(y.ax, 3 * c.nz, sizeof(R)), st, y, tw,
                      spec, tz);
}

template <typename R>
static cudaError_t mx_conv_t(const ConvK& c, const MxPlan& p, const FftLen L[3], const void* tw_, const void* const s[3],
                             void* spec_, const void* tz, void* const h[3], bool fx, bool ix, cudaStream_t st)
{
    typedef typename CT<R>::T C;
    const C* tw = static_cast<const C*>(tw_);
    C* spec = static_cast<C*>(spec_);
    MxX x = p.x;
    MxYZ y = p.yz;
    x.run_if = y.run_if = c.run_if;
    y.g = c.g;
    cudaError_t e = cudaSuccess;
    if (fx && (e = mx_fx<R>(x, p, tw + L[0].tw_off, s, spec, st)) != cudaSuccess) return e;
    if ((e = mx_yz<R>(c, y, tw + L[1].tw_off, spec, static_cast<const R*>(tz), st)) != cudaSuccess) return e;
    if (ix) e = mx_ix<R>(x, tw + L[0].tw_off, spec, h, st);
    return e;
}

cudaError_t launch_mx_conv(const ConvK& c, const MxPlan& p, const FftLen L[3], const void* tw, const void* const s[3],
                           void* spec, const void* tz, void* const h[3], bool fx, bool ix, int rb, cudaStream_t st)
{
    if (rb == 8) return mx_conv_t<double>(c, p, L, tw, s, spec, tz, h, fx, ix, st);
    return mx_conv_t<float>(c, p, L, tw, s, spec, tz, h, fx, ix, st);
}

template <typename K>
static cudaError_t mx_max_smem(K kern)
{
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MX_SMEM);
}

template <typename R>
static cudaError_t mx_configure_t()
{
    cudaError_t e;
    if ((e = mx_max_smem(k_mx_fx<R>)) != cudaSuccess || (e = mx_max_smem(k_mx_ix<R>)) != cudaSuccess) return e;
    for (int nz = 0; nz <= 8; nz++)
        if ((e = mx_max_smem(yz_kernel<R>(nz))) != cudaSuccess) return e;
    return cudaSuccess;
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
    if ((e = mx_configure_t<float>()) != cudaSuccess) return e;
    return mx_configure_t<double>();
}

} // namespace mlb
