// mx.cuh -- the kernels of mx.cu, one translation unit per state precision and with or
// without prime radices above 13 (mx_f32.cu, mx_f32_big.cu and so on), which compile
// side by side.
#pragma once
#include "device.cuh"
#include "fused.cuh"
#include "kparams.h"
#include "launch.h"
#include "mxradix.h"
#include "terms.cuh"

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

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

// ------------------------------------------------------------------ launches
namespace mlb {

template <typename R, bool BIG>
cudaError_t MxUnit<R, BIG>::init()
{
    static float2 hf[mx::NW];
    static double2 hd[mx::NW];
    for (int r = 1; r <= mx::MAXR; r++)
        for (int k = 0; k < r; k++) {
            const double a = 2.0 * M_PI * k / r;
            hd[r * (r - 1) / 2 + k] = make_double2(cos(a), -sin(a));
            hf[r * (r - 1) / 2 + k] = make_float2((float)cos(a), (float)-sin(a));
        }
    cudaError_t e;
    if ((e = cudaMemcpyToSymbol(mx::c_wf, hf, sizeof(hf))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(mx::c_wd, hd, sizeof(hd))) != cudaSuccess) return e;
    return cudaStreamSynchronize(nullptr);   // there for every stream
}

static dim3 mx_grid(const MxX& x) { return dim3((x.nr + x.rows - 1) / x.rows); }

template <typename R, bool BIG>
cudaError_t MxUnit<R, BIG>::fx(const MxX& x, size_t smem, const C* tw, const void* const s[3], C* spec, cudaStream_t st)
{
    return launch_pdl(k_mx_fx<R, BIG>, mx_grid(x), dim3(256), smem, st, x, tw, static_cast<const R*>(s[0]),
                      static_cast<const R*>(s[1]), static_cast<const R*>(s[2]), spec);
}

template <typename R, bool BIG>
cudaError_t MxUnit<R, BIG>::ix(const MxX& x, size_t smem, const C* tw, const C* spec, void* const h[3], cudaStream_t st)
{
    return launch_pdl(k_mx_ix<R, BIG>, mx_grid(x), dim3(256), smem, st, x, tw, spec, static_cast<R*>(h[0]),
                      static_cast<R*>(h[1]), static_cast<R*>(h[2]));
}

template <typename R, bool BIG>
cudaError_t MxUnit<R, BIG>::yz(const MxYZ& y, int Kx, size_t smem, const C* tw, C* spec, const R* tz, cudaStream_t st)
{
    void (*k)(MxYZ, const C*, C*, const R*) = k_mx_yz<R, 0, BIG>;
    switch (y.nz) {
    case 1: k = k_mx_yz<R, 1, BIG>; break;
    case 2: k = k_mx_yz<R, 2, BIG>; break;
    case 3: k = k_mx_yz<R, 3, BIG>; break;
    case 4: k = k_mx_yz<R, 4, BIG>; break;
    case 5: k = k_mx_yz<R, 5, BIG>; break;
    case 6: k = k_mx_yz<R, 6, BIG>; break;
    case 7: k = k_mx_yz<R, 7, BIG>; break;
    case 8: k = k_mx_yz<R, 8, BIG>; break;
    }
    return launch_pdl(k, dim3(Kx), dim3(y.threads), smem, st, y, tw, spec, tz);
}

template <typename R, bool BIG>
cudaError_t MxUnit<R, BIG>::lr2d(const MxYZ& y, int Kx, size_t smem, const LR2DScale& sc, int stream, const C* tw, C* spec,
                                 const C* Q, cudaStream_t st)
{
    return launch_pdl(k_mx_lr2d<R, BIG>, dim3(Kx), dim3(y.threads), smem, st, y, sc, stream, tw, spec, Q);
}

template <typename R, bool BIG>
cudaError_t MxUnit<R, BIG>::step(const MxX& x, size_t smem, const C* tw, C* spec, const FastKT<R>& F, const R* const s[3],
                                 R* const h[3], R* const o[3], cudaStream_t st)
{
    void (*k)(MxX, FastKT<R>, const C*, C*, const R*, const R*, const R*, R*, R*, R*, R*, R*, R*);
    if (F.llg_type == LLG_CART) {
        if (F.ani) k = F.th ? k_mx_step<R, LLG_CART, true, true, BIG> : k_mx_step<R, LLG_CART, true, false, BIG>;
        else k = F.th ? k_mx_step<R, LLG_CART, false, true, BIG> : k_mx_step<R, LLG_CART, false, false, BIG>;
    } else {
        if (F.ani) k = F.th ? k_mx_step<R, LLG_QUAT, true, true, BIG> : k_mx_step<R, LLG_QUAT, true, false, BIG>;
        else k = F.th ? k_mx_step<R, LLG_QUAT, false, true, BIG> : k_mx_step<R, LLG_QUAT, false, false, BIG>;
    }
    return launch_pdl(k, mx_grid(x), dim3(256), smem, st, x, F, tw, spec, s[0], s[1], s[2], h[0], h[1], h[2], o[0], o[1],
                      o[2]);
}

template <typename R, bool BIG>
cudaError_t MxUnit<R, BIG>::rk(const MxX& x, size_t smem, const C* tw, C* spec, const FastKT<R>& F, const RkRows<R>& rows,
                               const R* const s[3], R* const h[3], R* const o[3], cudaStream_t st)
{
    void (*k)(MxX, FastKT<R>, RkRows<R>, const C*, C*, const R*, const R*, const R*, R*, R*, R*, R*, R*, R*);
    if (F.llg_type == LLG_CART) k = F.ani ? k_mx_rk<R, LLG_CART, true, BIG> : k_mx_rk<R, LLG_CART, false, BIG>;
    else k = F.ani ? k_mx_rk<R, LLG_QUAT, true, BIG> : k_mx_rk<R, LLG_QUAT, false, BIG>;
    return launch_pdl(k, mx_grid(x), dim3(256), smem, st, x, F, rows, tw, spec, s[0], s[1], s[2], h[0], h[1], h[2], o[0],
                      o[1], o[2]);
}

template <typename R, bool BIG>
cudaError_t MxUnit<R, BIG>::gstep(const MxX& x, size_t smem, const C* tw, C* spec, const FusedK& P, double addw,
                                  double dt_sys, const DevStep* cur, DevStep* next, void* const h[3], cudaStream_t st)
{
    return launch_pdl(k_mx_gstep<R, BIG>, mx_grid(x), dim3(256), smem, st, x, P, addw, dt_sys, cur, next, tw, spec,
                      static_cast<R*>(h[0]), static_cast<R*>(h[1]), static_cast<R*>(h[2]));
}

} // namespace mlb
