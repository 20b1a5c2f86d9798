// yzls.cuh -- (y,z) pass of the dipole convolution with the sum over layers,
// power-of-two Py 16..512, up to 8 layers (to 64 rows up to 16), FP32 and FP64.
//
// One CTA per kx (and packed replica).  A line (component, layer) of Py = T E
// points belongs to T lanes of a warp:
//   1. lane t loads x[t + T j], transforms its E points in registers,
//      multiplies by w^{t k1} and stores row k1 of the line's [E][T + 1] buffer
//      at column t;
//   2. the lane that owns row k1 transforms its T values in place: place
//      (k1, k2) then holds frequency ky = k1 + E k2.
// The spectrum is not put in order: the layer tensor is stored by place.
//   3. the sum over source layers with T(kx, ky, dz) (see mx.cu: nz^2 real
//      multiplies per component pair instead of zero-padded transforms in z);
//      a thread keeps all target layers of one (component, place), so a
//      spectrum value is read once per component and a tensor value once;
//   4. the transforms of 2 and 1 backwards, data rows to SPEC.
// A plane is 3 nz lines of E (T + 1) values, with no second buffer: 52 KB for
// 256 x 8 where z spectra of 16 rows took 152 KB, so CTAs of several replicas or
// streams share an SM, and the CTA synchronises three times.
//
// Bound by one CTA's chain on single films (129 CTAs for 256 columns), by issue
// on packed replicas.  Measured against the passes with z spectra: 256x256x8
// 9.5 -> 8 us within a step of 30.2 -> 28.7, 512x512x4 step alone 71.9 -> 67.1,
// 64x64x8 12.6 -> 10.3, 16x256x4 20.7 -> 10.5, FP64 128x128x4 24.0 -> 18.3; the
// four (y,z) passes of 512 replicas 275 -> 189 us.
// One translation unit per state precision (yzls_f32.cu, yzls_f64.cu); yzls.cu chooses.
#pragma once
#include "device.cuh"
#include "fftreg.cuh"
#include "kparams.h"
#include "launch.h"

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace {

// Threads: one per (component, place) as far as the registers allow, for a
// lattice whose CTAs have an SM each; or (SM) PY or so, three items each, when
// many CTAs share an SM (packed replicas) or few layers leave the others idle.
template <int PY, typename C, bool SM>
struct LS {
    static constexpr int T = fr::Split<PY>::T, E = fr::Split<PY>::E;
    // registers: 80 per thread at 768 (512-point lines hold 32 points per lane)
    static constexpr int MAXT = sizeof(C) == 8 ? (PY == 512 ? 512 : 768) : 384;
    static constexpr int NT = SM ? (PY <= 64 ? 96 : PY) : (3 * PY < MAXT ? (3 * PY < 64 ? 64 : 3 * PY) : MAXT);
    static constexpr int MINB = SM && PY <= 128 ? 65536 / (NT * 88) : 1;
    static constexpr int NI = (3 * PY + NT - 1) / NT;   // (component, place) items per thread
    static constexpr int LINE = E * (T + 1);
    static constexpr int LPR = NT / T;                  // lines per round
    static size_t smem(int nz) { return ((size_t)PY + (size_t)3 * nz * LINE) * sizeof(C); }
};

// acc += w s for a real w: one packed multiply-add in FP32
__device__ __forceinline__ void axpy(float2& acc, float w, float2 s)
{
    unsigned long long a, b, c;
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(acc.x), "f"(acc.y));
    asm("mov.b64 %0, {%1, %1};" : "=l"(b) : "f"(w));
    asm("mov.b64 %0, {%1, %2};" : "=l"(c) : "f"(s.x), "f"(s.y));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(b), "l"(c));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(acc.x), "=f"(acc.y) : "l"(a));
}
__device__ __forceinline__ void axpy(double2& acc, double w, double2 s)
{
    acc.x = fm(w, s.x, acc.x);
    acc.y = fm(w, s.y, acc.y);
}

// NZ layers, or (UP) c.nz of them, up to NZ.
template <int PY, int NZ, typename C, bool SM, bool UP = false>
__global__ void __launch_bounds__(LS<PY, C, SM>::NT, LS<PY, C, SM>::MINB) k_yz_ls(ConvK c, const C* __restrict__ twy, C* __restrict__ spec,
                                                          const decltype(C().x)* __restrict__ tz)
{
    typedef decltype(C().x) R;
    using Y = LS<PY, C, SM>;
    constexpr int NT = Y::NT, T = Y::T, E = Y::E, LINE = Y::LINE, NI = Y::NI;
    extern __shared__ __align__(16) unsigned char smraw_ls[];
    C* twl = reinterpret_cast<C*>(smraw_ls);   // [PY]
    C* P = twl + PY;                           // [3 NZ][E][T + 1]
    const int kx = blockIdx.x, ny = c.ny, nz = UP ? c.nz : NZ, nl = 3 * nz;
    const R* Tk = tz + (size_t)kx * nz * 6 * PY;
    if (threadIdx.x == 0) {
        // this kx's tensor (constant between steps) starts towards L2
        const unsigned bytes = (unsigned)(nz * 6 * PY * sizeof(R));
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(Tk), "r"(bytes) : "memory");
    }
    for (int k = threadIdx.x; k < PY; k += NT) twl[k] = twy[k];
    pdl_trigger();
    pdl_wait();
    tl_start(c.tl);
    if (c.run_if && *c.run_if == 0) return;
    C* sp = spec + ((size_t)blockIdx.y * c.Kx + kx) * nl * ny;
    __syncthreads();
    const int lr = threadIdx.x / T, t = threadIdx.x % T;
    const unsigned mask = ((1u << T) - 1u) << (((threadIdx.x & 31) / T) * T);
    for (int l = lr; l < nl && lr < Y::LPR; l += Y::LPR) {   // whole T-lane groups share l
        C* ln = P + l * LINE;
        C v[E];
#pragma unroll
        for (int j = 0; j < E; j++) {
            const int y = t + T * j;
            v[j] = y < ny ? sp[l * ny + y] : cmk<C>(0, 0);
        }
        fr::RegFFT<E, -1, C>::run(v);
#pragma unroll
        for (int k1 = 0; k1 < E; k1++) {
            if (T > 1 && k1 > 0) v[k1] = cmul(v[k1], twl[(t * k1) & (PY - 1)]);
            ln[k1 * (T + 1) + t] = v[k1];
        }
        __syncwarp(mask);
#pragma unroll
        for (int q = 0; q < E / T; q++) {
            C* row = ln + (t + q * T) * (T + 1);
            C u[T];
#pragma unroll
            for (int s = 0; s < T; s++) u[s] = row[s];
            fr::RegFFT<T, -1, C>::run(u);
#pragma unroll
            for (int s = 0; s < T; s++) row[s] = u[s];
        }
    }
    __syncthreads();
    const R g = (R)c.g;
    C acc[NI][NZ];
#pragma unroll
    for (int i = 0; i < NI; i++) {
        const int item = threadIdx.x + i * NT;
        const int a = item / PY, p = item % PY;   // component, place
#pragma unroll
        for (int z = 0; z < NZ; z++) acc[i][z] = cmk<C>(0, 0);
        if (item >= 3 * PY) continue;
        const C* col = P + p + p / T;
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const int q = a == 0 ? b : (b == 0 ? a : a + b + 1);   // XX XY XZ YY YZ ZZ
            // XZ, YZ: imaginary and odd in dz
            const bool odd = (a == 2) != (b == 2);
            R w[NZ], wn[NZ];
#pragma unroll
            for (int d = 0; d < NZ; d++) {
                w[d] = !UP || d < nz ? __ldg(Tk + (d * 6 + q) * PY + p) : (R)0;
                wn[d] = odd ? -w[d] : w[d];
            }
#pragma unroll
            for (int zs = 0; zs < NZ; zs++) {
                if (UP && zs >= nz) break;
                const C m = col[(b * nz + zs) * LINE];
                const C s = odd ? cmk<C>(-m.y, m.x) : m;
#pragma unroll
                for (int zt = 0; zt < NZ; zt++) axpy(acc[i][zt], zt >= zs ? w[zt - zs] : wn[zs - zt], s);
            }
        }
    }
    __syncthreads();   // every spectrum value has been read
#pragma unroll
    for (int i = 0; i < NI; i++) {
        const int item = threadIdx.x + i * NT;
        const int a = item / PY, p = item % PY;
        if (item >= 3 * PY) continue;
#pragma unroll
        for (int z = 0; z < NZ; z++)
            if (!UP || z < nz) P[(a * nz + z) * LINE + p + p / T] = cmk<C>(g * acc[i][z].x, g * acc[i][z].y);
    }
    __syncthreads();
    for (int l = lr; l < nl && lr < Y::LPR; l += Y::LPR) {
        C* ln = P + l * LINE;
#pragma unroll
        for (int q = 0; q < E / T; q++) {
            const int k1 = t + q * T;
            C* row = ln + k1 * (T + 1);
            C u[T];
#pragma unroll
            for (int s = 0; s < T; s++) u[s] = row[s];
            fr::RegFFT<T, +1, C>::run(u);
#pragma unroll
            for (int s = 0; s < T; s++) {
                if (s > 0) u[s] = cmul(u[s], cconj(twl[(s * k1) & (PY - 1)]));
                row[s] = u[s];
            }
        }
        __syncwarp(mask);
        C v[E];
#pragma unroll
        for (int k1 = 0; k1 < E; k1++) v[k1] = ln[k1 * (T + 1) + t];
        fr::RegFFT<E, +1, C>::run(v);
#pragma unroll
        for (int j = 0; j < E; j++) {
            const int y = t + T * j;
            if (y < ny) sp[l * ny + y] = v[j];
        }
    }
    tl_end(c.tl);
}

template <typename C> using Kern = void (*)(ConvK, const C*, C*, const decltype(C().x)*);

// Up to 8 layers in planes of any width, 9 to 16 in planes of up to 64 rows: one kernel
// for 16, and one that leaves out what is missing to 16 (64x64x12 11.3 us a step where
// the z spectra took 14.9, 256x64x9 16.9 against 20.0, FP64 64x64x12 17.6 against
// 48.7; all 16 by it 12.8 against 11.9).  Wider planes keep the z spectra: the kernel
// would serve 128 and 256 rows too (64x128x9 24.8 -> 13.4, 256x256x16 54.6 -> 44.1), but
// its small-CTA form does not fit the registers there (4.7 KB spilled), and at 512
// rows it is slower (64x512x16 41 -> 48).
template <int PY, typename C, bool SM>
Kern<C> kern_py(int nz)
{
    switch (nz) {
    case 1: return k_yz_ls<PY, 1, C, SM>;
    case 2: return k_yz_ls<PY, 2, C, SM>;
    case 3: return k_yz_ls<PY, 3, C, SM>;
    case 4: return k_yz_ls<PY, 4, C, SM>;
    case 5: return k_yz_ls<PY, 5, C, SM>;
    case 6: return k_yz_ls<PY, 6, C, SM>;
    case 7: return k_yz_ls<PY, 7, C, SM>;
    case 8: return k_yz_ls<PY, 8, C, SM>;
    }
    if constexpr (PY <= 64)
        if (nz <= 16) return nz == 16 ? k_yz_ls<PY, 16, C, SM> : k_yz_ls<PY, 16, C, SM, true>;
    return nullptr;
}

template <typename C>
struct Sel {
    Kern<C> k = nullptr;
    int nt = 0;
    size_t smem = 0;
};
template <int PY, typename C>
Sel<C> sel_py(int nz, bool small)
{
    Sel<C> s;
    if constexpr (sizeof(C) == 8) {
        if (small) {
            s.k = kern_py<PY, C, true>(nz);
            s.nt = LS<PY, C, true>::NT;
            s.smem = LS<PY, C, true>::smem(nz);
            return s;
        }
    }
    s.k = kern_py<PY, C, false>(nz);
    s.nt = LS<PY, C, false>::NT;
    s.smem = LS<PY, C, false>::smem(nz);
    return s;
}
template <typename C>
Sel<C> sel(int Py, int nz, bool small)
{
    switch (Py) {
    case 16: return sel_py<16, C>(nz, small);
    case 32: return sel_py<32, C>(nz, small);
    case 64: return sel_py<64, C>(nz, small);
    case 128: return sel_py<128, C>(nz, small);
    case 256: return sel_py<256, C>(nz, small);
    case 512: return sel_py<512, C>(nz, small);
    }
    return Sel<C>();
}

} // namespace

namespace mlb {

constexpr size_t LS_SMEM = 227 * 1024;

template <typename C>
cudaError_t YzUnit<C>::init()
{
    return fr::fill_tables();
}
template <typename C>
bool YzUnit<C>::takes(int Py, int nz)
{
    const auto s = sel<C>(Py, nz, false);
    return s.k && s.smem <= LS_SMEM;
}
template <typename C>
cudaError_t YzUnit<C>::pass(const ConvK& c, const C* tw, C* spec, const R* tz, cudaStream_t st)
{
    bool small = false;
    if constexpr (sizeof(C) == 8) {
        // small CTAs where there are more of them than SMs (a step of 512x64x4 alone
        // 18.8 us against 31.7; 512 replicas 387 against 595) or where the lines
        // occupy little more than half of one (128x128x1 10.5 against 11.5); large ones for
        // the others (128x128x8 17.2 against 19.2)
        const int T = c.Py >= 256 ? 16 : (c.Py >= 64 ? 8 : 4), ns = sel<C>(c.Py, c.nz, true).nt;
        small = (long long)c.Kx * c.nrep > 148 || 5 * 3 * c.nz * T <= 3 * ns;
    }
    const auto s = sel<C>(c.Py, c.nz, small);
    return launch_pdl(s.k, dim3(c.Kx, c.nrep), dim3(s.nt), s.smem, st, c, tw, spec, tz);
}

} // namespace mlb
