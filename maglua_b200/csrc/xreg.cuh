// xreg.cuh -- FP32 x lines of 32 to 256 points in shared memory, transformed in
// registers (conv_fast.cu, xstep.cuh).
#pragma once
#include "device.cuh"
#include "fftreg.cuh"

// FP32 x lines of 32 to 256 points: the four-step register FFT of
// fr::line_fft (Split<N>::T lanes x Split<N>::E points, one warp-synchronous
// exchange through ex, E (T + 1) elements per line), in place on a
// natural-order line: the lanes have read the whole line before any of them
// writes it back; SELF: the line's own buffer serves for the exchange.
template <int N>
struct XReg {
    static constexpr bool OK = N >= 32 && N <= 256;
    static constexpr int T = fr::Split<N>::T, E = fr::Split<N>::E, EX = E * (T + 1);
};
// HZ: the data end before N / 2; the zeros behind them are not read (SIGN < 0)
// or what would be written there is left out (SIGN > 0).
template <int N, int SIGN, bool SELF = false, bool HZ = false>
__device__ __forceinline__ void xreg_line(float2* line, float2* ex, int t, unsigned mask, const float2* tw)
{
    constexpr int T = XReg<N>::T, E = XReg<N>::E;
    constexpr bool HI = HZ && SIGN < 0, HO = HZ && SIGN > 0;
    float2 v[E];
#pragma unroll
    for (int j = 0; j < (HI ? E / 2 : E); j++) v[j] = line[t + T * j];
    if (SELF) __syncwarp(mask);
    fr::line_fft<N, SIGN, float2, HI>(v, SELF ? line : ex, t, mask, tw);
#pragma unroll
    for (int r = 0; r < E; r++)
        if (!HO || E * (r % T) < N / 2) line[fr::out_index<N>(t, r)] = v[r];
}

// The CTA's nl lines (line l at base + l ls) in place, line l by threads
// T l .. T l + T - 1.  Every thread of the CTA calls this; the CTA is
// synchronised after the transforms.
// ex: exchange buffers of XReg<N>::EX elements per line; SELF: the lines
// themselves (ls >= XReg<N>::EX).
template <int N, int SIGN, bool SELF = false, bool HZ = false>
__device__ __forceinline__ void xreg_lines(float2* base, int ls, int nl, float2* ex, const float2* tw)
{
    constexpr int T = XReg<N>::T;
    const int l = threadIdx.x / T, t = threadIdx.x % T;
    if (l < nl) {
        const unsigned mask = ((1u << T) - 1u) << ((threadIdx.x & 31) & ~(T - 1));
        float2* ln = base + (size_t)l * ls;
        xreg_line<N, SIGN, SELF, HZ>(ln, SELF ? nullptr : ex + (size_t)l * XReg<N>::EX, t, mask, tw);
    }
    __syncthreads();
}
