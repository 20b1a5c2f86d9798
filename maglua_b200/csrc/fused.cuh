// fused.cuh -- one site of the fused step (field terms + LLG update) for
// uniform-parameter systems, FP32 or FP64, or two FP32 sites in packed arithmetic;
// shared by the fused-step kernels (conv_fast.cu), the fused x passes (xstep.cuh,
// mx.cuh) and the Runge-Kutta stages there.
#pragma once
#include "device.cuh"
#include "kparams.h"

#include <math.h>
#include <stdint.h>

// The step block's per-step values (swept field, thermal counter) read once
// per thread instead of once per site: the same values, so the same results.
template <typename R>
__device__ __forceinline__ FastKT<R> fastk_resolved(const FastKT<R>& F)
{
    FastKT<R> G = F;
    if (F.Bdev) {
        G.B[0] = (R)F.Bdev[0]; G.B[1] = (R)F.Bdev[1]; G.B[2] = (R)F.Bdev[2];
        G.Bdev = nullptr;
    }
    if (F.dctr) {
        G.counter = F.counter + *F.dctr;
        G.dctr = nullptr;
    }
    return G;
}

// Cubic anisotropy field of one axis set at the reduced moment (sx, sy, sz)
// = S / ms (M/cpu/anisotropy/..._cubic.cpp:308-390): axes n[0..2], n[3..5],
// n[6..8], constants K[0..2]; quirk keeps (n2s2 + n3s3) in the first K1 term.
// V: R, or p2 (two sites).
template <typename R, typename V = R>
__device__ __forceinline__ void cubic_field(V sx, V sy, V sz, const R* n, const R* K, int quirk, V& hx, V& hy, V& hz)
{
    const auto B = [](R a) { return bc<V, R>(a); };
    const V n1s = dot3(B(n[0]), sx, B(n[1]), sy, B(n[2]), sz);
    const V n2s = dot3(B(n[3]), sx, B(n[4]), sy, B(n[5]), sz);
    const V n3s = dot3(B(n[6]), sx, B(n[7]), sy, B(n[8]), sz);
    const V n1s2 = ml(n1s, n1s), n2s2 = ml(n2s, n2s), n3s2 = ml(n3s, n3s);
    const V n1s3 = ml(n1s2, n1s), n2s3 = ml(n2s2, n2s), n3s3 = ml(n3s2, n3s);
    const V n3s4 = ml(n3s2, n3s2), n2s4 = ml(n2s2, n2s2);
    const V q = quirk ? n3s3 : n3s2;
    const V k1 = B(ml((R)2, K[0])), k2 = B(ml((R)2, K[1])), k3 = B(ml((R)4, K[2]));
    const V p = ml(k2, ml(ml(n1s, n2s), n3s));
    // every sum a fused multiply-add of its own (the packed forms are
    // contracted otherwise)
    const V c1 = ml(ml(k3, n1s3), fm(n2s2, n2s2, n3s4)), c2 = ml(ml(k3, n2s3), fm(n1s2, n1s2, n3s4)),
            c3 = ml(ml(k3, n3s3), fm(n1s2, n1s2, n2s4));
    const V s1 = fm(ml(k1, n1s), fm(n2s, n2s, q), fm(p, ml(n2s, n3s), c1));
    const V s2 = fm(ml(k1, n2s), fm(n1s, n1s, n3s2), fm(p, ml(n1s, n3s), c2));
    const V s3 = fm(ml(k1, n3s), fm(n1s, n1s, n2s2), fm(p, ml(n1s, n2s), c3));
    hx = dot3(B(n[0]), s1, B(n[3]), s2, B(n[6]), s3);
    hy = dot3(B(n[1]), s1, B(n[4]), s2, B(n[7]), s3);
    hz = dot3(B(n[2]), s1, B(n[5]), s2, B(n[8]), s3);
}

// ------------------------------------------------------------------ fused step
// Uniform-parameter systems: ms, alpha, gamma, anisotropy and thermal scale
// the same on every site, exchange as a six-direction stencil.  Constants
// are folded on the host (FastK).
// One site of the fused step.  (x, y, z) are the site's coordinates inside
// its lattice of NX x NY x NZ sites and i its index in the (packed) arrays;
// neighbours are addressed relative to i, so several lattices can share the
// arrays back to back.
// The new spin of the site is returned in (rx, ry, rz); (Ax, Ay, Az) is the
// materialised addend (the dipole slot), used when ADD.
// reciprocal square root and sine/cosine in the state precision
__device__ __forceinline__ float fs_rsqrt(float v) { return rsqrtf(v); }
__device__ __forceinline__ double fs_rsqrt(double v) { return rsqrt(v); }

// The spins come through ld(c, j) (component c of site j): global loads, or
// shared-memory copies of some rows (the fused x pass).
template <typename R>
struct GlobalSpins {
    const R* __restrict__ s[3];
    __device__ __forceinline__ R operator()(int c, int j) const { return __ldg(s[c] + j); }
};

// The thermal site's three standard normals are those of thermal_normal3();
// a caller that drew them earlier passes them in pre (else nullptr).
template <typename R>
__device__ __forceinline__ float3 thermal_normal3(const FastKT<R>& F, int i)
{
    const uint64_t ctr = F.counter + (F.dctr ? *F.dctr : 0ull);
    return philox_normal3(F.seed, ctr, (uint32_t)i, 0x6d6c6232u);
}

// sine and cosine of the half rotation angle; in FP32 small angles by their
// Taylor series (|th| <= 0.1: truncation below 1e-10, under FP32 rounding),
// else (and always in FP64) sine and cosine
template <typename V>
__device__ __forceinline__ void taylor_sincos(V th, V& sn, V& cs)
{
    const auto B = [](float a) { return bc<V, float>(a); };
    const V t2 = ml(th, th), n2 = -t2, one = B(1.f);
    const V a = fm(n2, B(1.0f / 42.0f), one), b = fm(ml(n2, B(1.0f / 20.0f)), a, one);
    sn = ml(th, fm(ml(n2, B(1.0f / 6.0f)), b, one));
    const V c = fm(n2, B(1.0f / 56.0f), one), d = fm(ml(n2, B(1.0f / 30.0f)), c, one);
    const V e = fm(ml(n2, B(1.0f / 12.0f)), d, one);
    cs = fm(ml(n2, B(0.5f)), e, one);
}
__device__ __forceinline__ void half_sincos(float th, float& sn, float& cs)
{
    if (fabsf(th) <= 0.1f) taylor_sincos<float>(th, sn, cs);
    else sincosf(th, &sn, &cs);
}
__device__ __forceinline__ void half_sincos(double th, double& sn, double& cs) { sincos(th, &sn, &cs); }
__device__ __forceinline__ void half_sincos(p2 th, p2& sn, p2& cs)
{
    const float2 t = up(th);
    if (fmaxf(fabsf(t.x), fabsf(t.y)) <= 0.1f) {
        taylor_sincos<p2>(th, sn, cs);
    } else {
        float s0, c0, s1, c1;
        half_sincos(t.x, s0, c0);
        half_sincos(t.y, s1, c1);
        sn = pk(s0, s1);
        cs = pk(c0, c1);
    }
}
__device__ __forceinline__ p2 fs_rsqrt(p2 v)
{
    const float2 u = up(v);
    return pk(rsqrtf(u.x), rsqrtf(u.y));
}
// lanes of a where the lane of m is positive (not zero), else of b
__device__ __forceinline__ float where_pos(float m, float a, float b) { return m > 0.f ? a : b; }
__device__ __forceinline__ double where_pos(double m, double a, double b) { return m > 0.0 ? a : b; }
__device__ __forceinline__ p2 where_pos(p2 m, p2 a, p2 b)
{
    const float2 u = up(m), x = up(a), y = up(b);
    return pk(u.x > 0.f ? x.x : y.x, u.y > 0.f ? x.y : y.y);
}
__device__ __forceinline__ float where_nz(float m, float a, float b) { return m != 0.f ? a : b; }
__device__ __forceinline__ double where_nz(double m, double a, double b) { return m != 0.0 ? a : b; }
__device__ __forceinline__ p2 where_nz(p2 m, p2 a, p2 b)
{
    const float2 u = up(m), x = up(a), y = up(b);
    return pk(u.x != 0.f ? x.x : y.x, u.y != 0.f ? x.y : y.y);
}
// 0 in every lane? (x 0 is 0 for a finite x, else not a number)
__device__ __forceinline__ bool all_zero(float a) { return a == 0.f; }
__device__ __forceinline__ bool all_zero(double a) { return a == 0.0; }
__device__ __forceinline__ bool all_zero(p2 a)
{
    const float2 u = up(a);
    return u.x == 0.f && u.y == 0.f;
}

// Adds to the Zeeman and exchange fields H of a spin S its anisotropy, the addend
// A and the thermal field (nrm: its standard normals); g: the field the terms
// without the thermal part see.  V: R for one site, p2 for two, each lane the
// same operations.
template <bool ANI, bool TH, bool ADD, typename R, typename V>
__device__ __forceinline__ void fused_field(const FastKT<R>& F, V Sx, V Sy, V Sz, V& Hx, V& Hy, V& Hz, V nrmx, V nrmy,
                                            V nrmz, V Ax, V Ay, V Az, V& gx, V& gy, V& gz)
{
    const auto B = [](R a) { return bc<V, R>(a); };
    if (ANI) {
        if (F.ani == 2) {
            // one uniform cubic axis set
            V cx, cy, cz;
            const V im = B(F.cub_ims);
            cubic_field<R, V>(ml(Sx, im), ml(Sy, im), ml(Sz, im), F.cub_n, F.cub_K, F.cub_quirk, cx, cy, cz);
            Hx = ad(Hx, cx); Hy = ad(Hy, cy); Hz = ad(Hz, cz);
        } else {
            const V ax = B(F.axis[0]), ay = B(F.axis[1]), az = B(F.axis[2]);
            const V v = ml(B(F.ani_c), dot3(Sx, ax, Sy, ay, Sz, az));
            Hx = fm(v, ax, Hx); Hy = fm(v, ay, Hy); Hz = fm(v, az, Hz);
        }
    }
    if (ADD) {
        const V w = B(F.addw);
        Hx = fm(w, Ax, Hx); Hy = fm(w, Ay, Hy); Hz = fm(w, Az, Hz);
    }
    gx = Hx; gy = Hy; gz = Hz;
    if (TH) {
        const V sg = B(F.sigma);
        Hx = fm(sg, nrmx, Hx); Hy = fm(sg, nrmy, Hy); Hz = fm(sg, nrmz, Hz);
        if (!F.tof) { gx = Hx; gy = Hy; gz = Hz; }
    }
}

// Length restored to ms.
template <typename R, typename V>
__device__ __forceinline__ void fused_renorm(R ms, V& x, V& y, V& z)
{
    const V mm = dot3(x, x, y, y, z, z);
    const V inv = ml(bc<V, R>(ms), fs_rsqrt(mm));
    x = where_nz(mm, ml(x, inv), x);
    y = where_nz(mm, ml(y, inv), y);
    z = where_nz(mm, ml(z, inv), z);
}

// The LLG update of the spin S by the torque of the spin M in the field H (g
// without its thermal part) over dt (c_rot: its half angle per field).
template <int LT, typename R, typename V>
__device__ __forceinline__ void fused_llg(const FastKT<R>& F, R dt_, R c_rot, V Sx, V Sy, V Sz, V Mx, V My, V Mz, V Hx,
                                          V Hy, V Hz, V gx, V gy, V gz, V& rx, V& ry, V& rz)
{
    const auto B = [](R a) { return bc<V, R>(a); };
    V nx_ = Sx, ny_ = Sy, nz_ = Sz;
    if (LT == LLG_CART) {
        if (!F.dt_zero) {
            // dM = -p gaa M x H - d (a/ms) gaa M x (M x h), h = H - Hth
            const V mhx = crs(My, gz, Mz, gy), mhy = crs(Mz, gx, Mx, gz), mhz = crs(Mx, gy, My, gx);
            const V mmx = crs(My, mhz, Mz, mhy), mmy = crs(Mz, mhx, Mx, mhz), mmz = crs(Mx, mhy, My, mhx);
            const V MHx = crs(My, Hz, Mz, Hy), MHy = crs(Mz, Hx, Mx, Hz), MHz = crs(Mx, Hy, My, Hx);
            const V dt = B(dt_), cp = B(F.c_prec), cd = B(F.c_damp);
            nx_ = fm(dt, crs(cp, MHx, cd, mmx), Sx);
            ny_ = fm(dt, crs(cp, MHy, cd, mmy), Sy);
            nz_ = fm(dt, crs(cp, MHz, cd, mmz), Sz);
        }
    } else {
        V Hpx, Hpy, Hpz;
        const V cd = B(F.c_damp);
        if (F.tof) {
            const V shx = crs(My, gz, Mz, gy), shy = crs(Mz, gx, Mx, gz), shz = crs(Mx, gy, My, gx);
            const V pr = B(F.precess);
            Hpx = fm(pr, Hx, ml(cd, shx));
            Hpy = fm(pr, Hy, ml(cd, shy));
            Hpz = fm(pr, Hz, ml(cd, shz));
        } else {
            const V shx = crs(Sy, Hz, Sz, Hy), shy = crs(Sz, Hx, Sx, Hz), shz = crs(Sx, Hy, Sy, Hx);
            Hpx = fm(cd, shx, Hx); Hpy = fm(cd, shy, Hy); Hpz = fm(cd, shz, Hz);
        }
        const V HL2 = dot3(Hpx, Hpx, Hpy, Hpy, Hpz, Hpz);
        const V iHL = fs_rsqrt(HL2);
        const V th = ml(B(c_rot), ml(HL2, iHL));
        V sn, cs;
        half_sincos(th, sn, cs);
        const V k = ml(sn, iHL);
        const V qw = cs, qx = ml(k, Hpx), qy = ml(k, Hpy), qz = ml(k, Hpz);
        const V nw = dot3(qx, Sx, qy, Sy, qz, Sz);   // -tw
        const V tx = fm(qw, Sx, crs(qy, Sz, qz, Sy));
        const V ty = fm(qw, Sy, crs(qz, Sx, qx, Sz));
        const V tz = fm(qw, Sz, crs(qx, Sy, qy, Sx));
        // no rotation without a field
        nx_ = where_pos(HL2, fm(qw, tx, fm(nw, qx, crs(tz, qy, ty, qz))), Sx);
        ny_ = where_pos(HL2, fm(qw, ty, fm(nw, qy, crs(tx, qz, tz, qx))), Sy);
        nz_ = where_pos(HL2, fm(qw, tz, fm(nw, qz, crs(ty, qx, tx, qy))), Sz);
    }
    if (F.renorm) fused_renorm<R, V>(F.ms, nx_, ny_, nz_);
    rx = nx_; ry = ny_; rz = nz_;
    if (F.status) {
        const V z = B((R)0);
        if (!all_zero(fm(nx_, z, fm(ny_, z, ml(nz_, z))))) atomicOr(F.status, 1u);
    }
}

// The rest of a site's step after the Zeeman and exchange fields H.
template <int LT, bool ANI, bool TH, bool ADD, typename R, typename V>
__device__ __forceinline__ void fused_update(const FastKT<R>& F, V Sx, V Sy, V Sz, V Hx, V Hy, V Hz, V nrmx, V nrmy,
                                             V nrmz, V Ax, V Ay, V Az, V& rx, V& ry, V& rz)
{
    V gx, gy, gz;
    fused_field<ANI, TH, ADD, R, V>(F, Sx, Sy, Sz, Hx, Hy, Hz, nrmx, nrmy, nrmz, Ax, Ay, Az, gx, gy, gz);
    fused_llg<LT, R, V>(F, F.dt, F.c_rot, Sx, Sy, Sz, Sx, Sy, Sz, Hx, Hy, Hz, gx, gy, gz, rx, ry, rz);
}

// Zeeman and (EXS) exchange fields H of site i.
template <bool EXS, typename R, class LD>
__device__ __forceinline__ void fused_near(const FastKT<R>& F, int NX, int NY, int NZ, int x, int y, int z, int i,
                                           const LD& ld, R& Hx, R& Hy, R& Hz)
{
    const int nxy = NX * NY;
    if (F.Bdev) { Hx = (R)F.Bdev[0]; Hy = (R)F.Bdev[1]; Hz = (R)F.Bdev[2]; }
    else { Hx = F.B[0]; Hy = F.B[1]; Hz = F.B[2]; }
    if (EXS) {
        // the six neighbours (+x, -x, +y, -y, +z, -z; wrapped where periodic,
        // absent (-1) at an open edge); all eighteen loads are issued before
        // the first sum (an absent neighbour loads the site itself and is not
        // added), then the terms are added in the fixed neighbour order
        int f[6];
        f[0] = x + 1 < NX ? i + 1 : (F.pbc[0] ? i + 1 - NX : -1);
        f[1] = x > 0 ? i - 1 : (F.pbc[0] ? i + NX - 1 : -1);
        f[2] = y + 1 < NY ? i + NX : (F.pbc[1] ? i + NX - nxy : -1);
        f[3] = y > 0 ? i - NX : (F.pbc[1] ? i + nxy - NX : -1);
        f[4] = z + 1 < NZ ? i + nxy : (F.pbc[2] ? i + nxy - nxy * NZ : -1);
        f[5] = z > 0 ? i - nxy : (F.pbc[2] ? i + nxy * NZ - nxy : -1);
        R nb[6][3];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const int j = f[k] >= 0 ? f[k] : i;
            nb[k][0] = ld(0, j); nb[k][1] = ld(1, j); nb[k][2] = ld(2, j);
        }
        R ex = 0, ey = 0, ez = 0;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const R J = F.J[k];
            if (J != (R)0 && f[k] >= 0) {
                ex = fm(J, nb[k][0], ex); ey = fm(J, nb[k][1], ey); ez = fm(J, nb[k][2], ez);
            }
        }
        Hx = ad(Hx, ex); Hy = ad(Hy, ey); Hz = ad(Hz, ez);
    }
}

template <int LT, bool EXS, bool ANI, bool TH, bool ADD, typename R, class LD>
__device__ __forceinline__ void fused_site_ld(const FastKT<R>& F, int NX, int NY, int NZ, int x, int y, int z, int i,
                                              const LD& ld, R Ax, R Ay, R Az, R& rx, R& ry, R& rz,
                                              const float3* pre = nullptr)
{
    const R Sx = ld(0, i), Sy = ld(1, i), Sz = ld(2, i);
    R Hx, Hy, Hz;
    fused_near<EXS, R>(F, NX, NY, NZ, x, y, z, i, ld, Hx, Hy, Hz);
    float3 nrm = make_float3(0.f, 0.f, 0.f);
    if (TH) nrm = pre ? *pre : thermal_normal3(F, i);
    fused_update<LT, ANI, TH, ADD, R, R>(F, Sx, Sy, Sz, Hx, Hy, Hz, (R)nrm.x, (R)nrm.y, (R)nrm.z, Ax, Ay, Az, rx, ry, rz);
}

template <int LT, bool EXS, bool ANI, bool TH, bool ADD, typename R = float>
__device__ __forceinline__ void fused_site_v(const FastKT<R>& F, int NX, int NY, int NZ, int x, int y, int z, int i,
                                             const R* __restrict__ sx, const R* __restrict__ sy,
                                             const R* __restrict__ sz, R Ax, R Ay, R Az, R& rx, R& ry, R& rz,
                                             const float3* pre = nullptr)
{
    const GlobalSpins<R> g{{sx, sy, sz}};
    fused_site_ld<LT, EXS, ANI, TH, ADD, R>(F, NX, NY, NZ, x, y, z, i, g, Ax, Ay, Az, rx, ry, rz, pre);
}

// Two sites of a FP32 lattice at once, i and i + NX: rows y and y + 1 of one
// layer (y + 1 < NY), addends A packed (row y, row y + 1).  Every lane repeats
// fused_site_v's operations (an absent neighbour or an unused direction adds
// 0 times the site itself there instead of nothing), two per packed
// instruction; the rows are each other's y neighbours, and the neighbours'
// offsets serve both.  Byte offsets are 32 bits: at most 2^30 sites.
__device__ __forceinline__ void pair_near(const FastK& F, int NX, int NY, int NZ, int x, int y, int z, int i,
                                          const float* __restrict__ sx, const float* __restrict__ sy,
                                          const float* __restrict__ sz, p2 S[3], p2 H[3])
{
    const auto ld = [](const float* s, unsigned off) {
        return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(s) + off));
    };
    const int nxy = NX * NY;
    const unsigned o0 = 4u * (unsigned)i, o1 = o0 + 4u * (unsigned)NX;
    // offsets in bytes (0: absent) and weights of the neighbours
    int dxp = 4, dxm = -4, dyp = 4 * NX, dym = -4 * NX, dzp = 4 * nxy, dzm = -4 * nxy;
    float jxp = F.J[0], jxm = F.J[1], jyp = F.J[2], jym = F.J[3], jzp = F.J[4], jzm = F.J[5];
    if (x + 1 >= NX) { dxp = F.pbc[0] ? 4 - 4 * NX : 0; jxp = F.pbc[0] ? jxp : 0.f; }
    if (x == 0) { dxm = F.pbc[0] ? 4 * NX - 4 : 0; jxm = F.pbc[0] ? jxm : 0.f; }
    if (y + 2 >= NY) { dyp = F.pbc[1] ? 4 * NX - 4 * nxy : 0; jyp = F.pbc[1] ? jyp : 0.f; }
    if (y == 0) { dym = F.pbc[1] ? 4 * nxy - 4 * NX : 0; jym = F.pbc[1] ? jym : 0.f; }
    if (z + 1 >= NZ) { dzp = F.pbc[2] ? 4 * nxy - 4 * nxy * NZ : 0; jzp = F.pbc[2] ? jzp : 0.f; }
    if (z == 0) { dzm = F.pbc[2] ? 4 * nxy * NZ - 4 * nxy : 0; jzm = F.pbc[2] ? jzm : 0.f; }
    const float* s[3] = {sx, sy, sz};
    float own[3][2], nb[3][10];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        own[c][0] = ld(s[c], o0);
        own[c][1] = ld(s[c], o1);
        nb[c][0] = ld(s[c], o0 + dxp); nb[c][1] = ld(s[c], o1 + dxp);
        nb[c][2] = ld(s[c], o0 + dxm); nb[c][3] = ld(s[c], o1 + dxm);
        nb[c][4] = ld(s[c], o1 + dyp);
        nb[c][5] = ld(s[c], o0 + dym);
        nb[c][6] = ld(s[c], o0 + dzp); nb[c][7] = ld(s[c], o1 + dzp);
        nb[c][8] = ld(s[c], o0 + dzm); nb[c][9] = ld(s[c], o1 + dzm);
    }
    const p2 wx0 = pk(jxp, jxp), wx1 = pk(jxm, jxm), wy0 = pk(F.J[2], jyp), wy1 = pk(jym, F.J[3]);
    const p2 wz0 = pk(jzp, jzp), wz1 = pk(jzm, jzm);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        S[c] = pk(own[c][0], own[c][1]);
        p2 e = pk(0.f, 0.f);
        if (F.J[0] != 0.f) e = fm(wx0, pk(nb[c][0], nb[c][1]), e);
        if (F.J[1] != 0.f) e = fm(wx1, pk(nb[c][2], nb[c][3]), e);
        if (F.J[2] != 0.f) e = fm(wy0, pk(own[c][1], nb[c][4]), e);
        if (F.J[3] != 0.f) e = fm(wy1, pk(nb[c][5], own[c][0]), e);
        if (F.J[4] != 0.f) e = fm(wz0, pk(nb[c][6], nb[c][7]), e);
        if (F.J[5] != 0.f) e = fm(wz1, pk(nb[c][8], nb[c][9]), e);
        H[c] = ad(pk(F.B[c], F.B[c]), e);
    }
}

template <int LT, bool ANI, bool TH>
__device__ __forceinline__ void fused_pair(const FastK& F, int NX, int NY, int NZ, int x, int y, int z, int i,
                                           const float* __restrict__ sx, const float* __restrict__ sy,
                                           const float* __restrict__ sz, const p2 A[3], const p2 nrm[3], p2 r[3])
{
    p2 S[3], H[3];
    pair_near(F, NX, NY, NZ, x, y, z, i, sx, sy, sz, S, H);
    fused_update<LT, ANI, TH, true, float, p2>(F, S[0], S[1], S[2], H[0], H[1], H[2], nrm[0], nrm[1], nrm[2], A[0], A[1],
                                               A[2], r[0], r[1], r[2]);
}

// ------------------------------------------------------------------ Runge-Kutta stages
// The rows of a scheme a stage contributes to: row r advances by this stage's
// torque over dt (c_rot) from its running value (base; null: the stage's own
// spin M; fresh: from a copy of the base system's spin, which an update over
// no time leaves with its length restored) and is kept in dst.
template <int LT, typename R, typename V, class Load, class Store>
__device__ __forceinline__ void rk_rows(const FastKT<R>& F, const RkRows<R>& rows, const V M[3], const V H[3],
                                        const Load& load, const Store& store, V first[3])
{
#pragma unroll 1
    for (int r = 0; r < rows.n; r++) {
        const auto& w = rows.row[r];
        V b[3] = {M[0], M[1], M[2]}, o[3];
        if (w.base[0]) {
            for (int c = 0; c < 3; c++) b[c] = load(w.base[c]);
            if (w.fresh && F.renorm) fused_renorm<R, V>(F.ms, b[0], b[1], b[2]);
        }
        fused_llg<LT, R, V>(F, w.dt, w.c_rot, b[0], b[1], b[2], M[0], M[1], M[2], H[0], H[1], H[2], H[0], H[1], H[2], o[0],
                            o[1], o[2]);
        if (r == 0) {
            for (int c = 0; c < 3; c++) first[c] = o[c];
        } else {
            for (int c = 0; c < 3; c++) store(w.dst[c], o[c]);
        }
    }
}
