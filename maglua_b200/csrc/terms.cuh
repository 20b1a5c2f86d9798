// terms.cuh -- field terms and LLG update of one site in the general form
// (per-site parameters, pathway lists, several addends), FP32 or FP64 state;
// shared by the general step kernels (kernels.cu) and the fused x passes
// (xstep.cuh, mx.cuh).  Reference semantics are cited per function.
#pragma once
#include "device.cuh"
#include "fused.cuh"
#include "kparams.h"

#include <math.h>
#include <stdint.h>

// ------------------------------------------------------------ helpers
template <typename R>
struct V3 {
    R x, y, z;
};
template <typename R> __device__ __forceinline__ V3<R> v3(R a, R b, R c) { V3<R> v; v.x = a; v.y = b; v.z = c; return v; }
template <typename R> __device__ __forceinline__ V3<R> add3(V3<R> a, V3<R> b) { return v3<R>(ad(a.x, b.x), ad(a.y, b.y), ad(a.z, b.z)); }
template <typename R> __device__ __forceinline__ V3<R> sub3(V3<R> a, V3<R> b) { return v3<R>(ad(a.x, -b.x), ad(a.y, -b.y), ad(a.z, -b.z)); }
template <typename R> __device__ __forceinline__ V3<R> scl3(R a, V3<R> b) { return v3<R>(ml(a, b.x), ml(a, b.y), ml(a, b.z)); }
// h + a b
template <typename R> __device__ __forceinline__ V3<R> fma3(R a, V3<R> b, V3<R> h) { return v3<R>(fm(a, b.x, h.x), fm(a, b.y, h.y), fm(a, b.z, h.z)); }
template <typename R> __device__ __forceinline__ V3<R> cross3(V3<R> a, V3<R> b)
{
    return v3<R>(crs(a.y, b.z, a.z, b.y), crs(a.z, b.x, a.x, b.z), crs(a.x, b.y, a.y, b.x));
}
template <typename R> __device__ __forceinline__ R ldr(const void* p, int i) { return __ldg(static_cast<const R*>(p) + i); }
template <typename R> __device__ __forceinline__ R ms_at(const SysK& s, int i) { return s.ms_uniform ? (R)s.ms_u : ldr<R>(s.ms, i); }
template <typename R> __device__ __forceinline__ R alpha_at(const SysK& s, int i) { return s.site_alpha ? ldr<R>(s.site_alpha, i) : (R)s.alpha; }
template <typename R> __device__ __forceinline__ R gamma_at(const SysK& s, int i) { return s.site_gamma ? ldr<R>(s.site_gamma, i) : (R)s.gamma; }
template <typename R> __device__ __forceinline__ V3<R> spin_at(const SysK& s, int i)
{
    return v3<R>(ldr<R>(s.x, i), ldr<R>(s.y, i), ldr<R>(s.z, i));
}
template <typename R> __device__ __forceinline__ R rsq(R v);
template <> __device__ __forceinline__ float rsq<float>(float v) { return sqrtf(v); }
template <> __device__ __forceinline__ double rsq<double>(double v) { return sqrt(v); }
__device__ __forceinline__ void sincos_r(float v, float* s, float* c) { sincosf(v, s, c); }
__device__ __forceinline__ void sincos_r(double v, double* s, double* c) { sincos(v, s, c); }

// ------------------------------------------------------------ field terms
// Exchange: h_t += J s_f / (m_f m_t) (normalised) or J s_f / m_f, only for
// m_f != 0 (M/cpu/exchange/spinoperationexchange.cpp:134-213).
template <typename R>
__device__ __forceinline__ V3<R> ex_term(const ExchangeK& e, const SysK& s, int i, R mt)
{
    V3<R> h = v3<R>(0, 0, 0);
    if (e.mode == EX_STENCIL) {
        const int ix = i % s.nx;
        const int iy = (i / s.nx) % s.ny;
        const int iz = i / (s.nx * s.ny);
        const int nxy = s.nx * s.ny;
        // the six neighbours' loads are all issued before the first sum (an
        // absent one loads the site itself and is not added)
        int f[6];
        R mf[6];
        V3<R> sf[6];
#pragma unroll
        for (int d = 0; d < 6; d++) {
            const int ax = d >> 1;
            const int sg = (d & 1) ? -1 : 1;
            const int c0 = ax == 0 ? ix : (ax == 1 ? iy : iz);
            const int n = ax == 0 ? s.nx : (ax == 1 ? s.ny : s.nz);
            const int st = ax == 0 ? 1 : (ax == 1 ? s.nx : nxy);
            int c = c0 + sg;
            bool on = e.J[d] != 0.0;
            if (c < 0 || c >= n) {
                on = on && e.pbc[ax];
                c = c < 0 ? c + n : c - n;
            }
            f[d] = on ? i + (c - c0) * st : -1;
            const int j = on ? f[d] : i;
            mf[d] = ms_at<R>(s, j);
            sf[d] = spin_at<R>(s, j);
        }
#pragma unroll
        for (int d = 0; d < 6; d++)
            if (f[d] >= 0 && mf[d] != (R)0)
                h = fma3((R)e.J[d] / (e.normalize ? ml(mf[d], mt) : mf[d]), sf[d], h);   // one division per neighbour
    } else if (e.mode == EX_CSR) {
        // the site's pathways six at a time, the loads of a round issued
        // together (two dependent memory latencies per round instead of two
        // per pathway: 128 x 128 x 4 grains, the step alone 22.4 -> 19.2 us)
        const int p0 = __ldg(e.ptr + i), p1 = __ldg(e.ptr + i + 1);
        for (int p = p0; p < p1; p += 6) {
            int f[6];
            R J[6], mf[6];
            V3<R> sf[6];
#pragma unroll
            for (int u = 0; u < 6; u++) {
                const int q = min(p + u, p1 - 1);
                f[u] = __ldg(e.col + q);
                J[u] = (R)__ldg(e.val + q);
            }
#pragma unroll
            for (int u = 0; u < 6; u++) {
                mf[u] = ms_at<R>(s, f[u]);
                sf[u] = spin_at<R>(s, f[u]);
            }
#pragma unroll
            for (int u = 0; u < 6; u++)
                if (p + u < p1 && mf[u] != (R)0)
                    h = fma3(J[u] / (e.normalize ? ml(mf[u], mt) : mf[u]), sf[u], h);
        }
    }
    return h;
}

// Anisotropy: H = 2K (s.n)/ms^2 n for ms > 0
// (M/cpu/anisotropy/spinoperationanisotropy.cpp:247-283).
template <typename R>
__device__ __forceinline__ V3<R> ani_one(V3<R> sp, R ms, R n0, R n1, R n2, R K)
{
    const R sda = dot3(sp.x, n0, sp.y, n1, sp.z, n2);
    const R v = ml(ml((R)2, K), sda) / ml(ms, ms);
    return v3<R>(ml(n0, v), ml(n1, v), ml(n2, v));
}
template <typename R>
__device__ __forceinline__ V3<R> ani_term(const AniK& a, V3<R> sp, R ms, int i)
{
    V3<R> h = v3<R>(0, 0, 0);
    if (!(ms > (R)0)) return h;
    if (a.mode == ANI_UNIFORM) return ani_one<R>(sp, ms, (R)a.axis[0], (R)a.axis[1], (R)a.axis[2], (R)a.K);
    if (a.mode == ANI_CSR) {
        const int p0 = __ldg(a.ptr + i), p1 = __ldg(a.ptr + i + 1);
        for (int p = p0; p < p1; p++)
            h = add3(h, ani_one<R>(sp, ms, (R)__ldg(a.axes + 3 * p), (R)__ldg(a.axes + 3 * p + 1),
                                   (R)__ldg(a.axes + 3 * p + 2), (R)__ldg(a.Ks + p)));
    }
    return h;
}

// Uniaxial: [2K1 u + 4K2 u^3] n with u = s.n of the unit spin; quirk keeps
// the reference's sz*nx (..._uniaxial.cpp:250-298, :287).
template <typename R>
__device__ __forceinline__ V3<R> uni_one(V3<R> u3, R n0, R n1, R n2, R K1, R K2, int quirk)
{
    const R u = dot3(u3.x, n0, u3.y, n1, u3.z, quirk ? n0 : n2);
    const R mag = fm(ml((R)2, K1), u, ml(ml((R)4, K2), ml(ml(u, u), u)));
    return v3<R>(ml(n0, mag), ml(n1, mag), ml(n2, mag));
}
template <typename R>
__device__ __forceinline__ V3<R> uni_term(const UniK& a, V3<R> sp, R ms, int i)
{
    V3<R> h = v3<R>(0, 0, 0);
    if (!(ms > (R)0) || a.mode == ANI_NONE) return h;
    const V3<R> u = v3<R>(sp.x / ms, sp.y / ms, sp.z / ms);
    if (a.mode == ANI_UNIFORM)
        return uni_one<R>(u, (R)a.axis[0], (R)a.axis[1], (R)a.axis[2], (R)a.K1, (R)a.K2, a.quirk);
    const int p0 = __ldg(a.ptr + i), p1 = __ldg(a.ptr + i + 1);
    for (int p = p0; p < p1; p++)
        h = add3(h, uni_one<R>(u, (R)__ldg(a.axes + 3 * p), (R)__ldg(a.axes + 3 * p + 1), (R)__ldg(a.axes + 3 * p + 2),
                               (R)__ldg(a.K12 + 2 * p), (R)__ldg(a.K12 + 2 * p + 1), a.quirk));
    return h;
}

// Cubic (..._cubic.cpp:308-390): cubic_field (fused.cuh) on a V3.
template <typename R>
__device__ __forceinline__ V3<R> cub_one(V3<R> s, const R* n, const R* K, int quirk)
{
    V3<R> h;
    cubic_field<R>(s.x, s.y, s.z, n, K, quirk, h.x, h.y, h.z);
    return h;
}
template <typename R>
__device__ __forceinline__ V3<R> cub_term(const CubK& a, V3<R> sp, R ms, int i)
{
    V3<R> h = v3<R>(0, 0, 0);
    if (!(ms > (R)0) || a.mode == ANI_NONE) return h;
    const V3<R> u = v3<R>(sp.x / ms, sp.y / ms, sp.z / ms);
    R n[9], K[3];
    if (a.mode == ANI_UNIFORM) {
#pragma unroll
        for (int q = 0; q < 9; q++) n[q] = (R)a.axes[q];
#pragma unroll
        for (int q = 0; q < 3; q++) K[q] = (R)a.K[q];
        return cub_one<R>(u, n, K, a.quirk);
    }
    const int p0 = __ldg(a.ptr + i), p1 = __ldg(a.ptr + i + 1);
    for (int p = p0; p < p1; p++) {
#pragma unroll
        for (int q = 0; q < 9; q++) n[q] = (R)__ldg(a.axs + 9 * p + q);
#pragma unroll
        for (int q = 0; q < 3; q++) K[q] = (R)__ldg(a.Ks + 3 * p + q);
        h = add3(h, cub_one<R>(u, n, K, a.quirk));
    }
    return h;
}

// Thermal: sigma = sqrt(2 alpha T scale / (ms dt gamma)) times N(0,1) per
// component, zero where ms == 0, T == 0 or gamma <= 0
// (M/cpu/thermal/spinoperationthermal.cpp:135-191).
template <typename R>
__device__ __forceinline__ V3<R> th_term(const ThermalK& t, const SysK& s, R dt_sys, int i, R ms)
{
    V3<R> h = v3<R>(0, 0, 0);
    if (t.mode == TH_NONE || ms == (R)0 || t.T == 0.0) return h;
    const R a = alpha_at<R>(s, i), g = gamma_at<R>(s, i);
    if (!(g > (R)0)) return h;
    const R sc = t.scale ? (R)__ldg(t.scale + i) : (R)1;
    const R sd = rsq<R>(ml(ml(ml((R)2, a), (R)t.T), sc) / ml(ml(ms, dt_sys), g));
    V3<R> n;
    if (t.mode == TH_PHILOX) {
        const uint64_t ctr = t.counter + (t.dctr ? *t.dctr : 0ull);
        const float3 f = philox_normal3(t.seed, ctr, (uint32_t)i, 0x6d6c6232u);
        n = v3<R>((R)f.x, (R)f.y, (R)f.z);
    } else {
        n = v3<R>((R)__ldg(t.nx + i), (R)__ldg(t.ny + i), (R)__ldg(t.nz + i));
    }
    return scl3(sd, n);
}

template <typename R>
struct Fields {
    V3<R> H;
    V3<R> Hth;
};

// Every term of TermsK at site i.  H is the would-be "Total" slot, Hth the
// "Thermal" slot that LLG subtracts (llgcartesian.cpp:160-172).
template <typename R>
__device__ __forceinline__ Fields<R> eval_terms(const TermsK& T, const SysK& s, R dt_sys, int i)
{
    const R ms = ms_at<R>(s, i);
    const V3<R> sp = spin_at<R>(s, i);
    V3<R> H = v3<R>(0, 0, 0);
    V3<R> Hth = v3<R>(0, 0, 0);
    if (T.ex.mode != EX_NONE) H = add3(H, scl3((R)T.ex_gs, ex_term<R>(T.ex, s, i, ms)));
    if (T.ani.mode != ANI_NONE) H = add3(H, ani_term<R>(T.ani, sp, ms, i));
    if (T.uni.mode != ANI_NONE) H = add3(H, uni_term<R>(T.uni, sp, ms, i));
    if (T.cub.mode != ANI_NONE) H = add3(H, cub_term<R>(T.cub, sp, ms, i));
    if (T.th.mode != TH_NONE) { Hth = th_term<R>(T.th, s, dt_sys, i, ms); H = add3(H, Hth); }
    if (T.zee.on) {
        const V3<R> B = T.zee.Bdev ? v3<R>((R)T.zee.Bdev[0], (R)T.zee.Bdev[1], (R)T.zee.Bdev[2])
                                   : v3<R>((R)T.zee.B[0], (R)T.zee.B[1], (R)T.zee.B[2]);
        H = add3(H, B);
    }
    for (int a = 0; a < T.nadd; a++) {
        const V3<R> v = v3<R>(ldr<R>(T.add[a][0], i), ldr<R>(T.add[a][1], i), ldr<R>(T.add[a][2], i));
        const R w = (R)T.addw[a];
        H = fma3(w, v, H);
        if (T.add_is_thermal[a]) Hth = add3(Hth, v);
    }
    Fields<R> f;
    f.H = H;
    f.Hth = Hth;
    return f;
}

// ------------------------------------------------------------ LLG
// Cartesian Euler step (M/cpu/llg/llgcartesian.cpp:90-278) or quaternion
// rotation (M/cpu/llg/llgquat.cpp:126-378) for one site with ms > 0.
// S: from-spin, M: dmdt-spin, H: Total, Hth: Thermal.
template <typename R>
__device__ __forceinline__ V3<R> llg_site(const LlgK& L, V3<R> S, V3<R> M, V3<R> H, V3<R> Hth, R ms, R a, R g)
{
    const R dt = (R)L.dt, p = (R)L.precess, d = (R)L.damp;
    if (L.type == LLG_CART) {
        if (L.dt_zero) return S;
        const R gaa = g / fm(a, a, (R)1);
        if (L.thermal_only_first_term) {
            const V3<R> h = sub3(H, Hth);
            const V3<R> Mh = cross3(M, h);
            const V3<R> MMH = cross3(M, Mh);
            const V3<R> MH = cross3(M, H);
            const V3<R> dM = fma3(ml(p, -gaa), MH, scl3(-ml(ml(d, a / ms), gaa), MMH));
            return fma3(dt, dM, S);
        }
        const V3<R> MH = cross3(M, H);
        const V3<R> MMH = cross3(M, MH);
        const V3<R> dM = fma3(-gaa, MH, scl3(-ml(a / ms, gaa), MMH));
        return fma3(dt, dM, S);
    }
    // quaternion
    const R inv = (R)1 / ms;
    V3<R> Hp;
    if (L.thermal_only_first_term) {
        const V3<R> h = sub3(H, Hth);
        const V3<R> Sh = cross3(M, h);
        Hp = fma3(p, H, scl3(ml(ml(d, a), inv), Sh));
    } else {
        const V3<R> SH = cross3(S, H);
        Hp = fma3(ml(a, inv), SH, H);
    }
    const R HLen = rsq<R>(dot3(Hp.x, Hp.x, Hp.y, Hp.y, Hp.z, Hp.z));
    if (!(HLen > (R)0)) return S;
    const R iHLen = (R)1 / HLen;
    const R ra = ml(g, HLen) / fm(a, a, (R)1);
    R sint, cost;
    sincos_r(ml(ml((R)0.5, ra), dt), &sint, &cost);
    // qRot = (cost, sint * Hp/|Hp|); qRes = qRot * (0,S) * conj(qRot)
    const R k = ml(sint, iHLen);
    const R qw = cost, qx = ml(k, Hp.x), qy = ml(k, Hp.y), qz = ml(k, Hp.z);
    const R tw = -dot3(qx, S.x, qy, S.y, qz, S.z);
    const R tx = fm(qw, S.x, crs(qy, S.z, qz, S.y));
    const R ty = fm(qw, S.y, crs(qz, S.x, qx, S.z));
    const R tz = fm(qw, S.z, crs(qx, S.y, qy, S.x));
    V3<R> r;
    r.x = fm(qw, tx, fm(-tw, qx, crs(tz, qy, ty, qz)));
    r.y = fm(qw, ty, fm(-tw, qy, crs(tx, qz, tz, qx)));
    r.z = fm(qw, tz, fm(-tw, qz, crs(ty, qx, tx, qy)));
    return r;
}

template <typename R>
__device__ __forceinline__ V3<R> renorm(V3<R> v, R ms)
{
    const R mm = dot3(v.x, v.x, v.y, v.y, v.z, v.z);
    if (mm != (R)0) {
        const R inv = ms / rsq<R>(mm);
        return scl3(inv, v);
    }
    return v;
}

// The LLG update of site i in the field F: sites with ms <= 0 keep their
// spin; length restored, non-finite results flagged.
template <typename R>
__device__ __forceinline__ V3<R> step_site(const FusedK& P, const Fields<R>& F, V3<R> S, R ms, int i)
{
    V3<R> out = S;
    if (ms > (R)0) out = llg_site<R>(P.llg, S, S, F.H, F.Hth, ms, alpha_at<R>(P.sys, i), gamma_at<R>(P.sys, i));
    if (P.llg.renorm) out = renorm<R>(out, ms);
    if (P.llg.status && !(isfinite(out.x) && isfinite(out.y) && isfinite(out.z))) atomicOr(P.llg.status, 1u);
    return out;
}
