// site_pack.cuh -- the per-site Ginzburg-Landau stencils: energy, gradient,
// line quartic, B and J.
//
// Packs.  Every per-component quantity is a pack: the number itself for one
// component, both components' values for two (FP32: a float2 on the packed
// FP32x2 pipes; paired FP64: a packed float-float; FP64: two doubles).  What
// carries no component (A, the magnetic views, the couplings) is scalar.
//
// Form of the terms.  A link i -> j with a = q A dx at its ends (lattice
// units), Delta = psi_j - psi_i and the reference's linearised covariant
// differences u0..u3 (nlcg.cu:149-203) has
//
//   sum u^2 / 2 = |Delta|^2 + s (y_i Dx - x_i Dy) + (a_i^2 |psi_i|^2 + a_j^2 |psi_j|^2) / 2,
//   s = a_i + a_j,
//
// because y_i Dx - x_i Dy = y_j Dx - x_j Dy.  The last two terms belong to
// the sites, with the weights of both links that meet there, so a link costs
// the product of Delta with (Dx + s y, Dy - s x) and nothing per end; its
// force on site i is -2 (Delta +- (s / 2) (y_j, -x_j)) + a_i^2 psi_i.  The
// differences Delta are formed before anything is multiplied, as in u0..u3.
// Where A is strong (vortices) the three terms cancel and leave rounding errors
// of their own size.  So a = q A dx is rounded once and used in all of them, and
// 1 / (2 m dx^2) is one constant: a rounded constant is then a slightly other dx
// or m, no mismatch between the terms.  With (q dx)^2 / (4 m dx^2) a constant of
// its own, the energy of 100 vortices on 300 x 300 sites was 2.7e-7 off in FP32
// and 1.5e-14 in float-float; 5.3e-8 and 5.3e-15 this way, 3.9e-8 and 1.3e-15
// with the u squared.  The energy by itself (site_energy) squares the u, which
// costs about as much there; in the quartic it would be a tenth of a float-float
// step (256 x 256 x 64, four steps: 5.8 against 6.6 ms; FP64, two: 7.7 against
// 8.1).  Spacings are folded into the parameters: the gradient's kinetic and
// magnetic terms carry no 1/dx (dx^2 / dx^2 = 1).
//
// Why: GB300 issues two FP64 operations per SM and clock, so the double
// passes take 16 clocks per warp instruction and are bound by their count
// alone (95 % of that rate measured); the float-float and FP32 passes are
// bound by issue.  The forms the reference writes out cost 345 FP64
// instructions per two-component site in the gradient and 486 in the
// quartic.  These forms alone, on the two-component 256 x 256 string of 64
// images, took an FP64 step from 6.43 to 4.60 ms (3.83 with the strips), FP32
// reparametrization and ten steps from 2.66 to 2.42 (2.27).
#pragma once

#include "site_ops.cuh"

namespace mepgl {

// ------------------------------------------------------------------- packs
struct dp2 {
    double x, y;
};

template <class S, int NC> struct PackOf { using type = S; };
template <> struct PackOf<float, 2> { using type = float2; };
template <> struct PackOf<double, 2> { using type = dp2; };
template <> struct PackOf<ff, 2> { using type = ffp; };
template <class S, int NC> using pack_t = typename PackOf<S, NC>::type;

__device__ __forceinline__ float fma1(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma1(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ ff fma1(ff a, ff b, ff c) { return a * b + c; }

__device__ __forceinline__ float padd(float a, float b) { return a + b; }
__device__ __forceinline__ float psub(float a, float b) { return a - b; }
__device__ __forceinline__ float pmul(float a, float b) { return a * b; }
__device__ __forceinline__ float pfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float pnfma(float a, float b, float c) { return __fmaf_rn(-a, b, c); }

__device__ __forceinline__ double padd(double a, double b) { return a + b; }
__device__ __forceinline__ double psub(double a, double b) { return a - b; }
__device__ __forceinline__ double pmul(double a, double b) { return a * b; }
__device__ __forceinline__ double pfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double pnfma(double a, double b, double c) { return __fma_rn(-a, b, c); }

__device__ __forceinline__ ff padd(ff a, ff b) { return a + b; }
__device__ __forceinline__ ff psub(ff a, ff b) { return a - b; }
__device__ __forceinline__ ff pmul(ff a, ff b) { return a * b; }
__device__ __forceinline__ ff pfma(ff a, ff b, ff c) { return a * b + c; }
__device__ __forceinline__ ff pnfma(ff a, ff b, ff c) { return c - a * b; }

__device__ __forceinline__ dp2 padd(dp2 a, dp2 b) { return dp2{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ dp2 psub(dp2 a, dp2 b) { return dp2{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ dp2 pmul(dp2 a, dp2 b) { return dp2{a.x * b.x, a.y * b.y}; }
__device__ __forceinline__ dp2 pfma(dp2 a, dp2 b, dp2 c) { return dp2{__fma_rn(a.x, b.x, c.x), __fma_rn(a.y, b.y, c.y)}; }
__device__ __forceinline__ dp2 pnfma(dp2 a, dp2 b, dp2 c)
{
    return dp2{__fma_rn(-a.x, b.x, c.x), __fma_rn(-a.y, b.y, c.y)};
}

__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
// a - b (b * -1 is exact, so this rounds once, as a - b does)
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 pnfma(float2 a, float2 b, float2 c) { return __ffma2_rn(neg2f(a), b, c); }

__device__ __forceinline__ ffp padd(ffp a, ffp b) { return a + b; }
__device__ __forceinline__ ffp psub(ffp a, ffp b) { return a - b; }
__device__ __forceinline__ ffp pmul(ffp a, ffp b) { return a * b; }
__device__ __forceinline__ ffp pfma(ffp a, ffp b, ffp c) { return a * b + c; }
__device__ __forceinline__ ffp pnfma(ffp a, ffp b, ffp c) { return c - a * b; }

// same value in every component; one value per component; sum over them; one of them
template <class S, int NC> struct Pk {
    using P = pack_t<S, NC>;
    static __device__ __forceinline__ P bc(S a)
    {
        if constexpr (NC == 1) return a;
        else return mk(a, a);
    }
    static __device__ __forceinline__ P mk(S a, S b)
    {
        if constexpr (NC == 1) return a;
        else if constexpr (std::is_same<S, ff>::value) return ffp{make_float2(a.hi, b.hi), make_float2(a.lo, b.lo)};
        else if constexpr (std::is_same<S, float>::value) return make_float2(a, b);
        else return dp2{a, b};
    }
    template <int C> static __device__ __forceinline__ S lane(P p)
    {
        if constexpr (NC == 1) return p;
        else if constexpr (std::is_same<S, ff>::value) return C == 0 ? ff(p.hi.x, p.lo.x) : ff(p.hi.y, p.lo.y);
        else return C == 0 ? p.x : p.y;
    }
    static __device__ __forceinline__ S sum(P p)
    {
        if constexpr (NC == 1) return p;
        else return lane<0>(p) + lane<1>(p);
    }
};

// Neighbourhood of one site: A and Re / Im psi packs at (dx, dy) = [dy + 1][dx + 1].
template <class S, int NC>
struct PackView {
    using P = pack_t<S, NC>;
    vec2_t<S> a[3][3];
    P px[3][3], py[3][3];
};

// Value of a site in one of PairSites' arrays.
__device__ __forceinline__ ff pair_site(const void *p, int s)
{
    const float2 v = static_cast<const float2 *>(p)[s];
    return ff(v.x, v.y);
}

// Parameters as the stencils use them: read from the descriptor, and the
// site's own where the string has per-site arrays.
template <class S, int NC>
struct PackParams {
    using P = pack_t<S, NC>;
    using K = Pk<S, NC>;
    P qd, hqd, nhqd, kq, qi;        // q dx, +- half of it, (q + 1) dx, q / dx
    P hmx, hmy, n2hmx, n2hmy;       // 1 / (2 m), -1 / m
    P hhmx, hhmy;                   // 1 / (4 m dx^2) (not per site)
    P jmx, jmy;                     // qi / (2 m)
    P hmxi, hmyi, hmxil, hmyid;     // 1 / (2 m dx^2); at the left / lower neighbour (their forward links end here)
    P aob, b, a2, b2;               // a / b, b; 2 a dx^2, 2 b dx^2
    S eta, gamma, delta, h, idx, idx4, idx8;
    S etad, gammad, deltad, hd, hl; // couplings times dx^2; h dx, and what h lost in rounding to float
    __device__ __forceinline__ void load(const StringDesc &D)
    {
        const Uniform<S> &U = D.template u<S>();
        qd = K::mk(U.qd[0], U.qd[1]);
        hqd = K::mk(U.hqd[0], U.hqd[1]);
        nhqd = K::mk(U.nhqd[0], U.nhqd[1]);
        kq = K::mk(U.kq[0], U.kq[1]);
        qi = K::mk(U.qi[0], U.qi[1]);
        hmx = K::mk(U.hmx[0], U.hmx[1]);
        hmy = K::mk(U.hmy[0], U.hmy[1]);
        hmxi = hmxil = K::mk(U.hmxi[0], U.hmxi[1]);
        hmyi = hmyid = K::mk(U.hmyi[0], U.hmyi[1]);
        jmx = K::mk(U.jmx[0], U.jmx[1]);
        jmy = K::mk(U.jmy[0], U.jmy[1]);
        hhmx = K::mk(U.hhmx[0], U.hhmx[1]);
        hhmy = K::mk(U.hhmy[0], U.hhmy[1]);
        n2hmx = K::mk(U.n2hmx[0], U.n2hmx[1]);
        n2hmy = K::mk(U.n2hmy[0], U.n2hmy[1]);
        aob = K::mk(U.aob[0], U.aob[1]);
        b = K::mk(U.b[0], U.b[1]);
        a2 = K::mk(U.a2[0], U.a2[1]);
        b2 = K::mk(U.b2[0], U.b2[1]);
        eta = U.eta;
        gamma = U.gamma;
        delta = U.delta;
        h = U.h;
        idx = U.idx;
        idx4 = U.idx4;
        idx8 = U.idx8;
        etad = U.etad;
        gammad = U.gammad;
        deltad = U.deltad;
        hd = U.hd;
        hl = U.hl;
    }
    // Per-site strings: the parameters of site s = (i, j).  All loads stand before the
    // first division: a division may branch, loads are not moved across that, and a
    // site's loads then wait for each other (FP32, two components, 256 x 256 x 32, with
    // FieldSites ahead of them: gradients 81 -> 61 us, energies 66 -> 55, five steps
    // 1019 -> 744; one component 56 -> 49, 54 -> 45, 683 -> 598).
    __device__ __forceinline__ void load_site(const StringDesc &D, int i, int j, int s)
    {
        using St = store_t<S>;
        St ra[NC], rb[NC], mx[NC], my[NC], ml[NC], md[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            ra[c] = static_cast<const St *>(D.pa[c])[s];
            rb[c] = static_cast<const St *>(D.pb[c])[s];
            mx[c] = static_cast<const St *>(D.pmxx[c])[s];
            my[c] = static_cast<const St *>(D.pmyy[c])[s];
            ml[c] = static_cast<const St *>(D.pmxx[c])[i > 0 ? s - 1 : s];
            md[c] = static_cast<const St *>(D.pmyy[c])[j > 0 ? s - D.nx : s];
        }
        const St rh = static_cast<const St *>(D.ph)[s];
        SiteParams<S> p;
        p.load_uniform(D);
        S x[2], y[2];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            p.a[c] = from_store<S>(ra[c]);
            p.b[c] = from_store<S>(rb[c]);
            p.hmx[c] = from_store<S>((St)0.5 / mx[c]);
            p.hmy[c] = from_store<S>((St)0.5 / my[c]);
            p.aob[c] = from_store<S>(ra[c] / rb[c]);
            x[c] = from_store<S>((St)0.5 / ml[c]);
            y[c] = from_store<S>((St)0.5 / md[c]);
        }
        p.h = from_store<S>(rh);
        take_site(p, x, y);
    }
    // in the NLCG passes, whose float-float ones have them as pairs
    __device__ __forceinline__ void load_pass_site(const StringDesc &D, int i, int j, int s)
    {
        if constexpr (!std::is_same<S, ff>::value) return load_site(D, i, j, s);
        else load_pairs(D, i, j, s);
    }
    __device__ __forceinline__ void load_pairs(const StringDesc &D, int i, int j, int s)
    {
        SiteParams<S> p;
        p.load_uniform(D);
        S x[2], y[2];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            p.a[c] = pair_site(D.pairs.a[c], s);
            p.b[c] = pair_site(D.pairs.b[c], s);
            p.hmx[c] = pair_site(D.pairs.hmx[c], s);
            p.hmy[c] = pair_site(D.pairs.hmy[c], s);
            p.aob[c] = pair_site(D.pairs.aob[c], s);
            x[c] = pair_site(D.pairs.hmx[c], i > 0 ? s - 1 : s);
            y[c] = pair_site(D.pairs.hmy[c], j > 0 ? s - D.nx : s);
        }
        p.h = pair_site(D.pairs.h, s);
        take_site(p, x, y);
    }
    // x, y: 1 / (2 m) at the left and the lower neighbour
    __device__ __forceinline__ void take_site(const SiteParams<S> &p, const S (&x)[2], const S (&y)[2])
    {
        const S d2 = p.dx2, two = S(2.0f), n2 = S(-2.0f);
        const P i2 = K::bc(idx * idx);
        hmx = K::mk(p.hmx[0], p.hmx[NC - 1]);
        hmy = K::mk(p.hmy[0], p.hmy[NC - 1]);
        hmxi = pmul(hmx, i2);
        hmyi = pmul(hmy, i2);
        hmxil = pmul(K::mk(x[0], x[NC - 1]), i2);
        hmyid = pmul(K::mk(y[0], y[NC - 1]), i2);
        jmx = pmul(hmx, qi);
        jmy = pmul(hmy, qi);
        n2hmx = pmul(hmx, K::bc(n2));
        n2hmy = pmul(hmy, K::bc(n2));
        aob = K::mk(p.aob[0], p.aob[NC - 1]);
        b = K::mk(p.b[0], p.b[NC - 1]);
        a2 = K::mk(two * p.a[0] * d2, two * p.a[NC - 1] * d2);
        b2 = K::mk(two * p.b[0] * d2, two * p.b[NC - 1] * d2);
        h = p.h;
        hd = p.h * p.dx;
        hl = S(0.0f);
    }
};

// Weights of a site whose neighbours all lie inside both domains, as
// constants (FP64 strips: a row of such sites drops every multiplication by a
// weight, some 26 of the instructions of the gradient and 24 of the quartic).
// Without per-site arrays the quartic's link sums also leave out the mass, which
// multiplies them once per strip (16 more; steps of 256 x 256 x 64 3 % quicker).
struct Ones {
    static constexpr bool interior = true, masses = false;   // masses: each site's own, so they stay in the links' sums
    static constexpr double area = 1, wfx = 1, wbx = 1, wfy = 1, wby = 1, wsx = 2, wsy = 2;
    static constexpr double vUR = 1, vUL = 1, vLL = 1, vLR = 1, ivs = 0.25;
};

struct OnesPerSite : Ones {
    static constexpr bool masses = true;
};

// FP64: a biquadratic coupling of zero is skipped (a uniform branch; its 26
// instructions cost 26 x 16 clocks per warp).  FP32 and float-float keep the
// straight line (the branch measured slower there).
template <class S> struct SkipZeroDelta { static constexpr bool v = std::is_same<S, double>::value; };

// Four collocated views of (curl A - h) dx at one site, from the forward and
// backward differences of A_y along x (yp, ym) and of A_x along y (xp, xm).
template <class S>
struct Curl {
    S yp, ym, xp, xm;
    template <class V> __device__ __forceinline__ Curl(const V (&a)[3][3])
    {
        yp = a[1][2].y - a[1][1].y;
        ym = a[1][1].y - a[1][0].y;
        xp = a[2][1].x - a[1][1].x;
        xm = a[1][1].x - a[0][1].x;
    }
    // FP32: the views' field is a rounded constant, and much of the energy of a
    // string is its square, so the remainder is taken off the differences, where
    // it still counts (256 x 256 x 64 at h = 0.9, relaxed: energies 3.5e-7 from 64
    // bits without, 4.5e-8 with)
    __device__ __forceinline__ void field(S hl)
    {
        if constexpr (std::is_same<S, float>::value) {
            xp += hl;
            xm += hl;
        }
    }
};

// ------------------------------------------------------------------ energy
// Free-energy density (freeEnergyDensity, nlcg.cu:105-214); the caller
// multiplies the image's sum by dx^2.
//
// The energy and the quartic are sums of terms that cancel against one another
// (the field's h^2 / 2 against the couplings' gain in the benchmark strings),
// so their parameters stay as given and the spacing enters as one common
// factor of the whole sum: folding dx^2 into each parameter, with a rounding
// each, left an FP32 energy 6.4e-7 off where it is 3.6e-7 with the factor
// outside.
template <class S, int NC, class Wt>
__device__ __forceinline__ S site_energy(const PackView<S, NC> &v, const PackParams<S, NC> &pp, const Wt &w,
                                         int thin_film)
{
    using K = Pk<S, NC>;
    using P = pack_t<S, NC>;
    constexpr bool ones = Wt::interior;
    const P X = v.px[1][1], Y = v.py[1][1];
    const P r = pfma(Y, Y, pmul(X, X)), n = padd(r, pp.aob);
    const P bh = pmul(pp.b, K::bc(ones ? S(0.5f) : S(0.5f) * S(w.area)));
    P k = K::bc(S(0.0f));
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
        const S Ai = dir == 0 ? v.a[1][1].x : v.a[1][1].y, Aj = dir == 0 ? v.a[1][2].x : v.a[2][1].y;
        const P xj = dir == 0 ? v.px[1][2] : v.px[2][1], yj = dir == 0 ? v.py[1][2] : v.py[2][1];
        const P hm = dir == 0 ? pp.hmxi : pp.hmyi;
        const P f = ones ? hm : pmul(hm, K::bc(S(dir == 0 ? w.wfx : w.wfy)));
        const P ai = pmul(pp.qd, K::bc(Ai)), aj = pmul(pp.qd, K::bc(Aj));
        const P Dx = psub(xj, X), Dy = psub(Y, yj);       // Dy: -(y_j - y_i)
        const P u0 = pfma(ai, Y, Dx), u1 = pfma(aj, yj, Dx), u2 = pfma(ai, X, Dy), u3 = pfma(aj, xj, Dy);
        k = pfma(f, pfma(u0, u0, pfma(u1, u1, pfma(u2, u2, pmul(u3, u3)))), k);
    }
    const P e = pfma(K::bc(S(0.5f)), k, pmul(pmul(bh, n), n));
    S t = K::sum(e);
    if constexpr (NC == 2) {
        const S x1 = K::template lane<0>(X), y1 = K::template lane<0>(Y);
        const S x2 = K::template lane<1>(X), y2 = K::template lane<1>(Y);
        const S r1 = K::template lane<0>(r), r2 = K::template lane<1>(r);
        const S R = fma1(y1, y2, x1 * x2), I = fma1(x1, y2, -(y1 * x2));
        S cp = pp.eta * R;
        cp = fma1(S(0.5f) * pp.gamma * r1, r2, cp);
        cp = fma1(S(0.5f) * pp.delta, fma1(R, R, -(I * I)), cp);
        t = ones ? t + cp : fma1(S(w.area), cp, t);
    }
    if (!thin_film) {
        Curl<S> c(v.a);
        c.field(pp.hl);
        const S nh = -pp.h;
        const S r0 = fma1(pp.idx, c.yp - c.xp, nh), r1 = fma1(pp.idx, c.ym - c.xp, nh);
        const S r2 = fma1(pp.idx, c.ym - c.xm, nh), r3 = fma1(pp.idx, c.yp - c.xm, nh);
        S em = ones ? r0 * r0 : (S(w.vUR) * r0) * r0;
        em = fma1(ones ? r1 : S(w.vUL) * r1, r1, em);
        em = fma1(ones ? r2 : S(w.vLL) * r2, r2, em);
        em = fma1(ones ? r3 : S(w.vLR) * r3, r3, em);
        t = fma1(S(0.125f), em, t);
    }
    return t;
}

// Partial derivatives of the energy at fixed fields with respect to a uniform
// shift of the applied field h, to eta and to gamma (no reference
// counterpart), summed without their constants: h += sum over the views of
// w_v (curl - h) (times -dx^2 / 4), eta += area Re(psi1 psi2*) (dx^2), gamma
// += area |psi1|^2 |psi2|^2 (dx^2 / 2).
template <class S, int NC, class Wt>
__device__ __forceinline__ void site_param_adjoint(const PackView<S, NC> &v, const PackParams<S, NC> &pp, const Wt &w,
                                                   int thin_film, S &h, S &eta, S &gamma)
{
    using K = Pk<S, NC>;
    constexpr bool ones = Wt::interior;
    if constexpr (NC == 2) {
        const S x1 = K::template lane<0>(v.px[1][1]), y1 = K::template lane<0>(v.py[1][1]);
        const S x2 = K::template lane<1>(v.px[1][1]), y2 = K::template lane<1>(v.py[1][1]);
        const S R = fma1(y1, y2, x1 * x2), r1 = fma1(y1, y1, x1 * x1), r2 = fma1(y2, y2, x2 * x2);
        eta = ones ? eta + R : fma1(S(w.area), R, eta);
        gamma = fma1(ones ? r1 : S(w.area) * r1, r2, gamma);
    }
    if (!thin_film) {
        const Curl<S> c(v.a);
        const S nh = -pp.h;
        if constexpr (ones) {   // the four views add up to twice the central differences
            const S d = (c.yp + c.ym) - (c.xp + c.xm);
            h = h + fma1(S(2.0f) * pp.idx, d, S(4.0f) * nh);
        } else {
            h = fma1(S(w.vUR), fma1(pp.idx, c.yp - c.xp, nh), h);
            h = fma1(S(w.vUL), fma1(pp.idx, c.ym - c.xp, nh), h);
            h = fma1(S(w.vLL), fma1(pp.idx, c.ym - c.xm, nh), h);
            h = fma1(S(w.vLR), fma1(pp.idx, c.yp - c.xm, nh), h);
        }
    }
}

// ---------------------------------------------------------------- gradient
// (h + h_neighbour) dx towards the upper, lower, right and left neighbour.
template <class S>
struct FieldSums {
    S u, d, r, l;
};

// a - 2 b
__device__ __forceinline__ float sub_twice(float a, float b) { return __fmaf_rn(-2.0f, b, a); }
__device__ __forceinline__ double sub_twice(double a, double b) { return __fma_rn(-2.0, b, a); }
__device__ __forceinline__ ff sub_twice(ff a, ff b) { return a - ff(b.hi + b.hi, b.lo + b.lo); }

// What a walk down a column hands from row to row: of the y-link below the
// row (from row j - 1 to row j) its pull on the upper site and its current,
// without the mass; of the magnetic views below it the sums and differences
// that both rows read, without the field.
template <class S, int NC>
struct GradCarry {
    pack_t<S, NC> tx, ty, cr;
    S s1, s2, ey, ql, qr, ex, exm;
};

// A row of the window as the gradient reads it: A and psi of the column, A of
// the columns left and right of it.
template <class S, int NC>
struct GradView {
    vec2_t<S> a, al, ar;
    pack_t<S, NC> x, y;
};

// The upper side of row c (the carry into the row above, u): its y-link and
// magnetic views.  wy: weight of the link.
template <class S, int NC>
__device__ __forceinline__ void grad_up(const GradView<S, NC> &c, const GradView<S, NC> &u, const PackParams<S, NC> &pp,
                                        S wy, S ex0, S exm0, GradCarry<S, NC> &k)
{
    using K = Pk<S, NC>;
    using P = pack_t<S, NC>;
    const P w = K::bc(wy), dx = psub(u.x, c.x), dy = psub(u.y, c.y), sf = pmul(pp.hqd, K::bc(c.a.y + u.a.y));
    k.tx = pmul(w, pfma(sf, c.y, dx));
    k.ty = pmul(w, pnfma(sf, c.x, dy));
    k.cr = pmul(w, pnfma(c.x, dy, pmul(c.y, dx)));
    const S ey0 = u.a.x - c.a.x, eyr = u.ar.x - c.ar.x, eyl = u.al.x - c.al.x;
    k.ex = u.ar.y - u.a.y;
    k.exm = u.a.y - u.al.y;
    k.s1 = ex0 + k.ex;
    k.s2 = exm0 + k.exm;
    k.ey = ey0;
    k.qr = ey0 + eyr;
    k.ql = ey0 + eyl;
}

// Gradient dF/dA (out[0..1]) and dF/dpsi_c (out[2 + 2c..]) at one site of row c
// with the row u above it, restating gradientPsi (nlcg.cu:504-744) and
// gradientA (nlcg.cu:746-888).  Both link ends use the mass of this site, as
// the reference does.  xl, yl, xr, yr: psi of the columns left and right.  k:
// the carry from the row below, replaced by the one into the row above.  W:
// Wts or Ones.  per_site: the sums of h differ.
template <class S, int NC, class W>
__device__ __forceinline__ void site_gradient(const GradView<S, NC> &c, const GradView<S, NC> &u,
                                              const pack_t<S, NC> &xl, const pack_t<S, NC> &yl,
                                              const pack_t<S, NC> &xr, const pack_t<S, NC> &yr,
                                              const PackParams<S, NC> &pp, const W &w, const FieldSums<S> &h,
                                              int per_site, int maxwell, int thin_film, GradCarry<S, NC> &k, S *out)
{
    using K = Pk<S, NC>;
    using P = pack_t<S, NC>;
    constexpr bool ones = W::interior;
    const P X = c.x, Y = c.y;
    const P r2 = pfma(Y, Y, pmul(X, X));
    const P m2r = ones ? padd(r2, r2) : pmul(r2, K::bc(S(-2.0f)));
    P gx, gy, dg, ga0, ga1, ax, ay, Wx, Wy;
    {   // x-links; weights -2 w / (2 m) of the forward and backward one
        const P f = ones ? pp.n2hmx : pmul(pp.n2hmx, K::bc(S(w.wfx)));
        const P b = ones ? pp.n2hmx : pmul(pp.n2hmx, K::bc(S(w.wbx)));
        const P dxf = psub(xr, X), dyf = psub(yr, Y), dxb = psub(xl, X), dyb = psub(yl, Y);
        const P sf = pmul(pp.hqd, K::bc(c.a.x + c.ar.x)), sb = pmul(pp.nhqd, K::bc(c.a.x + c.al.x));
        gx = pfma(b, pfma(sb, yl, dxb), pmul(f, pfma(sf, yr, dxf)));
        gy = pfma(b, pnfma(sb, xl, dyb), pmul(f, pnfma(sf, xr, dyf)));
        // site term a^2 psi of both links, and the current through them
        if constexpr (ones) {   // without the constants that weights of 2 leave (2 FP64 steps of 256^2 x 64: 7.59 -> 7.51 ms)
            ax = pmul(pp.qd, K::bc(c.a.x));
            Wx = pmul(pp.n2hmx, ax);
        } else {
            ax = pmul(pp.nhqd, K::bc(c.a.x));                                // -a / 2
            Wx = pmul(pmul(pp.n2hmx, K::bc(S(w.wsx))), ax);                  // W a
            dg = pmul(Wx, ax);                                               // -W a^2 / 2
        }
        const P cu = pfma(f, pnfma(X, dyf, pmul(Y, dxf)), pmul(Wx, m2r));
        ga0 = pnfma(b, pnfma(X, dyb, pmul(Y, dxb)), cu);
    }
    const P cr_below = k.cr;
    {   // y-links: the one above, and the carried pull of the one below
        const P dx = psub(u.x, X), dy = psub(u.y, Y), sf = pmul(pp.hqd, K::bc(c.a.y + u.a.y));
        const P f = ones ? pp.n2hmy : pmul(pp.n2hmy, K::bc(S(w.wfy)));
        gx = pfma(f, pfma(sf, u.y, dx), pnfma(pp.n2hmy, k.tx, gx));
        gy = pfma(f, pnfma(sf, u.x, dy), pnfma(pp.n2hmy, k.ty, gy));
        const P tx = pfma(sf, Y, dx), ty = pnfma(sf, X, dy), cr = pnfma(X, dy, pmul(Y, dx));
        const P wf = K::bc(S(w.wfy));
        k.tx = ones ? tx : pmul(wf, tx);
        k.ty = ones ? ty : pmul(wf, ty);
        k.cr = ones ? cr : pmul(wf, cr);
        if constexpr (ones) {
            ay = pmul(pp.qd, K::bc(c.a.y));
            Wy = pmul(pp.n2hmy, ay);
        } else {
            ay = pmul(pp.nhqd, K::bc(c.a.y));
            Wy = pmul(pmul(pp.n2hmy, K::bc(S(w.wsy))), ay);
            dg = pfma(Wy, ay, dg);
        }
        ga1 = pfma(pp.n2hmy, padd(k.cr, cr_below), pmul(Wy, m2r));
    }
    const S g0 = K::sum(pmul(pp.nhqd, ga0)), g1 = K::sum(pmul(pp.nhqd, ga1));
    // condensation: 2 psi (a + b |psi|^2); density coupling with the other component
    P kk = pfma(pp.b2, r2, pp.a2);
    const P m2 = K::bc(S(-2.0f));
    if constexpr (NC == 2) {
        const S x1 = K::template lane<0>(X), y1 = K::template lane<0>(Y);
        const S x2 = K::template lane<1>(X), y2 = K::template lane<1>(Y);
        kk = pfma(K::bc(pp.gammad), K::mk(K::template lane<1>(r2), K::template lane<0>(r2)), kk);
        kk = ones ? pnfma(Wy, ay, pnfma(Wx, ax, kk)) : pfma(kk, K::bc(S(w.area)), pmul(dg, m2));
        gx = pfma(kk, X, gx);
        gy = pfma(kk, Y, gy);
        // eta psi_2 + delta (psi_1* psi_2) psi_2-like terms: e = eta + delta R, i = delta I
        const S R = fma1(y1, y2, x1 * x2), I = fma1(x1, y2, -(y1 * x2));
        S e = fma1(pp.deltad, R, pp.etad), i = pp.deltad * I;
        if (!ones) {
            e = e * S(w.area);
            i = i * S(w.area);
        }
        out[2] = fma1(-i, y2, fma1(e, x2, K::template lane<0>(gx)));
        out[3] = fma1(i, x2, fma1(e, y2, K::template lane<0>(gy)));
        out[4] = fma1(i, y1, fma1(e, x1, K::template lane<1>(gx)));
        out[5] = fma1(-i, x1, fma1(e, y1, K::template lane<1>(gy)));
    } else {
        kk = ones ? pnfma(Wy, ay, pnfma(Wx, ax, kk)) : pfma(kk, K::bc(S(w.area)), pmul(dg, m2));
        out[2] = pfma(kk, X, gx);
        out[3] = pfma(kk, Y, gy);
    }
    if (maxwell)
#pragma unroll
        for (int q = 2; q < 2 + 2 * NC; ++q) out[q] = S(0.0f);
    // magnetic views of this site and the neighbours' views of the same plaquettes
    // (nlcg.cu:852-883), from the link differences ex(i,j) = A_y(i+1,j) - A_y(i,j)
    // and ey(i,j) = A_x(i,j+1) - A_x(i,j); the lower side comes with the carry.  The
    // views' fields are left out and added up by themselves: a uniform one cancels
    // between the sides of a site whose views are all there, and a view that holds
    // it rounds at its size, not at the curl's (512^2 x 16 in FP64: dF/dA 1.11e-15
    // from 64 bits with the field in the views, 8.0e-16 this way; A after four
    // float-float steps of 256^2 x 64: 7.6e-15, 3.7e-15)
    const S s3 = k.s2, s4 = k.s1, eyd = k.ey, ql = k.ql, qr = k.qr, ex0 = k.ex, exm = k.exm, two = S(2.0f);
    {
        const S ey0 = u.a.x - c.a.x, eyr = u.ar.x - c.ar.x, eyl = u.al.x - c.al.x;
        k.ex = u.ar.y - u.a.y;
        k.exm = u.a.y - u.al.y;
        k.s1 = ex0 + k.ex;
        k.s2 = exm + k.exm;
        k.ey = ey0;
        k.qr = ey0 + eyr;
        k.ql = ey0 + eyl;
    }
    if (!thin_film) {
        S mx, my;
        if constexpr (ones) {
            mx = fma1(S(4.0f), eyd - k.ey, (k.s1 + k.s2) - (s3 + s4));
            my = fma1(S(4.0f), exm - ex0, (k.qr + qr) - (k.ql + ql));
            if (per_site) {
                mx = fma1(two, h.d - h.u, mx);
                my = fma1(two, h.r - h.l, my);
            }
        } else {
            if (per_site) {
                mx = fma1(S(w.vLL) + S(w.vLR), h.d, -((S(w.vUR) + S(w.vUL)) * h.u));
                my = fma1(S(w.vUR) + S(w.vLR), h.r, -((S(w.vUL) + S(w.vLL)) * h.l));
            } else {
                mx = S(w.vdx) * h.u;
                my = S(w.vdy) * h.u;
            }
            mx = fma1(S(w.vUR), sub_twice(k.s1, k.ey), mx);
            mx = fma1(S(w.vUL), sub_twice(k.s2, k.ey), mx);
            mx = fma1(S(w.vLL), -sub_twice(s3, eyd), mx);
            mx = fma1(S(w.vLR), -sub_twice(s4, eyd), mx);
            my = fma1(S(w.vUR), sub_twice(k.qr, ex0), my);
            my = fma1(S(w.vUL), -sub_twice(k.ql, exm), my);
            my = fma1(S(w.vLL), -sub_twice(ql, exm), my);
            my = fma1(S(w.vLR), sub_twice(qr, ex0), my);
        }
        out[0] = fma1(S(0.25f), mx, g0);
        out[1] = fma1(S(0.25f), my, g1);
    } else {
        out[0] = S(0.0f);
        out[1] = S(0.0f);
    }
}

// ------------------------------------------------------------ line quartic
// Sums of the coefficients {A, B, C, D, E} of F(x + t d): per-component packs,
// scalars, and the magnetic sums with their factors outside.
template <class S, int NC>
struct PolySum {
    // FP64 rows of interior sites: the links' sums without their mass, per direction
    static constexpr int LINKS = std::is_same<S, double>::value ? 2 : 1;
    pack_t<S, NC> ka, kb, kc, kd, ke, la[LINKS], lb[LINKS], lc[LINKS], ld[LINKS];
    S e, b, c, d, e4, em0, em1, em2;
    __device__ __forceinline__ void zero()
    {
        ka = kb = kc = kd = ke = Pk<S, NC>::bc(S(0.0f));
#pragma unroll
        for (int q = 0; q < LINKS; ++q) la[q] = lb[q] = lc[q] = ld[q] = ka;
        e = b = c = d = e4 = em0 = em1 = em2 = S(0.0f);
    }
    __device__ __forceinline__ void total(const PackParams<S, NC> &pp, bool links, int compat, S (&o)[5])
    {
        using K = Pk<S, NC>;
        if constexpr (LINKS == 2) if (links) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const auto f = q == 0 ? pp.hmxi : pp.hmyi;
                ka = pfma(f, la[q], ka);
                kb = pfma(f, lb[q], kb);
                kc = pfma(f, lc[q], kc);
                kd = pfma(q == 1 && compat ? pmul(f, K::bc(S(0.5f))) : f, ld[q], kd);
            }
        }
        o[0] = fma1(S(0.125f), em0, e + K::sum(ka));
        o[1] = fma1(pp.idx4, em1, b + K::sum(kb));
        o[2] = fma1(pp.idx8, em2, c + K::sum(kc));
        o[3] = d + K::sum(kd);
        o[4] = e4 + K::sum(ke);
    }
};

// Adds the coefficients {A, B, C, D, E} of F(x + t d) at one site, without the
// common dx^2 (polynomialExpansion, nlcg.cu:997-1370).  compat keeps the reference's
// x-link first-order slip (its t-linear field term uses charge -1) and the
// halved cubic coefficient of the y-links, as corrections to the exact form.
template <class S, int NC, class Wt>
__device__ __forceinline__ void site_poly(const PackView<S, NC> &v, const PackView<S, NC> &dv,
                                          const PackParams<S, NC> &pp, const Wt &w, int per_site, int compat,
                                          int thin_film, PolySum<S, NC> &sum)
{
    constexpr bool ones = Wt::interior, bare = ones && !Wt::masses;
    constexpr int LINKS = PolySum<S, NC>::LINKS;
    using K = Pk<S, NC>;
    using P = pack_t<S, NC>;
    const S half = S(0.5f);
    const P X = v.px[1][1], Y = v.py[1][1], U = dv.px[1][1], Vd = dv.py[1][1];
    // |psi + t d|^2 = r0 + n1 t + n2 t^2 (rh = n1 / 2); n0 = a / b + r0
    const P r0 = pfma(Y, Y, pmul(X, X)), n0 = padd(r0, pp.aob);
    const P rh = pfma(Y, Vd, pmul(X, U)), n1 = padd(rh, rh);
    const P n2 = pfma(Vd, Vd, pmul(U, U));
    P w0, w1, w2, kd_y;   // site term (a + t b)^2 |psi + t d|^2 / 2 of the links: coefficients of its first factor
    P ka = sum.ka, kb = sum.kb, kc = sum.kc, kd = sum.kd;
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
        // forward link i -> j: i the site, j its +x (dir 0) or +y (dir 1) neighbour
        const S Ai = dir == 0 ? v.a[1][1].x : v.a[1][1].y, Aj = dir == 0 ? v.a[1][2].x : v.a[2][1].y;
        const S ai = dir == 0 ? dv.a[1][1].x : dv.a[1][1].y, aj = dir == 0 ? dv.a[1][2].x : dv.a[2][1].y;
        const P xj = dir == 0 ? v.px[1][2] : v.px[2][1], yj = dir == 0 ? v.py[1][2] : v.py[2][1];
        const P uj = dir == 0 ? dv.px[1][2] : dv.px[2][1], vj = dir == 0 ? dv.py[1][2] : dv.py[2][1];
        const P hm = dir == 0 ? pp.hmxi : pp.hmyi, hb = dir == 0 ? pp.hmxil : pp.hmyid;
        const S wf = S(dir == 0 ? w.wfx : w.wfy), wb = S(dir == 0 ? w.wbx : w.wby), ws = S(dir == 0 ? w.wsx : w.wsy);
        const P f = ones ? hm : pmul(hm, K::bc(wf));
        // half the weights (over m dx^2) of both links of this direction at the site
        const P W = per_site ? pmul(K::bc(half), pfma(hb, K::bc(wb), f))
                    : ones   ? hm
                             : pmul(dir == 0 ? pp.hhmx : pp.hhmy, K::bc(ws));
        const P a = pmul(pp.qd, K::bc(Ai)), b = pmul(pp.qd, K::bc(ai)), Wa = pmul(W, a), Wb = pmul(W, b);
        // Delta (Dy, Ey with the opposite sign), and Delta + s (y, x)
        const P Dx = psub(xj, X), Dy = psub(Y, yj), Ex = psub(uj, U), Ey = psub(Vd, vj);
        const P s0 = pmul(pp.qd, K::bc(Ai + Aj)), s1 = pmul(pp.qd, K::bc(ai + aj));
        const P P0 = pfma(s0, Y, Dx), P1 = pfma(s0, Vd, pfma(s1, Y, Ex)), P2 = pmul(s1, Vd);
        const P Q0 = pfma(s0, X, Dy), Q1 = pfma(s0, U, pfma(s1, X, Ey)), Q2 = pmul(s1, U);
        const P fDx = bare ? Dx : pmul(f, Dx), fDy = bare ? Dy : pmul(f, Dy);
        const P fEx = bare ? Ex : pmul(f, Ex), fEy = bare ? Ey : pmul(f, Ey);
        P &la = bare ? sum.la[dir % LINKS] : ka, &lb = bare ? sum.lb[dir % LINKS] : kb;
        P &lc = bare ? sum.lc[dir % LINKS] : kc, &ld = bare ? sum.ld[dir % LINKS] : kd;
        if (dir == 0) {
            w0 = pmul(Wa, a);
            w1 = pmul(Wa, b);
            w2 = pmul(Wb, b);
        } else {
            w0 = pfma(Wa, a, w0);
            w1 = pfma(Wa, b, w1);
            w2 = pfma(Wb, b, w2);
        }
        la = pfma(fDx, P0, la);
        lb = pfma(fEx, P0, pfma(fDx, P1, lb));
        lc = pfma(fEx, P1, pfma(fDx, P2, lc));
        ld = pfma(fEx, P2, ld);
        la = pfma(fDy, Q0, la);
        lb = pfma(fEy, Q0, pfma(fDy, Q1, lb));
        lc = pfma(fEy, Q1, pfma(fDy, Q2, lc));
        ld = pfma(fEy, Q2, ld);
        if (compat) {
            if (dir == 0) {
                // t1 carries charge -1 instead of q in its field term: t1 += e, e_k = (q + 1) dx a psi;
                // B += t0.e, C += t1.e + e.e / 2, D += e.t2
                const P ci = pmul(pp.kq, K::bc(ai)), cj = pmul(pp.kq, K::bc(aj));
                const P Qj = pmul(pp.qd, K::bc(Aj)), qj = pmul(pp.qd, K::bc(aj));
                const P rj = pfma(yj, yj, pmul(xj, xj)), rhj = pfma(yj, vj, pmul(xj, uj));
                const P nK0 = pfma(X, Dy, pmul(Y, Dx));                 // -(x Dy - y Dx)
                const P ti = padd(nK0, pmul(a, r0)), tj = padd(nK0, pmul(Qj, rj));
                kb = pnfma(f, pfma(cj, tj, pmul(ci, ti)), kb);
                const P si = pfma(b, r0, pfma(a, rh, pfma(X, Ey, pmul(Y, Ex))));
                const P sj = pfma(qj, rj, pfma(Qj, rhj, pfma(xj, Ey, pmul(yj, Ex))));
                kc = pnfma(f, pfma(cj, sj, pmul(ci, si)), kc);
                const P ee = pfma(pmul(cj, cj), rj, pmul(pmul(ci, ci), r0));
                kc = pfma(pmul(f, K::bc(half)), ee, kc);
                kd = pnfma(f, pfma(cj, pmul(qj, rhj), pmul(ci, pmul(b, rh))), kd);
            } else {
                const P ab = pmul(Wa, b);
                kd_y = pfma(n2, padd(ab, ab), pmul(n1, pmul(Wb, b)));
                if (!bare) kd_y = pfma(fEx, P2, pfma(fEy, Q2, kd_y));
            }
        }
    }
    w1 = padd(w1, w1);
    // condensation b/2 (n0 + n1 t + n2 t^2)^2 and the site terms
    const P bA = ones ? pp.b : pmul(pp.b, K::bc(S(w.area))), bh = pmul(bA, K::bc(half));
    const P U0 = pfma(bA, n0, w0), U1 = pfma(bA, n1, w1), V1 = pfma(bh, n1, w1), U2 = pfma(bh, n2, w2);
    sum.ka = pfma(w0, r0, pfma(pmul(bh, n0), n0, ka));
    sum.kb = pfma(w1, r0, pfma(n1, U0, kb));
    sum.kc = pfma(w2, r0, pfma(n1, V1, pfma(n2, U0, kc)));
    kd = pfma(w2, n1, pfma(n2, U1, kd));
    if (compat) kd = pnfma(kd_y, K::bc(half), kd);
    sum.kd = kd;
    sum.ke = pfma(n2, U2, sum.ke);
    if constexpr (NC == 2) {   // couplings between the components
        const S x1 = K::template lane<0>(X), y1 = K::template lane<0>(Y), x2 = K::template lane<1>(X), y2 = K::template lane<1>(Y);
        const S u1 = K::template lane<0>(U), v1 = K::template lane<0>(Vd), u2 = K::template lane<1>(U), v2 = K::template lane<1>(Vd);
        const S R0 = fma1(y1, y2, x1 * x2), R2 = fma1(v1, v2, u1 * u2);
        const S R1 = fma1(y1, v2, fma1(x1, u2, fma1(v1, y2, u1 * x2)));
        S e = sum.e, b1 = sum.b, c2 = sum.c, d3 = sum.d, e4 = sum.e4;
        const S ea = ones ? pp.eta : pp.eta * S(w.area);
        e = fma1(ea, R0, e);
        b1 = fma1(ea, R1, b1);
        c2 = fma1(ea, R2, c2);
        const S ga = ones ? half * pp.gamma : half * pp.gamma * S(w.area);
        const S g0 = ga * K::template lane<0>(r0), g1 = ga * K::template lane<0>(n1), g2 = ga * K::template lane<0>(n2);
        const S s0 = K::template lane<1>(r0), s1 = K::template lane<1>(n1), s2 = K::template lane<1>(n2);
        e = fma1(g0, s0, e);
        b1 = fma1(g1, s0, fma1(g0, s1, b1));
        c2 = fma1(g2, s0, fma1(g1, s1, fma1(g0, s2, c2)));
        d3 = fma1(g2, s1, fma1(g1, s2, d3));
        e4 = fma1(g2, s2, e4);
        if (!SkipZeroDelta<S>::v || pp.delta != S(0.0f)) {
            const S I0 = fma1(x1, y2, -(y1 * x2)), I2 = fma1(u1, v2, -(v1 * u2));
            const S I1 = fma1(-v1, x2, fma1(-y1, u2, fma1(u1, y2, x1 * v2)));
            const S d2 = ones ? pp.delta : pp.delta * S(w.area), da = half * d2;
            e = fma1(da, fma1(R0, R0, -(I0 * I0)), e);
            b1 = fma1(d2, fma1(R1, R0, -(I1 * I0)), b1);
            c2 = fma1(da, fma1(R1, R1, -(I1 * I1)), c2);
            c2 = fma1(d2, fma1(R0, R2, -(I0 * I2)), c2);
            d3 = fma1(d2, fma1(R1, R2, -(I1 * I2)), d3);
            e4 = fma1(da, fma1(R2, R2, -(I2 * I2)), e4);
        }
        sum.e = e;
        sum.b = b1;
        sum.c = c2;
        sum.d = d3;
        sum.e4 = e4;
    }
    if (!thin_film) {
        Curl<S> c(v.a), q(dv.a);
        c.field(pp.hl);
        const S nh = -pp.h;
        S em0 = sum.em0, em1 = sum.em1, em2 = sum.em2;
#define EMV(wv, yy, xx, dyy, dxx)                                                                        \
    {                                                                                                    \
        const S m0 = fma1(pp.idx, yy - xx, nh), m1 = dyy - dxx;                                          \
        const S z0 = ones ? m0 : S(wv) * m0, z1 = ones ? m1 : S(wv) * m1;                                \
        em0 = fma1(z0, m0, em0);                                                                         \
        em1 = fma1(z0, m1, em1);                                                                         \
        em2 = fma1(z1, m1, em2);                                                                         \
    }
        EMV(w.vUR, c.yp, c.xp, q.yp, q.xp)
        EMV(w.vUL, c.ym, c.xp, q.ym, q.xp)
        EMV(w.vLL, c.ym, c.xm, q.ym, q.xm)
        EMV(w.vLR, c.yp, c.xm, q.yp, q.xm)
#undef EMV
        sum.em0 = em0;
        sum.em1 = em1;
        sum.em2 = em2;
    }
}

// B at one site: mean of the views inside the domain.
template <class S, class Wt>
__device__ __forceinline__ S site_b(const vec2_t<S> (&a)[3][3], S idx, const Wt &w)
{
    const Curl<S> c(a);
    if constexpr (Wt::interior) {
        return ((c.yp + c.ym) - (c.xp + c.xm)) * (S(0.5f) * idx);
    } else {
        S b = S(w.vUR) * (c.yp - c.xp);
        b = fma1(S(w.vUL), c.ym - c.xp, b);
        b = fma1(S(w.vLL), c.ym - c.xm, b);
        b = fma1(S(w.vLR), c.yp - c.xm, b);
        return b * idx * S(w.ivs);
    }
}

// B and J at one site (computeJBKernel, nlcg.cu:243-364).
template <class S, int NC, class Wt>
__device__ __forceinline__ void site_jb(const PackView<S, NC> &v, const PackParams<S, NC> &pp, const Wt &w,
                                        S *out /* 1+2NC */)
{
    using K = Pk<S, NC>;
    using P = pack_t<S, NC>;
    constexpr bool ones = Wt::interior;
    out[0] = site_b<S>(v.a, pp.idx, w);
    const P X = v.px[1][1], Y = v.py[1][1];
    const P nqr = pmul(pmul(pp.nhqd, K::bc(S(2.0f))), pfma(Y, Y, pmul(X, X)));   // -q dx |psi|^2
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
        const S A = dir == 0 ? v.a[1][1].x : v.a[1][1].y;
        const P xf = dir == 0 ? v.px[1][2] : v.px[2][1], yf = dir == 0 ? v.py[1][2] : v.py[2][1];
        const P xb = dir == 0 ? v.px[1][0] : v.px[0][1], yb = dir == 0 ? v.py[1][0] : v.py[0][1];
        // lattice current of each link: x Dy - y Dx - a |psi|^2
        const P nar = pmul(nqr, K::bc(A));
        P j;
        if constexpr (ones) {
            j = pnfma(Y, psub(xf, xb), pfma(X, psub(yf, yb), padd(nar, nar)));
        } else {
            const P jf = pnfma(Y, psub(xf, X), pfma(X, psub(yf, Y), nar));
            const P jb = pnfma(Y, psub(X, xb), pfma(X, psub(Y, yb), nar));
            j = pfma(K::bc(S(dir == 0 ? w.lbx : w.lby)), jb, pmul(K::bc(S(dir == 0 ? w.lfx : w.lfy)), jf));
        }
        j = pmul(dir == 0 ? pp.jmx : pp.jmy, j);
        out[1 + dir] = K::template lane<0>(j);
        if (NC == 2) out[3 + dir] = K::template lane<1>(j);
    }
}

}  // namespace mepgl
