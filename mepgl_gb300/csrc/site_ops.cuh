// site_ops.cuh -- what the per-site stencils share: mask weights and site
// parameters; and the gauge-link functional, which has no packed form.
//
// The discretisation is the reference's (mepgl/src/nlcg.cu): psi and A live
// on sites; on a link i -> j along e the kinetic term uses the linearised
// covariant differences
//   u0 = -(Re psi_j - Re psi_i)/dx - q A_i,e Im psi_i   (u1: A_j, psi_j)
//   v0 = +(Im psi_j - Im psi_i)/dx - q A_i,e Re psi_i   (v1: A_j, psi_j)
// with energy (u0^2 + u1^2 + v0^2 + v1^2) / (4 m) times the fraction of the
// two superconducting plaquettes sharing the link; the magnetic term takes,
// at every site, four collocated views of curl A - h (forward/backward
// differences of A_y along x and of A_x along y), each weighted 1/8 when the
// plaquette is inside the computational domain.
//
// Domain handling is branchless: every link / plaquette term is multiplied
// by a weight that is zero when the reference would skip it.  The weights
// of a site come from two constant tables indexed by its 8-bit neighbour
// codes (bit order 0:+x 1:+x+y 2:+y 3:-x+y 4:-x 5:-x-y 6:-y 7:+x-y,
// nlcg.cu:48-103), so no bit arithmetic or int->float conversion runs per
// site.  Outside-lattice halo values are zero, so masked terms are finite.
#pragma once

#include "common.cuh"

namespace mepgl {

// Weights of a superconducting code: area fraction, link weights (forward
// x, backward x, forward y, backward y; zero when the link is absent), and
// the bare link bits (used by J).  Of a computational code: the validity
// (0/1) of the four curl views UR, UL, LL, LR.
template <class T>
struct MaskTable {
    T sc[256][12];    // area, wfx, wbx, wfy, wby, lfx, lbx, lfy, lby, wfx + wbx, wfy + wby, 0
    T cc[256][8];     // vUR, vUL, vLL, vLR, 1 / their sum, lower minus upper ones, right minus left ones, 0
};
// Defined here: kernels.cu is the only translation unit that includes this file.
__constant__ MaskTable<float> c_mask_f;
__constant__ MaskTable<double> c_mask_d;

template <class T> __device__ __forceinline__ const MaskTable<T> &mask_table();
template <> __device__ __forceinline__ const MaskTable<float> &mask_table<float>() { return c_mask_f; }
template <> __device__ __forceinline__ const MaskTable<double> &mask_table<double>() { return c_mask_d; }
// the weights are multiples of 1/4, exact in float: float-float reads the float table
template <class T> struct MaskOf { using type = T; };
template <> struct MaskOf<ff> { using type = float; };

template <class T>
struct Wts {
    static constexpr bool interior = false, masses = true;
    T area, wfx, wbx, wfy, wby, lfx, lbx, lfy, lby, wsx, wsy;
    T vUR, vUL, vLL, vLR, ivs, vdx, vdy;
    __device__ __forceinline__ void load(unsigned mk)
    {
        const auto &M = mask_table<typename MaskOf<T>::type>();
        const unsigned s = mk >> 8, c = mk & 0xffu;
        area = M.sc[s][0]; wfx = M.sc[s][1]; wbx = M.sc[s][2]; wfy = M.sc[s][3]; wby = M.sc[s][4];
        lfx = M.sc[s][5]; lbx = M.sc[s][6]; lfy = M.sc[s][7]; lby = M.sc[s][8];
        wsx = M.sc[s][9]; wsy = M.sc[s][10];
        vUR = M.cc[c][0]; vUL = M.cc[c][1]; vLL = M.cc[c][2]; vLR = M.cc[c][3]; ivs = M.cc[c][4];
        vdx = M.cc[c][5]; vdy = M.cc[c][6];
    }
};

// Host-side construction of the tables (same arithmetic as nlcg.cu:522-525,
// 186-187, 533-609 etc.: weights are exact multiples of 1/4).
template <class T>
inline void build_mask_table(MaskTable<T> &M)
{
    for (unsigned k = 0; k < 256; ++k) {
        auto b = [&](int n) { return (int)((k >> n) & 1u); };
        M.sc[k][0] = (T)(b(0) * b(1) * b(2) + b(2) * b(3) * b(4) + b(4) * b(5) * b(6) + b(6) * b(7) * b(0)) / (T)4;
        M.sc[k][1] = b(0) ? (T)(b(1) * b(2) + b(6) * b(7)) / (T)2 : (T)0;
        M.sc[k][2] = b(4) ? (T)(b(2) * b(3) + b(5) * b(6)) / (T)2 : (T)0;
        M.sc[k][3] = b(2) ? (T)(b(0) * b(1) + b(3) * b(4)) / (T)2 : (T)0;
        M.sc[k][4] = b(6) ? (T)(b(4) * b(5) + b(7) * b(0)) / (T)2 : (T)0;
        M.sc[k][5] = (T)b(0);
        M.sc[k][6] = (T)b(4);
        M.sc[k][7] = (T)b(2);
        M.sc[k][8] = (T)b(6);
        M.sc[k][9] = M.sc[k][1] + M.sc[k][2];
        M.sc[k][10] = M.sc[k][3] + M.sc[k][4];
        M.sc[k][11] = (T)0;
        M.cc[k][0] = (T)(b(0) & b(1) & b(2));
        M.cc[k][1] = (T)(b(2) & b(3) & b(4));
        M.cc[k][2] = (T)(b(4) & b(5) & b(6));
        M.cc[k][3] = (T)(b(6) & b(7) & b(0));
        const T v = M.cc[k][0] + M.cc[k][1] + M.cc[k][2] + M.cc[k][3];
        M.cc[k][4] = v > (T)0 ? (T)1 / v : (T)0;
        M.cc[k][5] = (M.cc[k][2] + M.cc[k][3]) - (M.cc[k][0] + M.cc[k][1]);
        M.cc[k][6] = (M.cc[k][0] + M.cc[k][3]) - (M.cc[k][1] + M.cc[k][2]);
        M.cc[k][7] = (T)0;
    }
}

// Parameters of one site (uniform strings read the descriptor).
template <class T>
struct SiteParams {
    T a[2], b[2], hmx[2], hmy[2], aob[2];  // hmx = 0.5 / m_xx
    T q[2], eta, gamma, delta, h, idx, dx2, dx;
    __device__ __forceinline__ void load_uniform(const StringDesc &S)
    {
        const Uniform<T> &U = S.template u<T>();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            a[c] = U.a[c]; b[c] = U.b[c]; hmx[c] = U.hmx[c]; hmy[c] = U.hmy[c]; aob[c] = U.aob[c]; q[c] = U.q[c];
        }
        eta = U.eta; gamma = U.gamma; delta = U.delta; h = U.h; idx = U.idx; dx2 = U.dx2; dx = U.dx;
    }
    // per-site overrides (strings whose parameter arrays are not uniform)
    __device__ __forceinline__ void load_site(const StringDesc &S, int s, int nc)
    {
        using St = store_t<T>;
        for (int c = 0; c < nc; ++c) {
            const St av = static_cast<const St *>(S.pa[c])[s], bv = static_cast<const St *>(S.pb[c])[s];
            a[c] = from_store<T>(av);
            b[c] = from_store<T>(bv);
            hmx[c] = from_store<T>((St)0.5 / static_cast<const St *>(S.pmxx[c])[s]);
            hmy[c] = from_store<T>((St)0.5 / static_cast<const St *>(S.pmyy[c])[s]);
            aob[c] = from_store<T>(av / bv);
        }
        h = from_store<T>(static_cast<const St *>(S.ph)[s]);
    }
};

#define TA(dx_, dy_) (t.A((dx_), (dy_)))
#define TP(c_, dx_, dy_) (t.P((c_), (dx_), (dy_)))

// ------------------------------------------------------- gauge links
// The link (Peierls) discretisation of the same functional (no reference
// counterpart): A_e at a site is the variable of the link to its +e
// neighbour; per link and component the kinetic energy is
// w_e / (2 m_e) |psi_t - U psi_s|^2 with U = exp(i q A_e dx); per plaquette
// (lower-left corner s) 1/2 v_UR (B - h)^2 dx^2 with
// B = (A_x(s) + A_y(s+x) - A_x(s+y) - A_y(s)) / dx.  Exactly invariant under
// psi -> psi e^{i q chi}, A_e(s) -> A_e(s) + (chi(s+e) - chi(s)) / dx.
template <class T> __device__ __forceinline__ void cis(T a, T &c, T &s);
template <> __device__ __forceinline__ void cis<float>(float a, float &c, float &s) { sincosf(a, &s, &c); }
template <> __device__ __forceinline__ void cis<double>(double a, double &c, double &s) { sincos(a, &s, &c); }

template <class T>
__device__ __forceinline__ T cond_density(const vec2_t<T> *P, int nc, const SiteParams<T> &p)
{
    T nl = 0;
    for (int c = 0; c < nc; ++c) {
        const T r = p.aob[c] + P[c].x * P[c].x + P[c].y * P[c].y;
        nl += p.b[c] * (T)0.5 * r * r;
    }
    if (nc == 2) {
        const T R = P[0].x * P[1].x + P[0].y * P[1].y, I = P[0].x * P[1].y - P[0].y * P[1].x;
        nl += p.eta * R + p.gamma * (T)0.5 * (P[0].x * P[0].x + P[0].y * P[0].y) * (P[1].x * P[1].x + P[1].y * P[1].y)
            + p.delta * (T)0.5 * (R * R - I * I);
    }
    return nl;
}

template <class T, int NC, class View>
__device__ __forceinline__ T site_energy_link(const View &t, const SiteParams<T> &p,
                                              const Wts<T> &w, int thin_film)
{
    vec2_t<T> P0[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) P0[c] = TP(c, 0, 0);
    const T nl = cond_density<T>(P0, NC, p);
    T kin = 0;
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
        const int ox = dir == 0 ? 1 : 0, oy = 1 - ox;
        const T Ae = dir == 0 ? TA(0, 0).x : TA(0, 0).y, wl = dir == 0 ? w.wfx : w.wfy;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            T cu, su;
            cis<T>(p.q[c] * Ae * p.dx, cu, su);
            const vec2_t<T> ps = P0[c], pt = TP(c, ox, oy);
            const T zr = pt.x - (cu * ps.x - su * ps.y), zi = pt.y - (su * ps.x + cu * ps.y);
            kin += wl * (dir == 0 ? p.hmx[c] : p.hmy[c]) * (zr * zr + zi * zi);
        }
    }
    T em = 0;
    if (!thin_film) {
        const T B = (TA(0, 0).x + TA(1, 0).y - TA(0, 1).x - TA(0, 0).y) * p.idx - p.h;
        em = (T)0.5 * w.vUR * B * B;
    }
    return kin + (nl * w.area + em) * p.dx2;
}

// Gradient of the link functional at one site (gather form): its own
// forward links, the backward links owned by its -x / -y neighbours (whose
// masses are hmx_l / hmy_d = 1 / (2 m) there), and the plaquettes with
// lower-left corners s, s-x, s-y (applied fields h, hl, hd).
template <class T, int NC, class View>
__device__ __forceinline__ void site_gradient_link(const View &t, const SiteParams<T> &p,
                                                   const Wts<T> &w, T hl, T hd, const T *hmx_l, const T *hmy_d,
                                                   int maxwell, int thin_film, T *out)
{
#pragma unroll
    for (int k = 0; k < 2 + 2 * NC; ++k) out[k] = 0;
    const T ar = w.area * p.dx2;
    vec2_t<T> P0[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) P0[c] = TP(c, 0, 0);
    if (!maxwell) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const T x = P0[c].x, y = P0[c].y, r2 = x * x + y * y;
            out[2 + 2 * c] += (T)2 * x * (p.a[c] + p.b[c] * r2) * ar;
            out[3 + 2 * c] += (T)2 * y * (p.a[c] + p.b[c] * r2) * ar;
        }
        if (NC == 2) {
            const T x1 = P0[0].x, y1 = P0[0].y, x2 = P0[NC - 1].x, y2 = P0[NC - 1].y;
            const T R = x1 * x2 + y1 * y2, I = x1 * y2 - y1 * x2, r1 = x1 * x1 + y1 * y1, r2 = x2 * x2 + y2 * y2;
            out[2] += (p.eta * x2 + p.gamma * x1 * r2 + p.delta * (R * x2 - I * y2)) * ar;
            out[3] += (p.eta * y2 + p.gamma * y1 * r2 + p.delta * (R * y2 + I * x2)) * ar;
            out[2 + 2 * (NC - 1)] += (p.eta * x1 + p.gamma * x2 * r1 + p.delta * (R * x1 + I * y1)) * ar;
            out[3 + 2 * (NC - 1)] += (p.eta * y1 + p.gamma * y2 * r1 + p.delta * (R * y1 - I * x1)) * ar;
        }
    }
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
        const int ox = dir == 0 ? 1 : 0, oy = 1 - ox;
        const T Ae = dir == 0 ? TA(0, 0).x : TA(0, 0).y, wf = dir == 0 ? w.wfx : w.wfy;
        const T Ab = dir == 0 ? TA(-1, 0).x : TA(0, -1).y, wb = dir == 0 ? w.wbx : w.wby;
        T ga = 0;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const T q = p.q[c];
            // own forward link s -> s + e
            const T kf = wf * (dir == 0 ? p.hmx[c] : p.hmy[c]);
            T cu, su;
            cis<T>(q * Ae * p.dx, cu, su);
            const vec2_t<T> ps = P0[c], pt = TP(c, ox, oy);
            const T ur = cu * ps.x - su * ps.y, ui = su * ps.x + cu * ps.y;
            const T zr = pt.x - ur, zi = pt.y - ui;
            ga += (T)2 * kf * q * p.dx * (zr * ui - zi * ur);
            // backward link s - e -> s, owned by the neighbour
            const T kb = wb * (dir == 0 ? hmx_l[c] : hmy_d[c]);
            T cb, sb;
            cis<T>(q * Ab * p.dx, cb, sb);
            const vec2_t<T> pb = TP(c, -ox, -oy);
            const T br = ps.x - (cb * pb.x - sb * pb.y), bi = ps.y - (sb * pb.x + cb * pb.y);
            if (!maxwell) {
                out[2 + 2 * c] += (T)2 * kb * br - (T)2 * kf * (cu * zr + su * zi);
                out[3 + 2 * c] += (T)2 * kb * bi - (T)2 * kf * (cu * zi - su * zr);
            }
        }
        if (!thin_film) out[dir] += ga;
    }
    if (!thin_film) {
        const T r0 = w.vUR * ((TA(0, 0).x + TA(1, 0).y - TA(0, 1).x - TA(0, 0).y) * p.idx - p.h) * p.dx;
        const T rd = w.vLR * ((TA(0, -1).x + TA(1, -1).y - TA(0, 0).x - TA(0, -1).y) * p.idx - hd) * p.dx;
        const T rl = w.vUL * ((TA(-1, 0).x + TA(0, 0).y - TA(-1, 1).x - TA(-1, 0).y) * p.idx - hl) * p.dx;
        out[0] += r0 - rd;
        out[1] += rl - r0;
    }
}

// dF/dH of the link functional at one site: -v_UR (B - h) dx^2.
template <class T, int NC, class View>
__device__ __forceinline__ T site_dh_link(const View &t, const SiteParams<T> &p,
                                          const Wts<T> &w)
{
    return -w.vUR * ((TA(0, 0).x + TA(1, 0).y - TA(0, 1).x - TA(0, 0).y) * p.idx - p.h) * p.dx2;
}

#undef TA
#undef TP

}  // namespace mepgl
