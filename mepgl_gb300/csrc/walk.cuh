// walk.cuh -- kernels that read a string's fields and form something of every
// site: energies, parameter adjoints, gradients, B and J, flux.  Included by
// kernels.cu inside its anonymous namespace, after strip.cuh.
//
// Work is shared out as in the NLCG passes: a warp walks down the rows of one
// strip (32 columns of an image) with a three-row window in registers, the
// next row's loads in flight, x-neighbours by shuffles, halo columns by
// cp.async.  What is formed at a site is the operation's; its sums run over
// the strip and leave once, so an FP64 energy does not pay 5 to 15 FP64
// additions per 32 sites for the reduction tree (a 256-thread tile did), and
// rows of interior sites skip the weights.

// Sum over a strip of a lane's terms: in float for FP32, over eight rows at most
// (walk_rows), then in double.  No conversion before the strip's end: the three sums
// of the adjoints of 768 x 512 x 12 sites in FP32 took 85 us with one conversion each,
// 122 with two and an FP64 addition (three rows in flight).
template <class T>
struct RowSum {
    T v;
    __device__ __forceinline__ RowSum() : v((T)0) {}
    __device__ __forceinline__ double total() const { return (double)v; }
};

// strip_code, also of a descriptor that brings int32 codes instead of the mask
// (the allocation-free energy).
__device__ __forceinline__ uint16_t walk_code(const StringDesc &S, const StripLane &L, int j)
{
    if (S.mask) return strip_code(S, L, j);
    if (!(j >= 0 && j < S.ny && L.cok)) return 0;
    const int s = L.gi + S.nx * j;
    return (uint16_t)((S.code_comp[s] & 0xff) | ((S.code_sc[s] & 0xff) << 8));
}

// Where a lane is: image of the string, site and row of the strip.
struct WalkPos {
    int n, gi, j, s, r;
};

// Neighbourhood of a site as the gauge-link terms read it.
template <class T, int NC>
struct LinkView {
    const PackView<T, NC> &v;
    __device__ __forceinline__ vec2_t<T> A(int dx, int dy) const { return v.a[dy + 1][dx + 1]; }
    __device__ __forceinline__ vec2_t<T> P(int c, int dx, int dy) const
    {
        vec2_t<T> p;
        p.x = c == 0 ? Pk<T, NC>::template lane<0>(v.px[dy + 1][dx + 1]) : Pk<T, NC>::template lane<NC - 1>(v.px[dy + 1][dx + 1]);
        p.y = c == 0 ? Pk<T, NC>::template lane<0>(v.py[dy + 1][dx + 1]) : Pk<T, NC>::template lane<NC - 1>(v.py[dy + 1][dx + 1]);
        return p;
    }
};

template <class T>
__device__ __forceinline__ SiteParams<T> site_params(const StringDesc &S, int s, int nc)
{
    SiteParams<T> p;
    p.load_uniform(S);
    if (S.per_site) p.load_site(S, s, nc);
    return p;
}

// ------------------------------------------------------------- operations
// Free energy per image (computeFreeEnergy).
struct EnergyOp {
    static constexpr bool psi = true, field = false;
    double *out;
    template <class T, int NC>
    struct State {
        RowSum<T> e;
        template <class W>
        __device__ __forceinline__ void site(const EnergyOp &, const PackView<T, NC> &v, const StringDesc &S,
                                             PackParams<T, NC> &pp, const W &w, const WalkPos &q)
        {
            e.v += site_energy<T, NC>(v, pp, w, S.thin_film);
        }
        __device__ __forceinline__ void link(const EnergyOp &, const PackView<T, NC> &v, const StringDesc &S,
                                             PackParams<T, NC> &, const Wts<T> &w, const WalkPos &q)
        {
            e.v += site_energy_link<T, NC>(LinkView<T, NC>{v}, site_params<T>(S, q.s, NC), w, S.thin_film);
        }
        __device__ __forceinline__ void finish(const EnergyOp &op, const StringDesc &S, const Scalars &sc, int u, int n,
                                               int tpi, int img)
        {
            const double v[1] = {e.total()};
            double tot[1];
            if (finish_image_warp<1>(v, sc, u, n * tpi, tpi, tpi, img, tot) &&
                (threadIdx.x & 31) == 0)
                op.out[img] = S.disc ? tot[0] : tot[0] * S.ud.dx2;
        }
    };
};

// Sums of the parameter adjoints (site_param_adjoint).
template <class T, int NC>
struct AdjointSums {
    RowSum<T> h, eta, gamma;
    template <class W>
    __device__ __forceinline__ void site(const PackView<T, NC> &v, const StringDesc &S, const PackParams<T, NC> &pp,
                                         const W &w)
    {
        site_param_adjoint<T, NC>(v, pp, w, S.thin_film, h.v, eta.v, gamma.v);
    }
    __device__ __forceinline__ void link(const PackView<T, NC> &v, const StringDesc &S, PackParams<T, NC> &pp,
                                         const Wts<T> &w, const WalkPos &q)
    {
        site_param_adjoint<T, NC>(v, pp, w, 1, h.v, eta.v, gamma.v);
        if (!S.thin_film) h.v += site_dh_link<T, NC>(LinkView<T, NC>{v}, site_params<T>(S, q.s, NC), w);
    }
    // out[3 img + k] = dF/dH, dF/deta, dF/dgamma
    __device__ __forceinline__ void finish(double *out, const StringDesc &S, const Scalars &sc, int u, int n, int tpi, int img)
    {
        const double v[3] = {h.total(), eta.total(), gamma.total()};
        double tot[3];
        if (finish_image_warp<3>(v, sc, u, n * tpi, tpi, tpi, img, tot) &&
            (threadIdx.x & 31) == 0) {
            out[3 * img] = tot[0] * (S.disc ? 1.0 : -0.25 * S.ud.dx2);
            out[3 * img + 1] = tot[1] * S.ud.dx2;
            out[3 * img + 2] = tot[2] * (0.5 * S.ud.dx2);
        }
    }
};

struct AdjointOp {
    static constexpr bool psi = true, field = false;
    double *out;
    template <class T, int NC>
    struct State {
        AdjointSums<T, NC> a;
        template <class W>
        __device__ __forceinline__ void site(const AdjointOp &, const PackView<T, NC> &v, const StringDesc &S,
                                             PackParams<T, NC> &pp, const W &w, const WalkPos &)
        {
            a.site(v, S, pp, w);
        }
        __device__ __forceinline__ void link(const AdjointOp &, const PackView<T, NC> &v, const StringDesc &S,
                                             PackParams<T, NC> &pp, const Wts<T> &w, const WalkPos &q)
        {
            a.link(v, S, pp, w, q);
        }
        __device__ __forceinline__ void finish(const AdjointOp &op, const StringDesc &S, const Scalars &sc, int u, int n,
                                               int tpi, int img)
        {
            a.finish(op.out, S, sc, u, n, tpi, img);
        }
    };
};

// Gradient of every site into three arrays, each image's times weights[n]
// (null: 1); ADJ: the parameter adjoints from the same walk.  A backward pass
// wants all three; one launch and one wait instead of a gradient, a scaling of
// its arrays and a walk for the adjoints take energy and gradient of
// 512 x 512 x 16 in FP64 from 3.09 to 2.90 ms, and of 97 x 113 x 6 gauge links
// in FP32 from 0.78 to 0.65 ms.
template <bool ADJ>
struct GradientOp {
    static constexpr bool psi = true, field = true;
    void *p[3];
    int maxwell;
    const double *weights;
    double *adj;
    template <class T, int NC>
    struct State {
        GradCarry<T, NC> up;
        AdjointSums<T, NC> a;
        FieldSites<T> near;   // of a per-site string, loaded with the site's parameters
        __device__ __forceinline__ void ahead(const StringDesc &S, const WalkPos &q) { near.load(S, q.gi, q.j, q.s); }
        __device__ __forceinline__ void store(const GradientOp &op, const StringDesc &S, const T *g, const WalkPos &q) const
        {
            const size_t k = (size_t)q.n * S.nx * S.ny + q.s;
            T f = (T)1;
            if (op.weights) f = (T)(store_t<T>)op.weights[q.n];
#pragma unroll
            for (int c = 0; c < 1 + NC; ++c) {
                vec2_t<T> gv;
                gv.x = op.weights ? g[2 * c] * f : g[2 * c];
                gv.y = op.weights ? g[2 * c + 1] * f : g[2 * c + 1];
                store2<T>(static_cast<vec2_t<store_t<T>> *>(op.p[c]) + k, gv);
            }
        }
        template <class W>
        __device__ __forceinline__ void site(const GradientOp &op, const PackView<T, NC> &v, const StringDesc &S,
                                             PackParams<T, NC> &pp, const W &w, const WalkPos &q)
        {
            const FieldSums<T> h = field_sums(S, pp, near, q.gi, q.j, q.s);
            const GradView<T, NC> c{v.a[1][1], v.a[1][0], v.a[1][2], v.px[1][1], v.py[1][1]};
            const GradView<T, NC> u{v.a[2][1], v.a[2][0], v.a[2][2], v.px[2][1], v.py[2][1]};
            if (q.r == 0) {
                const GradView<T, NC> d{v.a[0][1], v.a[0][0], v.a[0][2], v.px[0][1], v.py[0][1]};
                grad_up<T, NC>(d, c, pp, T(w.wby), d.ar.y - d.a.y, d.a.y - d.al.y, up);
            }
            T g[2 + 2 * NC];
            site_gradient<T, NC>(c, u, v.px[1][0], v.py[1][0], v.px[1][2], v.py[1][2], pp, w, h, S.per_site, op.maxwell, S.thin_film,
                                 up, g);
            store(op, S, g, q);
            if constexpr (ADJ) a.site(v, S, pp, w);
        }
        __device__ __forceinline__ void link(const GradientOp &op, const PackView<T, NC> &v, const StringDesc &S,
                                             PackParams<T, NC> &pp, const Wts<T> &w, const WalkPos &q)
        {
            if constexpr (!std::is_same<T, ff>::value) {   // float-float: the reference form only
                const SiteParams<T> p = site_params<T>(S, q.s, NC);
                T hl = p.h, hd = p.h, hmx_l[2] = {p.hmx[0], p.hmx[1]}, hmy_d[2] = {p.hmy[0], p.hmy[1]};
                if (S.per_site) {
                    hl = static_cast<const T *>(S.ph)[q.s > 0 ? q.s - 1 : q.s];
                    hd = static_cast<const T *>(S.ph)[q.j > 0 ? q.s - S.nx : q.s];
                    for (int c = 0; c < NC; ++c) {
                        if (q.gi > 0) hmx_l[c] = (T)0.5 / static_cast<const T *>(S.pmxx[c])[q.s - 1];
                        if (q.j > 0) hmy_d[c] = (T)0.5 / static_cast<const T *>(S.pmyy[c])[q.s - S.nx];
                    }
                }
                T g[2 + 2 * NC];
                site_gradient_link<T, NC>(LinkView<T, NC>{v}, p, w, hl, hd, hmx_l, hmy_d, op.maxwell, S.thin_film, g);
                store(op, S, g, q);
                if constexpr (ADJ) a.link(v, S, pp, w, q);
            }
        }
        __device__ __forceinline__ void finish(const GradientOp &op, const StringDesc &S, const Scalars &sc, int u, int n,
                                               int tpi, int img)
        {
            if constexpr (ADJ) a.finish(op.adj, S, sc, u, n, tpi, img);
        }
    };
};

// B (reals) and J (pairs) of every site (computeJB).
struct JbOp {
    static constexpr bool psi = true, field = false;
    void *b, *j1, *j2;
    template <class T, int NC>
    struct State {
        template <class W>
        __device__ __forceinline__ void site(const JbOp &op, const PackView<T, NC> &v, const StringDesc &S,
                                             PackParams<T, NC> &pp, const W &w, const WalkPos &q)
        {
            T o[1 + 2 * NC];
            site_jb<T, NC>(v, pp, w, o);
            const size_t k = (size_t)q.n * S.nx * S.ny + q.s;
            static_cast<T *>(op.b)[k] = o[0];
            vec2_t<T> j;
            j.x = o[1];
            j.y = o[2];
            static_cast<vec2_t<T> *>(op.j1)[k] = j;
            if (NC == 2) {
                j.x = o[3];
                j.y = o[4];
                static_cast<vec2_t<T> *>(op.j2)[k] = j;
            }
        }
        __device__ __forceinline__ void link(const JbOp &op, const PackView<T, NC> &v, const StringDesc &S,
                                             PackParams<T, NC> &pp, const Wts<T> &w, const WalkPos &q)
        {
            site(op, v, S, pp, w, q);
        }
        __device__ __forceinline__ void finish(const JbOp &, const StringDesc &, const Scalars &, int, int, int, int) {}
    };
};

// Magnetic flux of every image, Phi = dx^2 sum of B (post.py:131-133): reads A
// only.  Sums in double.
struct FluxOp {
    static constexpr bool psi = false, field = false;
    double *out;      // by image of the string
    template <class T, int NC>
    struct State {
        double b = 0.0;
        template <class W>
        __device__ __forceinline__ void site(const FluxOp &, const PackView<T, NC> &v, const StringDesc &,
                                             PackParams<T, NC> &pp, const W &w, const WalkPos &)
        {
            b += (double)site_b<T>(v.a, pp.idx, w);
        }
        __device__ __forceinline__ void link(const FluxOp &op, const PackView<T, NC> &v, const StringDesc &S,
                                             PackParams<T, NC> &pp, const Wts<T> &w, const WalkPos &q)
        {
            site(op, v, S, pp, w, q);
        }
        __device__ __forceinline__ void finish(const FluxOp &op, const StringDesc &S, const Scalars &sc, int u, int n,
                                               int tpi, int img)
        {
            const double v[1] = {b};
            double tot[1];
            if (finish_image_warp<1>(v, sc, u, n * tpi, tpi, tpi, img, tot) &&
                (threadIdx.x & 31) == 0)
                op.out[n] = tot[0] * S.ud.dx2;
        }
    };
};

// ------------------------------------------------------------------ kernel
// One strip per single-warp block; strips of the string in (image, row, column)
// order.  Rows in flight beyond the window: a walk reads a third of what an
// NLCG pass does per row, so where it is bound by memory (FP32, and the flux)
// one row per warp keeps few bytes in flight; a third costs registers (FP32, two
// components, 768 x 512 x 12, whole calls at 1, 2, 3 rows: energies 78, 79, 91 us,
// adjoints 74, 74, 85, gradients 87, 89, 93; 200 x 160 x 24 with holes, gradients:
// 49, 47, 51).
#ifndef MEPGL_WALK_AHEAD
#define MEPGL_WALK_AHEAD 2
#endif
// Blocks per SM: FP32 is bound by the latency of its loads.  One component fits 20
// warps' registers (gradients at 16 / 20 / 24 blocks: 180 x 150 x 24 with per-site
// parameters 31 / 25 / 29 us, uniform 24 / 22 / 25; 512 x 512 x 32 165 / 148 / 182
// and 113 / 109 / 145), two lose beyond 16 (512 x 512 x 32 at 16 / 20: 145 / 175).
template <class T, int NC>
struct WalkBlocks {
    static constexpr int v = sizeof(T) == 4 ? (NC == 1 ? 20 : 16) : 8;
};
template <class T, int NC, class Op>
__global__ void __launch_bounds__(NTS, WalkBlocks<T, NC>::v) k_walk(const __grid_constant__ StringDesc S, Scalars sc,
                                                                    int xbuf, Op op)
{
    using St = store_t<T>;
    using V = vec2_t<T>;
    using M = vec2_t<St>;
    constexpr int NF = Op::psi ? 1 + NC : 1, NP = Op::psi ? NC : 0;
    constexpr int PF = sizeof(T) == 4 || !Op::psi ? MEPGL_WALK_AHEAD : 1, RS = PF + 2;
    __shared__ __align__(16) M ring[RS][2][1][NF];
    const int u = blockIdx.x, tpi = S.tiles_x * S.wtiles_y, n = u / tpi, ur = u - n * tpi, ty = ur / S.tiles_x;
    const int i0 = (ur - ty * S.tiles_x) * TX, j0 = ty * S.wrows;
    const StripLane L = strip_lane(S, i0);
    const M *src[1][NF];
#pragma unroll
    for (int c = 0; c < NF; ++c) src[0][c] = static_cast<const M *>(S.x[xbuf][c]) + (size_t)n * S.nx * S.ny;
    PackParams<T, NC> pp;
    pp.load(S);
    struct Row {
        V x[NF], al, ar;
        uint16_t m;
    };
    M rc[PF][1][NF];
    uint16_t rm[PF];
    auto field = [](M v) {
        V r;
        r.x = from_store<T>(v.x);
        r.y = from_store<T>(v.y);
        return r;
    };
    auto take = [&](Row &R, int j, V (&hp)[NP + 1], const M (&raw)[1][NF], uint16_t m) {
        const M(&h)[NF] = ring[(j + RS) % RS][L.lane == 0 ? 0 : 1][0];
#pragma unroll
        for (int c = 0; c < NF; ++c) R.x[c] = field(raw[0][c]);
#pragma unroll
        for (int c = 0; c < NP; ++c) hp[c] = field(h[1 + c]);
        const V ha = field(h[0]);
        R.al = from_left2<T>(R.x[0], ha, L.lane);
        R.ar = from_right<T>(R.x[0], ha, L.lane);
        R.m = m;
    };
    const int rows = S.ny - j0 < S.wrows ? S.ny - j0 : S.wrows;
    // row j (nothing past the row above the strip; every call commits one group)
    auto load = [&](M (&raw)[1][NF], uint16_t &m, int j) {
        const bool issue = j <= j0 + rows;
        strip_load<St, NF - 1, 1>(raw, src, S, L, j, issue ? 1u : 0u);
        strip_halo<St, NF - 1, 1, 1>(ring[(j + RS) % RS], src, S, L, j, 1u, issue);
        m = issue ? walk_code(S, L, j) : 0;
    };
    Row Rm, R0, Rp;
    V hp0[NP + 1], hp1[NP + 1];
    {
        M ra[1][NF], rb[1][NF];
        uint16_t ma, mb;
        load(ra, ma, j0 - 1);
        load(rb, mb, j0);
#pragma unroll
        for (int k = 0; k < PF; ++k) load(rc[k], rm[k], j0 + 1 + k);
        cp_async_wait_groups<PF>();
        take(Rm, j0 - 1, hp0, ra, ma);
        take(R0, j0, hp0, rb, mb);
    }
    typename Op::template State<T, NC> st;
#pragma unroll 1
    for (int r = 0; r < rows; ++r) {
        const int j = j0 + r;
        cp_async_wait_groups<PF - 1>();   // row j + 1 has arrived
        take(Rp, j + 1, hp1, rc[0], rm[0]);
#pragma unroll
        for (int k = 0; k + 1 < PF; ++k) {
#pragma unroll
            for (int c = 0; c < NF; ++c) rc[k][0][c] = rc[k + 1][0][c];
            rm[k] = rm[k + 1];
        }
        load(rc[PF - 1], rm[PF - 1], j + 1 + PF);
        PackView<T, NC> v;
        const V z = zero2<T>();
        v.a[0][0] = Rm.al; v.a[0][1] = Rm.x[0]; v.a[0][2] = Rm.ar;
        v.a[1][0] = R0.al; v.a[1][1] = R0.x[0]; v.a[1][2] = R0.ar;
        v.a[2][0] = Rp.al; v.a[2][1] = Rp.x[0]; v.a[2][2] = Rp.ar;
        auto psi = [&](int dy, int dx, V p1, V p2) {
            v.px[dy][dx] = Pk<T, NC>::mk(p1.x, p2.x);
            v.py[dy][dx] = Pk<T, NC>::mk(p1.y, p2.y);
        };
        psi(0, 0, z, z); psi(0, 2, z, z); psi(2, 0, z, z); psi(2, 2, z, z);
        if constexpr (NP > 0) {
            V pl[NC], pr[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                pl[c] = from_left2<T>(R0.x[1 + c], hp0[c], L.lane);
                pr[c] = from_right<T>(R0.x[1 + c], hp0[c], L.lane);
            }
            psi(0, 1, Rm.x[1], Rm.x[NC]);
            psi(1, 1, R0.x[1], R0.x[NC]);
            psi(2, 1, Rp.x[1], Rp.x[NC]);
            psi(1, 0, pl[0], pl[NC - 1]);
            psi(1, 2, pr[0], pr[NC - 1]);
        } else {
            psi(0, 1, z, z); psi(1, 0, z, z); psi(1, 1, z, z); psi(1, 2, z, z); psi(2, 1, z, z);
        }
        bool inner = false;
        if constexpr (std::is_same<T, double>::value) inner = !S.disc && __all_sync(FULL_MASK, !L.cok || R0.m == 0xffffu);
        if (L.cok) {
            const WalkPos q{n, L.gi, j, L.gi + S.nx * j, r};
            if (S.per_site) {
                if constexpr (Op::field) st.ahead(S, q);
                pp.load_site(S, q.gi, q.j, q.s);
            }
            if (inner) {
                if constexpr (std::is_same<T, double>::value) st.site(op, v, S, pp, Ones(), q);
            } else {
                Wts<T> w;
                w.load(R0.m);
                if (S.disc) st.link(op, v, S, pp, w, q);
                else st.site(op, v, S, pp, w, q);
            }
        }
        Rm = R0;
        R0 = Rp;
#pragma unroll
        for (int c = 0; c < NP; ++c) hp0[c] = hp1[c];
    }
    st.finish(op, S, sc, u, n, tpi, S.img_base + n);
}

// ------------------------------------------------------------- arc lengths
// Squared distances between adjacent images (interpolation.cu:39-92: every
// site, no mask, no dx^2) in the field metric and in the (B, J) metric, FP32.
// A block walks a strip of ARC_ROWS rows through a chunk of images and keeps
// the image before in shared memory, so that each image is read once and B and
// J are never stored (256 x 256 x 64: 77 us; B and J written, then they and the
// fields read: 53 + 26 + 25).  part[n nb + strip]: sum over image n against
// image n - 1.
constexpr int ARC_ROWS = 8;

template <int NC>
__global__ void __launch_bounds__(NTS, 16) k_arc_walk(const __grid_constant__ StringDesc S, int xbuf, int chunk,
                                                      double *part_f, double *part_jb)
{
    using T = float;
    constexpr int K = 3 + 4 * NC;   // B, J; the fields
    using V = vec2_t<T>;
    __shared__ __align__(16) V ring[3][2][1][1 + NC];
    __shared__ T prev[ARC_ROWS][K][NTS];
    const int u = blockIdx.x, nb = gridDim.x, ty = u / S.tiles_x;
    const int i0 = (u - ty * S.tiles_x) * TX, j0 = ty * ARC_ROWS;
    const StripLane L = strip_lane(S, i0);
    PackParams<T, NC> pp;
    pp.load(S);
    const int rows = S.ny - j0 < ARC_ROWS ? S.ny - j0 : ARC_ROWS;
    const int c0 = blockIdx.y * chunk, c1 = c0 + chunk < S.F ? c0 + chunk : S.F, first = c0 > 0 ? c0 - 1 : 0;
    struct Row {
        V x[1 + NC], al, ar;
        uint16_t m;
    };
    for (int n = first; n < c1; ++n) {
        const V *src[1][1 + NC];
#pragma unroll
        for (int c = 0; c < 1 + NC; ++c) src[0][c] = static_cast<const V *>(S.x[xbuf][c]) + (size_t)n * S.nx * S.ny;
        V rc[1][1 + NC];
        uint16_t rm;
        auto take = [&](Row &R, int j, V (&hp)[NC], const V (&raw)[1][1 + NC], uint16_t m) {
            cp_async_wait_groups<0>();
            const V(&h)[1 + NC] = ring[(j + 3) % 3][L.lane == 0 ? 0 : 1][0];
#pragma unroll
            for (int c = 0; c < 1 + NC; ++c) R.x[c] = raw[0][c];
#pragma unroll
            for (int c = 0; c < NC; ++c) hp[c] = h[1 + c];
            R.al = from_left2<T>(R.x[0], h[0], L.lane);
            R.ar = from_right<T>(R.x[0], h[0], L.lane);
            R.m = m;
        };
        auto load = [&](V (&raw)[1][1 + NC], uint16_t &m, int j) {
            strip_load<T, NC, 1>(raw, src, S, L, j, 1u);
            strip_halo<T, NC, 1, 1>(ring[(j + 3) % 3], src, S, L, j, 1u, true);
            m = strip_code(S, L, j);
        };
        Row Rm, R0, Rp;
        V hp0[NC], hp1[NC];
        {
            V ra[1][1 + NC], rb[1][1 + NC];
            uint16_t ma, mb;
            load(ra, ma, j0 - 1);
            load(rb, mb, j0);
            load(rc, rm, j0 + 1);
            take(Rm, j0 - 1, hp0, ra, ma);
            take(R0, j0, hp0, rb, mb);
        }
        const bool diff = n > first;
        T df = (T)0, dj = (T)0;
#pragma unroll 1
        for (int r = 0; r < rows; ++r) {
            const int j = j0 + r;
            take(Rp, j + 1, hp1, rc, rm);
            if (r + 1 < rows) load(rc, rm, j + 2);
            PackView<T, NC> v;
            {
                const V z = zero2<T>();
                v.a[0][0] = v.a[0][2] = v.a[2][0] = v.a[2][2] = z;
                v.a[0][1] = Rm.x[0];
                v.a[1][0] = R0.al; v.a[1][1] = R0.x[0]; v.a[1][2] = R0.ar;
                v.a[2][1] = Rp.x[0];
                V pl[NC], pr[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    pl[c] = from_left2<T>(R0.x[1 + c], hp0[c], L.lane);
                    pr[c] = from_right<T>(R0.x[1 + c], hp0[c], L.lane);
                }
                auto psi = [&](int dy, int dx, V p1, V p2) {
                    v.px[dy][dx] = Pk<T, NC>::mk(p1.x, p2.x);
                    v.py[dy][dx] = Pk<T, NC>::mk(p1.y, p2.y);
                };
                psi(0, 0, z, z); psi(0, 2, z, z); psi(2, 0, z, z); psi(2, 2, z, z);
                psi(0, 1, Rm.x[1], Rm.x[NC]);
                psi(1, 1, R0.x[1], R0.x[NC]);
                psi(2, 1, Rp.x[1], Rp.x[NC]);
                psi(1, 0, pl[0], pl[NC - 1]);
                psi(1, 2, pr[0], pr[NC - 1]);
            }
            if (L.cok) {
                T o[K];
                if (S.per_site) pp.load_site(S, L.gi, j, L.gi + S.nx * j);
                Wts<T> w;
                w.load(R0.m);
                site_jb<T, NC>(v, pp, w, o);
#pragma unroll
                for (int c = 0; c < 1 + NC; ++c) {
                    o[1 + 2 * NC + 2 * c] = R0.x[c].x;
                    o[2 + 2 * NC + 2 * c] = R0.x[c].y;
                }
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    T &p = prev[r][k][L.lane];
                    const T e = o[k] - p;
                    if (diff) {
                        if (k < 1 + 2 * NC) dj = fma1(e, e, dj);
                        else df = fma1(e, e, df);
                    }
                    p = o[k];
                }
            }
            Rm = R0;
            R0 = Rp;
#pragma unroll
            for (int c = 0; c < NC; ++c) hp0[c] = hp1[c];
        }
        if (n < c0) continue;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            df += __shfl_down_sync(FULL_MASK, df, o);
            dj += __shfl_down_sync(FULL_MASK, dj, o);
        }
        if (L.lane == 0) {
            part_f[(size_t)n * nb + u] = (double)df;
            part_jb[(size_t)n * nb + u] = (double)dj;
        }
    }
}
