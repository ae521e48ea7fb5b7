// strip.cuh -- the two NLCG passes as warp strips, for float, double and
// float-float fields, launched as two pass kernels per step or as one fused
// persistent launch per call (end of file).  Included by kernels.cu inside
// its anonymous namespace.
//
// A block is one warp.  In the pass kernels it owns one strip (TX = 32
// columns x S.rows rows of one image); in the fused kernel it takes strips
// from a work queue.  Everything that depends on the strip (pointers,
// parameters, row numbers) is uniform over the block.  Lane l holds column
// i0 + l and walks down the strip's rows with a three-row window of its
// column in registers; the x-neighbours come from the adjacent lanes by
// shuffles.  Lanes 0 and 31 copy the halo column next to them (i0 - 1, i0 +
// 32) into a three-row ring in shared memory with cp.async and read it back
// themselves, so no lane waits for another.  Rows j0 - 1 and j0 + S.rows are
// read as halo rows.  While a row is computed, the loads of the next row are
// in flight.  Every strip leaves one partial per quantity and group of S.grows
// rows, and the last strip of an image (atomic ticket) finishes it.  The groups
// follow from the string alone and a strip is one of them, or in a batch, where
// there are strips enough, several: a string's sums are the same in any batch.
//
// FP64: bound by the FP64 pipe, 64 clocks per warp instruction and SM
// quarter, so 8 warps per SM (255 registers; the fused launch of two components
// spills some 80 of its values around a pass) keep it busy and the strips' equal
// sharing of the quarters counts.  256 x 256 x 64, two components, per step: FP64
// 3.83 ms, float-float 1.33, against 6.5 and 1.7 as shared-memory tiles of 256
// threads; 64 x 64 x 16, one component, ten steps with reparametrization in FP64:
// 0.63 ms against 1.17.
#pragma once

constexpr int NTS = 32;   // threads per block of the strip kernels

// The window of a two-component string holds psi as the stencils' packs,
// (Re psi_1, Re psi_2) and (Im psi_1, Im psi_2), in the two pair slots of the
// components.
template <int NC>
struct StripPacked {
    static constexpr bool v = NC == 2;
};

// (re, im) of two components <-> (Re 1, Re 2), (Im 1, Im 2): a 2 x 2 transpose.
template <class V>
__device__ __forceinline__ void transpose_pair(V &a, V &b)
{
    const V p = a, q = b;
    a.x = p.x;
    a.y = q.x;
    b.x = p.y;
    b.y = q.y;
}

constexpr unsigned FULL_MASK = 0xffffffffu;

// Register window of one site; the strip kernels fill the entries their
// stencil reads and leave the others zero.
template <class T, int NC>
struct RegView {
    vec2_t<T> a[3][3];
    vec2_t<T> p[NC][3][3];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int y = 0; y < 3; ++y)
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                a[y][x].x = a[y][x].y = (T)0;
#pragma unroll
                for (int c = 0; c < NC; ++c) p[c][y][x].x = p[c][y][x].y = (T)0;
            }
    }
};

// The stencils' view of a register window (for two components its psi slots
// already hold the packs).
template <class T, int NC>
__device__ __forceinline__ PackView<T, NC> pack_view(const RegView<T, NC> &r)
{
    PackView<T, NC> v;
#pragma unroll
    for (int y = 0; y < 3; ++y)
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            v.a[y][x] = r.a[y][x];
            if constexpr (NC == 1) {
                v.px[y][x] = r.p[0][y][x].x;
                v.py[y][x] = r.p[0][y][x].y;
            } else {
                v.px[y][x] = Pk<T, NC>::mk(r.p[0][y][x].x, r.p[0][y][x].y);
                v.py[y][x] = Pk<T, NC>::mk(r.p[1][y][x].x, r.p[1][y][x].y);
            }
        }
    return v;
}

template <class T>
__device__ __forceinline__ vec2_t<T> zero2()
{
    vec2_t<T> z;
    z.x = z.y = (T)0;
    return z;
}

// Value of the lane to the right (column + 1); lane 31 takes its halo.
template <class T>
__device__ __forceinline__ vec2_t<T> from_right(vec2_t<T> v, vec2_t<T> halo, int lane)
{
    vec2_t<T> r;
    r.x = shfl_right(v.x);
    r.y = shfl_right(v.y);
    return lane == TX - 1 ? halo : r;
}

// Value of the lane to the left (column - 1); lane 0 takes its halo.
template <class T>
__device__ __forceinline__ T from_left(T v, T halo, int lane)
{
    const T l = shfl_left(v);
    return lane == 0 ? halo : l;
}

template <class T>
__device__ __forceinline__ vec2_t<T> from_left2(vec2_t<T> v, vec2_t<T> halo, int lane)
{
    vec2_t<T> l;
    l.x = from_left<T>(v.x, halo.x, lane);
    l.y = from_left<T>(v.y, halo.y, lane);
    return l;
}

// Column geometry of one lane within its tile.
struct StripLane {
    int lane, gi, hc;   // own column, halo column (lanes 0 and 31)
    bool cok, hok;      // own column / halo column inside the lattice
};

__device__ __forceinline__ StripLane strip_lane(const StringDesc &S, int i0)
{
    StripLane L;
    L.lane = threadIdx.x & 31;
    L.gi = i0 + L.lane;
    L.hc = L.lane == 0 ? i0 - 1 : i0 + TX;
    L.cok = L.gi < S.nx;
    L.hok = (L.lane == 0 || L.lane == TX - 1) && L.hc >= 0 && L.hc < S.nx;
    return L;
}

// Loads of one row j: NA arrays of (1 + NC) pair fields at the lane's
// column (zero outside the lattice); array a is read if bit a of cmask is set.
template <class T, int NC, int NA>
__device__ __forceinline__ void strip_load(vec2_t<T> (&c)[NA][1 + NC], const vec2_t<T> *const (&src)[NA][1 + NC],
                                           const StringDesc &S, const StripLane &L, int j, unsigned cmask)
{
    const bool rok = j >= 0 && j < S.ny;
    const int sc_ = rok && L.cok ? L.gi + S.nx * j : 0;
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int k = 0; k < 1 + NC; ++k) c[a][k] = zero2<T>();
#pragma unroll
    for (int a = 0; a < NA; ++a)
        if (((cmask >> a) & 1u) && rok && L.cok)
#pragma unroll
            for (int k = 0; k < 1 + NC; ++k) c[a][k] = src[a][k][sc_];
}

// Zeros in place of the arrays that are not in `keep`.
template <class T, int NC>
__device__ __forceinline__ void drop_arrays(vec2_t<T> (&c)[3][1 + NC], unsigned keep)
{
#pragma unroll
    for (int a = 1; a < 3; ++a)
        if (!((keep >> a) & 1u))
#pragma unroll
            for (int k = 0; k < 1 + NC; ++k) c[a][k] = zero2<T>();
}

// Halo column of row j: lanes 0 and 31 copy arrays a < NR of hmask at their
// halo column into slot[side][a] by cp.async (zero-filled outside the
// lattice).  Every lane commits one group per call (empty for the others,
// or when `issue` is false), so group counts stay uniform.
template <class T, int NC, int NR, int NA>
__device__ __forceinline__ void strip_halo(vec2_t<T> (&slot)[2][NR][1 + NC], const vec2_t<T> *const (&src)[NA][1 + NC],
                                           const StringDesc &S, const StripLane &L, int j, unsigned hmask, bool issue)
{
    if (issue && (L.lane == 0 || L.lane == TX - 1)) {
        const bool hv = j >= 0 && j < S.ny && L.hok;
        const int sh = hv ? L.hc + S.nx * j : 0;
        vec2_t<T>(&dst)[NR][1 + NC] = slot[L.lane == 0 ? 0 : 1];
#pragma unroll
        for (int a = 0; a < NR; ++a)
            if ((hmask >> a) & 1u)
#pragma unroll
                for (int k = 0; k < 1 + NC; ++k) cp_async<sizeof(vec2_t<T>)>(&dst[a][k], src[a][k] + sh, hv);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// Wait until at most N of this thread's newest cp.async groups are pending.
template <int N>
__device__ __forceinline__ void cp_async_wait_groups() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Strip g of the global strip order (strings in order, each from its
// stile_base: image, strip row, column), derived from the block index and
// the descriptors alone so that it is uniform over the block.
// ONE: the launch covers a single string (bt.n == 1); its descriptor is
// then read at fixed offsets, i.e. as constant operands, not through
// indexed constant loads.
template <bool ONE>
__device__ __forceinline__ StripRef strip_tile(const batch_t<ONE> &bt, int g)
{
    int s = 0;
    if (!ONE)
        for (int k = 1; k < bt.n; ++k)
            if (g >= bt.s[k].stile_base) s = k;
    const StringDesc &S = bt.s[s];
    const int r = g - S.stile_base, tpi = S.tiles_x * S.stiles_y, n = r / tpi, u = r - n * tpi, ty = u / S.tiles_x;
    StripRef t;
    t.s = s;
    t.ty = ty;
    t.tx = u - ty * S.tiles_x;
    t.n = n;
    return t;
}

// Slot of a strip's first partial sums (its next group's: tiles_x further).
__device__ __forceinline__ int strip_slot(const StringDesc &S, const StripRef &tr)
{
    return S.part_base + tr.n * S.groups + tr.ty * S.gper * S.tiles_x + tr.tx;
}

// Packed neighbour codes of the lane's site in row j (0 outside the lattice).
__device__ __forceinline__ uint16_t strip_code(const StringDesc &S, const StripLane &L, int j)
{
    if (!(j >= 0 && j < S.ny && L.cok)) return 0;
    return S.mask[L.gi + S.nx * j];
}

// Sums of N values over a warp with about N + 3 additions instead of 5 N: at
// each of the first distances a lane gives half of its values away and adds
// the other half, so that value k ends up in lane sum_lane<N>(k) (and in others).
template <int N>
__device__ constexpr int sum_lane(int k)
{
    int lane = 0;
    for (int n = N, o = 16; n > 1; n = (n + 1) / 2, o >>= 1)
        if (k >= (n + 1) / 2) {
            lane |= o;
            k -= (n + 1) / 2;
        }
    return lane;
}

template <int N, class T>
__device__ __forceinline__ T warp_sums(T (&w)[N])
{
    const int lane = threadIdx.x & 31;
    int n = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int h = (n + 1) / 2;
        const bool up = n > 1 && (lane & o);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (i >= h) continue;
            const T hi = n == 1 ? w[i] : i + h < n ? w[i + h < N ? i + h : i] : (T)0;
            const T keep = up ? hi : w[i], give = up ? w[i] : hi;
            w[i] = keep + shfl_xor(give, o);
        }
        n = h;
    }
    return w[0];
}

// Sums of n strips' partials (8 doubles each, NV used), added in index order
// per lane, to every lane.  AHEAD strips' loads are in flight per lane.
constexpr int AHEAD = 4;
template <int NV>
__device__ __forceinline__ void image_sums(const double *part, int n, double (&tot)[NV])
{
    const int lane = threadIdx.x & 31;
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = 0.0;
    for (int t0 = 0; t0 < n; t0 += 32 * AHEAD) {
        double q[AHEAD][NV];
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) {
            const int t = t0 + 32 * a + lane;
#pragma unroll
            for (int k = 0; k < NV; ++k) q[a][k] = t < n ? __ldcg(part + (size_t)t * 8 + k) : 0.0;
        }
#pragma unroll
        for (int a = 0; a < AHEAD; ++a)
#pragma unroll
            for (int k = 0; k < NV; ++k) acc[k] += q[a][k];
    }
    const double all = warp_sums<NV>(acc);
#pragma unroll
    for (int k = 0; k < NV; ++k) tot[k] = __shfl_sync(FULL_MASK, all, sum_lane<NV>(k));
}

// NV sums of a group of rows leave the warp.
template <int NV, class T>
__device__ __forceinline__ void store_sums(const T (&v)[NV], const Scalars &sc, int slot)
{
    const int lane = threadIdx.x & 31;
    T w[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) w[k] = v[k];
    const double mine = (double)warp_sums<NV>(w);
#pragma unroll
    for (int k = 0; k < NV; ++k)
        if (lane == sum_lane<NV>(k)) sc.part[(size_t)slot * 8 + k] = mine;
}

// The strip is done.  If it is the last of its image's `strips`, every lane
// receives the image sums (its `sums` partials from `first` on, added in index
// order) and the function returns true.  Everything that the lanes wrote before,
// the strip's partials among it, is visible to whoever learns from the ticket (or
// from what the last strip publishes) that the strip is done: the warp barrier
// orders the lanes' writes before lane 0's fence, which is cumulative.
template <int NV>
__device__ __forceinline__ bool finish_image(const Scalars &sc, int first, int sums, int strips, int img, double (&tot)[NV])
{
    const int lane = threadIdx.x & 31;
    __syncwarp();
    int last = 0;
    if (lane == 0) {
        __threadfence();
        last = atomicAdd(&sc.ticket[img], 1u) == (unsigned)strips - 1;
        if (last) __threadfence();
    }
    last = __shfl_sync(FULL_MASK, last, 0);
    if (!last) return false;
    __syncwarp();
    image_sums<NV>(sc.part + (size_t)first * 8, sums, tot);
    if (lane == 0) sc.ticket[img] = 0;
    return true;
}

// The same for a strip of one group of rows, whose NV sums leave the warp first.
template <int NV, class T>
__device__ __forceinline__ bool finish_image_warp(const T (&v)[NV], const Scalars &sc, int slot, int first, int sums,
                                                  int strips, int img, double (&tot)[NV])
{
    store_sums<NV>(v, sc, slot);
    return finish_image<NV>(sc, first, sums, strips, img, tot);
}

// One row of x + alpha d as the gradient window holds it: fields of the
// lane's column, A of the columns left and right, the row's previous
// gradient and neighbour codes.
template <class T, int NC>
struct GradRow {
    vec2_t<T> x[1 + NC], al, ar, gold[1 + NC];
    uint16_t m;
};

// Re and Im psi packs from a window row's psi slots.
template <class T, int NC>
__device__ __forceinline__ pack_t<T, NC> psi_x(const vec2_t<T> *p)
{
    if constexpr (NC == 1) return p[0].x;
    else return Pk<T, NC>::mk(p[0].x, p[0].y);
}
template <class T, int NC>
__device__ __forceinline__ pack_t<T, NC> psi_y(const vec2_t<T> *p)
{
    if constexpr (NC == 1) return p[0].y;
    else return Pk<T, NC>::mk(p[NC - 1].x, p[NC - 1].y);
}

template <class T, int NC>
__device__ __forceinline__ GradView<T, NC> grad_view(const GradRow<T, NC> &R)
{
    return GradView<T, NC>{R.x[0], R.al, R.ar, psi_x<T, NC>(R.x + 1), psi_y<T, NC>(R.x + 1)};
}

// The carry into row c from the row d below it.
template <class T, int NC>
__device__ __forceinline__ GradCarry<T, NC> grad_below(const GradRow<T, NC> &d, const GradRow<T, NC> &c,
                                                       const PackParams<T, NC> &pp, const Wts<T> &w)
{
    GradCarry<T, NC> k;
    const GradView<T, NC> vd = grad_view(d);
    grad_up<T, NC>(vd, grad_view(c), pp, w.wby, vd.ar.y - vd.a.y, vd.a.y - vd.al.y, k);
    return k;
}

// Halo ring of the gradient pass: [row % 3][side][x, d][field].
template <class T, int NC>
using GradRing = vec2_t<T>[3][2][2][1 + NC];

// Gradient pass on one strip: x <- x + alpha_pend d over the strip (+ halo),
// the gradient of every site, |g|^2 and g . (g - g_prev); the last strip of an
// image computes beta.  Returns true (in every lane) when this strip finished
// its image; a consumer in the same launch that has seen the image finished
// reads the field stores (finish_image).
template <class T, int NC, bool ONE, bool PS = true>
__device__ __forceinline__ bool grad_tile(const batch_t<ONE> &bt, const StripRef tr, const Scalars &sc, const StepFlags &f,
                                          GradRing<T, NC> &ring)
{
    using V = vec2_t<T>;
    const StringDesc &S = bt.s[ONE ? 0 : tr.s];
    const int img = S.img_base + tr.n;
    const int i0 = tr.tx * TX, j0 = tr.ty * S.rows;
    const size_t off = (size_t)tr.n * S.nx * S.ny;
    const StripLane L = strip_lane(S, i0);
    const V *src[3][1 + NC];
    V *xout[1 + NC], *gcur[1 + NC];
#pragma unroll
    for (int c = 0; c < 1 + NC; ++c) {
        src[0][c] = static_cast<const V *>(S.x[f.xin][c]) + off;
        src[1][c] = static_cast<const V *>(S.d[f.din][c]) + off;
        src[2][c] = static_cast<const V *>(S.g[f.gprev][c]) + off;
        xout[c] = static_cast<V *>(S.x[f.xout][c]) + off;
        gcur[c] = static_cast<V *>(S.g[f.gcur][c]) + off;
    }
    const double alpha_d = __ldcg(sc.alpha_pend + img), norm = f.use_cg ? __ldcg((f.gprev ? sc.gn1 : sc.gn0) + img) : INFINITY;
    // the first three rows are loaded together, and before the scalars are looked
    // at: one memory latency, not three or four.  What turns out not to be read
    // (below) is dropped again.
    V ra[3][1 + NC], rb[3][1 + NC], rc[3][1 + NC];
    uint16_t ma, mb, rm;
    auto load = [&](V (&raw)[3][1 + NC], uint16_t &m, int j, unsigned arrays) {
        strip_load<T, NC, 3>(raw, src, S, L, j, arrays);
        strip_halo<T, NC, 2, 3>(ring[(j + 3) % 3], src, S, L, j, arrays & 3u, true);
        m = strip_code(S, L, j);
    };
    load(ra, ma, j0 - 1, 3u);
    load(rb, mb, j0, f.use_cg ? 7u : 3u);
    load(rc, rm, j0 + 1, f.use_cg ? 7u : 3u);
    const T alpha = (T)alpha_d;
    // d is not read when nothing is pending, nor g_prev when it does not enter
    // beta (restarted image, steepest descent)
    const unsigned fields = (alpha != (T)0 ? 3u : 1u) | (norm <= 1.7976931348623157e308 ? 4u : 0u);
    drop_arrays<T, NC>(ra, fields);
    drop_arrays<T, NC>(rb, fields);
    drop_arrays<T, NC>(rc, fields);
    PackParams<T, NC> pp;
    pp.load(S);
    // raw row j -> window row (x + alpha d; left / right A by shuffles)
    auto take = [&](GradRow<T, NC> &R, int j, V (&hp)[NC], const V (&raw)[3][1 + NC], uint16_t m) {
        cp_async_wait_groups<0>();   // row j's halo is in the newest groups
        const V(&h)[2][1 + NC] = ring[(j + 3) % 3][L.lane == 0 ? 0 : 1];
        V hx[1 + NC];
#pragma unroll
        for (int c = 0; c < 1 + NC; ++c) {
            R.x[c].x = raw[0][c].x + alpha * raw[1][c].x;
            R.x[c].y = raw[0][c].y + alpha * raw[1][c].y;
            const V hv = h[0][c], hd = fields & 2u ? h[1][c] : zero2<T>();
            hx[c].x = hv.x + alpha * hd.x;
            hx[c].y = hv.y + alpha * hd.y;
            R.gold[c] = raw[2][c];
        }
        if constexpr (StripPacked<NC>::v) {
            transpose_pair(R.x[1], R.x[NC]);
            transpose_pair(hx[1], hx[NC]);
        }
        R.al = from_left2<T>(R.x[0], hx[0], L.lane);
        R.ar = from_right<T>(R.x[0], hx[0], L.lane);
#pragma unroll
        for (int c = 0; c < NC; ++c) hp[c] = hx[1 + c];
        R.m = m;
    };
    // FP64 and float-float rows hand their upper y-link and views on to the next
    // (21 FP64 instructions fewer a site); FP32 forms them again from the row below,
    // because the carry costs 20 registers, i.e. warps (sweep of 16 strings:
    // 15.8 ms against 16.5 with the carry)
    constexpr bool CARRY = !std::is_same<T, float>::value;
    GradRow<T, NC> Rm, R0, Rp;
    V hp0[NC], hp1[NC];
    GradCarry<T, NC> up;   // from the row below
    {
        take(Rm, j0 - 1, hp0, ra, ma);
        take(R0, j0, hp0, rb, mb);
        if constexpr (CARRY) {
            // the link from row j0 - 1 with the weight that row j0 knows it by
            Wts<T> w;
            w.load(R0.m);
            up = grad_below(Rm, R0, pp, w);
        }
    }
    const int rows = S.ny - j0 < S.rows ? S.ny - j0 : S.rows;
    T v[2] = {(T)0, (T)0};
    int slot = strip_slot(S, tr), left = S.grows;   // of the present group of rows; its rows to go
#pragma unroll 1
    for (int r = 0; r < rows; ++r) {
        const int j = j0 + r;
        take(Rp, j + 1, hp1, rc, rm);
        if (r + 1 < rows) load(rc, rm, j + 2, fields);
        const int s = L.gi + S.nx * j;
        if (L.cok) {
            V o[1 + NC];
#pragma unroll
            for (int c = 0; c < 1 + NC; ++c) o[c] = R0.x[c];
            if constexpr (StripPacked<NC>::v) transpose_pair(o[1], o[NC]);
#pragma unroll
            for (int c = 0; c < 1 + NC; ++c) xout[c][s] = o[c];
        }
        V pl[NC], pr[NC];   // psi of the columns left and right
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            pl[c] = from_left2<T>(R0.x[1 + c], hp0[c], L.lane);
            pr[c] = from_right<T>(R0.x[1 + c], hp0[c], L.lane);
        }
        bool inner = false;
        if constexpr (std::is_same<T, double>::value) inner = __all_sync(FULL_MASK, !L.cok || R0.m == 0xffffu);
        if (L.cok) {
            FieldSites<T> near;
            if (PS && S.per_site) {
                near.load(S, L.gi, j, s);
                pp.load_pass_site(S, L.gi, j, s);
            }
            const GradView<T, NC> vc = grad_view(R0), vu = grad_view(Rp);
            const FieldSums<T> h = field_sums<T, NC, true, PS>(S, pp, near, L.gi, j, s);
            T g[2 + 2 * NC];
            if (inner) {
                if constexpr (std::is_same<T, double>::value)
                    site_gradient<T, NC>(vc, vu, psi_x<T, NC>(pl), psi_y<T, NC>(pl), psi_x<T, NC>(pr), psi_y<T, NC>(pr),
                                         pp, Ones(), h, PS && S.per_site, f.maxwell, S.thin_film, up, g);
            } else {
                Wts<T> w;
                w.load(R0.m);
                if constexpr (!CARRY) up = grad_below(Rm, R0, pp, w);
                site_gradient<T, NC>(vc, vu, psi_x<T, NC>(pl), psi_y<T, NC>(pl), psi_x<T, NC>(pr), psi_y<T, NC>(pr), pp,
                                     w, h, PS && S.per_site, f.maxwell, S.thin_film, up, g);
            }
#pragma unroll
            for (int c = 0; c < 1 + NC; ++c) {
                V gv;
                gv.x = g[2 * c];
                gv.y = g[2 * c + 1];
                gcur[c][s] = gv;
                const V go = R0.gold[c];
                v[0] = fma1(gv.x, gv.x, fma1(gv.y, gv.y, v[0]));
                v[1] = fma1(gv.x, gv.x - go.x, fma1(gv.y, gv.y - go.y, v[1]));
            }
        }
        if constexpr (!ONE)
            if (--left == 0 || r + 1 == rows) {
                store_sums<2>(v, sc, slot);
                v[0] = v[1] = (T)0;
                slot += S.tiles_x;
                left = S.grows;
            }
        if constexpr (!CARRY) Rm = R0;
        R0 = Rp;
#pragma unroll
        for (int c = 0; c < NC; ++c) hp0[c] = hp1[c];
    }
    const int tpi = S.tiles_x * S.stiles_y;
    double tot[2];
    if constexpr (ONE) store_sums<2>(v, sc, slot);
    const bool fin = finish_image<2>(sc, S.part_base + tr.n * S.groups, S.groups, tpi, img, tot);
    if (fin && L.lane == 0) {
        (f.gcur ? sc.gn1 : sc.gn0)[img] = tot[0];
        sc.gdg[img] = tot[1];
        double beta = 0.0;
        if (f.use_cg) {
            beta = tot[1] / __ldcg((f.gprev ? sc.gn1 : sc.gn0) + img);   // again: a register pair held through the rows costs more
            beta = beta > 0.0 ? beta : 0.0;   // Polak-Ribiere clipped at 0; NaN -> 0
        }
        sc.beta[img] = beta;
    }
    return fin;
}

template <class T, int NC, bool ONE, bool PS = true>
__global__ void __launch_bounds__(NTS, (StripBlocks<T, NC, ONE>::grad)) k_grad_s(const __grid_constant__ batch_t<ONE> bt,
                                                                  int tile0, Scalars sc, StepFlags f)
{
    __shared__ __align__(16) GradRing<T, NC> ring;
    grad_tile<T, NC, ONE, PS>(bt, strip_tile<ONE>(bt, tile0 + (int)blockIdx.x), sc, f, ring);
}

// One row of the polynomial window: fields and new direction of the lane's
// column and the row's neighbour codes.
template <class T, int NC>
struct DirRow {
    vec2_t<T> x[1 + NC], d[1 + NC];
    uint16_t m;
};

// Halo ring of the direction pass: [row % 3][side][x, g, d][field].
template <class T, int NC>
using DirRing = vec2_t<T>[3][2][3][1 + NC];

// Direction pass on one strip: d <- -g + beta d over the strip (+ halo), the
// quartic coefficients of F(x + a d); the last strip of an image runs the line
// search.  Returns true (in every lane) when this strip finished its image.
template <class T, int NC, bool ONE, bool PS = true>
__device__ __forceinline__ bool dir_tile(const batch_t<ONE> &bt, const StripRef tr, const Scalars &sc, const StepFlags &f,
                                         DirRing<T, NC> &ring, double (&coef)[5])
{
    using V = vec2_t<T>;
    const StringDesc &S = bt.s[ONE ? 0 : tr.s];
    const int img = S.img_base + tr.n;
    const int i0 = tr.tx * TX, j0 = tr.ty * S.rows;
    const size_t off = (size_t)tr.n * S.nx * S.ny;
    const StripLane L = strip_lane(S, i0);
    const V *src[3][1 + NC];
    V *dout[1 + NC];
#pragma unroll
    for (int c = 0; c < 1 + NC; ++c) {
        src[0][c] = static_cast<const V *>(S.x[f.xout][c]) + off;
        src[1][c] = static_cast<const V *>(S.g[f.gcur][c]) + off;
        src[2][c] = static_cast<const V *>(S.d[f.din][c]) + off;
        dout[c] = static_cast<V *>(S.d[f.dout][c]) + off;
    }
    const double beta_d = __ldcg(sc.beta + img);
    V ra[3][1 + NC], rb[3][1 + NC], rc[3][1 + NC];   // as in grad_tile
    uint16_t ma, mb, rm;
    auto load = [&](V (&raw)[3][1 + NC], uint16_t &m, int j, unsigned arrays) {
        strip_load<T, NC, 3>(raw, src, S, L, j, arrays);
        strip_halo<T, NC, 3, 3>(ring[(j + 3) % 3], src, S, L, j, arrays, true);
        m = strip_code(S, L, j);
    };
    load(ra, ma, j0 - 1, f.use_cg ? 7u : 3u);
    load(rb, mb, j0, f.use_cg ? 7u : 3u);
    load(rc, rm, j0 + 1, f.use_cg ? 7u : 3u);
    const T beta = (T)beta_d;
    const unsigned fields = beta != (T)0 ? 7u : 3u;    // d is not read when it does not enter
    drop_arrays<T, NC>(ra, fields);
    drop_arrays<T, NC>(rb, fields);
    drop_arrays<T, NC>(rc, fields);
    PackParams<T, NC> pp;
    pp.load(S);
    auto take = [&](DirRow<T, NC> &R, const V (&raw)[3][1 + NC], uint16_t m) {
#pragma unroll
        for (int c = 0; c < 1 + NC; ++c) {
            R.x[c] = raw[0][c];
            R.d[c].x = -raw[1][c].x + beta * raw[2][c].x;
            R.d[c].y = -raw[1][c].y + beta * raw[2][c].y;
        }
        if constexpr (StripPacked<NC>::v) {
            transpose_pair(R.x[1], R.x[NC]);
            transpose_pair(R.d[1], R.d[NC]);
        }
        R.m = m;
    };
    DirRow<T, NC> R0, Rp;
    T xm_ax, dm_ax;   // row j - 1: only A_x of x and of d is read
    {
        take(R0, ra, ma);
        xm_ax = R0.x[0].x;
        dm_ax = R0.d[0].x;
        take(R0, rb, mb);
    }
    const int rows = S.ny - j0 < S.rows ? S.ny - j0 : S.rows;
    T v[5] = {(T)0, (T)0, (T)0, (T)0, (T)0};
    // FP32 adds up a site's terms first (they cancel); the wider types the strip's
    constexpr bool WIDE = !std::is_same<T, float>::value;
    PolySum<T, NC> sum;
    sum.zero();
    bool links = false;   // some row was one of interior sites
    int slot = strip_slot(S, tr), left = S.grows;   // of the present group of rows; its rows to go
#pragma unroll 1
    for (int r = 0; r < rows; ++r) {
        const int j = j0 + r;
        take(Rp, rc, rm);
        if (r + 1 < rows) load(rc, rm, j + 2, fields);
        else strip_halo<T, NC, 3, 3>(ring[0], src, S, L, j + 2, 0u, false);
        cp_async_wait_groups<2>();   // groups of rows j + 1 and j + 2 may still be pending
        const int s = L.gi + S.nx * j;
        if (L.cok) {
            V o[1 + NC];
#pragma unroll
            for (int c = 0; c < 1 + NC; ++c) o[c] = R0.d[c];
            if constexpr (StripPacked<NC>::v) transpose_pair(o[1], o[NC]);
#pragma unroll
            for (int c = 0; c < 1 + NC; ++c) dout[c][s] = o[c];
        }
        // halo column of row j (this lane's side), new direction formed here
        const V(&h)[3][1 + NC] = ring[j % 3][L.lane == 0 ? 0 : 1];
        V hx[1 + NC], hd[1 + NC];
#pragma unroll
        for (int c = 0; c < 1 + NC; ++c) {
            hx[c] = h[0][c];
            const V hg = h[1][c], hdd = fields & 4u ? h[2][c] : zero2<T>();
            hd[c].x = -hg.x + beta * hdd.x;
            hd[c].y = -hg.y + beta * hdd.y;
        }
        if constexpr (StripPacked<NC>::v) {
            transpose_pair(hx[1], hx[NC]);
            transpose_pair(hd[1], hd[NC]);
        }
        RegView<T, NC> vx, vd;
        vx.clear();
        vd.clear();
        vx.a[1][1] = R0.x[0];
        vd.a[1][1] = R0.d[0];
        vx.a[1][2] = from_right<T>(R0.x[0], hx[0], L.lane);
        vd.a[1][2] = from_right<T>(R0.d[0], hd[0], L.lane);
        vx.a[1][0].y = from_left<T>(R0.x[0].y, hx[0].y, L.lane);
        vd.a[1][0].y = from_left<T>(R0.d[0].y, hd[0].y, L.lane);
        vx.a[0][1].x = xm_ax;
        vd.a[0][1].x = dm_ax;
        vx.a[2][1] = Rp.x[0];
        vd.a[2][1] = Rp.d[0];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            vx.p[c][1][1] = R0.x[1 + c];
            vd.p[c][1][1] = R0.d[1 + c];
            vx.p[c][1][2] = from_right<T>(R0.x[1 + c], hx[1 + c], L.lane);
            vd.p[c][1][2] = from_right<T>(R0.d[1 + c], hd[1 + c], L.lane);
            vx.p[c][2][1] = Rp.x[1 + c];
            vd.p[c][2][1] = Rp.d[1 + c];
        }
        bool inner = false;
        if constexpr (std::is_same<T, double>::value) inner = __all_sync(FULL_MASK, !L.cok || R0.m == 0xffffu);
        links |= inner && !(PS && S.per_site);
        if (L.cok) {
            if (PS && S.per_site) pp.load_pass_site(S, L.gi, j, s);
            if constexpr (!WIDE) sum.zero();
            if (inner) {
                if constexpr (std::is_same<T, double>::value) {
                    if (PS && S.per_site)
                        site_poly<T, NC>(pack_view(vx), pack_view(vd), pp, OnesPerSite(), 1, f.poly_compat, S.thin_film, sum);
                    else
                        site_poly<T, NC>(pack_view(vx), pack_view(vd), pp, Ones(), 0, f.poly_compat, S.thin_film, sum);
                }
            } else {
                Wts<T> w;
                w.load(R0.m);
                site_poly<T, NC>(pack_view(vx), pack_view(vd), pp, w, PS && S.per_site, f.poly_compat, S.thin_film, sum);
            }
            if constexpr (!WIDE) {
                T o[5];
                sum.total(pp, false, f.poly_compat, o);
#pragma unroll
                for (int k = 0; k < 5; ++k) v[k] += o[k];
            }
        }
        if constexpr (!ONE)
            if (--left == 0 || r + 1 == rows) {
                if constexpr (WIDE) {
                    sum.total(pp, links, f.poly_compat, v);
                    sum.zero();
                    links = false;
                }
                store_sums<5>(v, sc, slot);
                if constexpr (!WIDE) v[0] = v[1] = v[2] = v[3] = v[4] = (T)0;
                slot += S.tiles_x;
                left = S.grows;
            }
        xm_ax = R0.x[0].x;
        dm_ax = R0.d[0].x;
        R0 = Rp;
    }
    // the halo copy of the row below the tile may still be in flight: complete it before the
    // ring can be reused (the fused kernel runs more tiles in the same block)
    cp_async_wait_groups<0>();
    if constexpr (ONE) {
        if constexpr (WIDE) sum.total(pp, links, f.poly_compat, v);
        store_sums<5>(v, sc, slot);
    }
    const int tpi = S.tiles_x * S.stiles_y;
    double tot[5];
    const bool fin = finish_image<5>(sc, S.part_base + tr.n * S.groups, S.groups, tpi, img, tot);
    if (fin) {
        if (L.lane == 0) {
#pragma unroll
            for (int k = 0; k < 5; ++k) coef[k] = tot[k] * S.ud.dx2;
            sc.fenergy[img] = coef[0];
#pragma unroll
            for (int k = 0; k < 4; ++k) sc.poly[4 * img + k] = coef[1 + k];
        }
        __syncwarp();
        const double alpha = line_search<store_t<T>>(coef, sc, f.ls_exact);
        if (L.lane == 0) {
            sc.alpha[img] = alpha;
            sc.alpha_pend[img] = alpha;
        }
        __syncwarp();
    }
    return fin;
}

template <class T, int NC, bool ONE, bool PS = true>
__global__ void __launch_bounds__(NTS, (StripBlocks<T, NC, ONE>::dir)) k_dir_poly_s(const __grid_constant__ batch_t<ONE> bt,
                                                                      int tile0, Scalars sc, StepFlags f)
{
    __shared__ __align__(16) DirRing<T, NC> ring;
    __shared__ double coef[5];
    dir_tile<T, NC, ONE, PS>(bt, strip_tile<ONE>(bt, tile0 + (int)blockIdx.x), sc, f, ring, coef);
}

// ------------------------------------------------------------ fused steps
// `steps` NLCG steps of one launch's tiles in a single persistent launch.
// Work items are (step, pass, tile) in that order, handed out by a global
// counter.  The direction pass of an image needs only that image's
// gradient pass of the same step, and the next gradient pass of an image
// needs only its direction pass (the step alpha), so an item waits on a
// per-image stage counter instead of a kernel boundary: stage = 2k + 1 once
// the gradient pass of step k finished the image, 2k + 2 once its
// direction pass did.  An item depends only on items handed out before it,
// and an item is only taken by a running block, so the waits always end;
// each is still bounded, and a wait that runs out sets status[0] and
// ends its block.
//
// A small string's pass is a chain of latencies (67 x 61 sites, 9 images: 8 us,
// of which the rows are 1.3): the wait's poll, three rows of loads, two rows of
// arithmetic, the strip's sums and ticket, the image's sums over its strips,
// the step, the publication.  So there is one fence in each of the last two
// and none in the wait, the image's partials are loaded four strips at a time,
// the stages lie a line apart and no more blocks run than a pass has strips
// (more of them only poll).  Ten steps: 293 us before these, 200 with them;
// 64 x 64 x 16 of two components in FP64 675 -> 632 with its reparametrization.

// Step plan of a fused launch: the buffers and gradient slot of step k
// follow from those of step 0 as the separate launches toggle them.
struct StepPlan {
    int xi0, di0, it0;   // x and d buffers read by step 0; iteration number of step 0
    StepFlags base;      // use_cg, maxwell and the line-search options
    __device__ __forceinline__ StepFlags step(int k) const
    {
        StepFlags f = base;
        f.gcur = (it0 + k) & 1;
        f.gprev = f.gcur ^ 1;
        f.xin = xi0 ^ (k & 1);
        f.xout = f.xin ^ 1;
        f.din = di0 ^ (k & 1);
        f.dout = f.din ^ 1;
        return f;
    }
};

// Lane 0 waits until stage >= need, polling at most max_polls times; false if
// the wait ran out.  Its acquire and the warp barrier order the whole warp's
// later loads after what the finishing block wrote.
__device__ __forceinline__ bool wait_stage(const unsigned *stage, unsigned need, unsigned max_polls, int *status)
{
    int ok = 1;
    if ((threadIdx.x & 31) == 0) {
        unsigned polls = 0, v;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(stage) : "memory");
            if (v >= need) break;
            if (++polls > max_polls) {
                atomicExch(status, 1);
                ok = 0;
                break;
            }
            __nanosleep(64);
        }
    }
    ok = __shfl_sync(FULL_MASK, ok, 0);
    __syncwarp();
    return ok != 0;
}

__device__ __forceinline__ void publish_stage(unsigned *stage, unsigned value)
{
    if ((threadIdx.x & 31) == 0) {
        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(stage), "r"(value) : "memory");
    }
    __syncwarp();
}

template <class T, int NC, bool ONE>
__global__ void __launch_bounds__(NTS, (StripBlocks<T, NC, ONE>::fused)) k_nlcg_s(const __grid_constant__ batch_t<ONE> bt, int tile0, int n_tiles, int steps,
                                            StepPlan plan, Scalars sc, unsigned long long *queue, unsigned *stage,
                                            unsigned max_polls)
{
    __shared__ __align__(16) GradRing<T, NC> gring;
    __shared__ __align__(16) DirRing<T, NC> dring;
    __shared__ double coef[5];
    const unsigned long long per_step = 2ull * (unsigned long long)n_tiles;
    const unsigned long long total = per_step * (unsigned long long)steps;
    for (;;) {
        unsigned long long item = 0;
        if ((threadIdx.x & 31) == 0) item = atomicAdd(queue, 1ull);
        item = __shfl_sync(FULL_MASK, item, 0);
        if (item >= total) return;
        const int k = (int)(item / per_step);
        const int r = (int)(item - (unsigned long long)k * per_step);
        const int pass = r >= n_tiles ? 1 : 0, u = r - pass * n_tiles;
        const StripRef tr = strip_tile<ONE>(bt, tile0 + u);
        const int img = bt.s[ONE ? 0 : tr.s].img_base + tr.n;
        const unsigned need = 2u * (unsigned)k + (unsigned)pass;
        if (need > 0 && !wait_stage(stage + (size_t)img * STAGE_STRIDE, need, max_polls, sc.status)) return;
        const StepFlags f = plan.step(k);
        if (pass == 0) {
            if (grad_tile<T, NC, ONE>(bt, tr, sc, f, gring)) publish_stage(stage + (size_t)img * STAGE_STRIDE, need + 1);
        } else {
            if (dir_tile<T, NC, ONE>(bt, tr, sc, f, dring, coef)) publish_stage(stage + (size_t)img * STAGE_STRIDE, need + 1);
        }
    }
}
