// kernels.cu -- CUDA kernels of libmepgl_gb300 (sm_103a).
//
// The NLCG iteration of the reference (nlcgSteps, mepgl/src/nlcg.cu:1462-1586:
// ~12 kernels, 4 two-level reductions, ~10 device-wide syncs per step) is two
// passes over the string here (strip.cuh):
//
//   gradient    x <- x + alpha_pend d   (the previous step's update, fused)
//               g  = dF/dx              (gradientPsi + gradientA)
//               |g|^2, g.(g - g_prev)   (gradientDensity + 2 sums)
//               last strip of an image: beta (computeStepDirection's scalar)
//   direction   d <- -g + beta d        (computeStepDirection)
//               quartic F(x + a d)      (polynomialExpansion + 2 sums)
//               last strip of an image: line search -> alpha (lineSearch)
//
// so one step reads x, d, g_prev, g (twice with halo, served mostly by L2)
// and writes x, g, d: 9 state-sized streams instead of the reference's ~20.
// x and d are ping-ponged because neighbouring strips read them as halo while
// they are being rewritten.
//
// Energies, gradients, adjoints and B, J of a string are formed by the same
// kind of walk (walk.cuh).
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "site_pack.cuh"

namespace mepgl {

// Resident single-warp blocks per SM asked of ptxas for the strip kernels
// (registers per thread: 65536 / (32 x blocks)).  FP64 and float-float strips
// hold twice the registers of FP32 ones; at 12 blocks they spill: a
// float-float step of the 256 x 256 string took 2.1 ms instead of 1.5, FP64
// gained nothing.  The passes of several one-component FP32 strings take 122
// registers if they may (16 blocks): ten steps of the 16 strings then take 17.9 ms,
// with 20, 22, 24 blocks 17.7, 16.8, 16.0.
#ifndef MEPGL_MINB_STRIP_GRAD
#define MEPGL_MINB_STRIP_GRAD 16
#endif
#ifndef MEPGL_MINB_STRIP_DIR
#define MEPGL_MINB_STRIP_DIR 16
#endif
#ifndef MEPGL_MINB_STRIP_DIR_SWEEP
#define MEPGL_MINB_STRIP_DIR_SWEEP 24
#endif
#ifndef MEPGL_MINB_STRIP_GRAD_SWEEP
#define MEPGL_MINB_STRIP_GRAD_SWEEP 24
#endif
#ifndef MEPGL_MINB_STRIP_FUSED
#define MEPGL_MINB_STRIP_FUSED 12
#endif
#ifndef MEPGL_MINB_STRIP_F64
#define MEPGL_MINB_STRIP_F64 8
#endif
template <class T, int NC, bool ONE> struct StripBlocks {
    static constexpr int grad = MEPGL_MINB_STRIP_F64, dir = MEPGL_MINB_STRIP_F64, fused = MEPGL_MINB_STRIP_F64;
};
template <int NC, bool ONE> struct StripBlocks<float, NC, ONE> {
    static constexpr int grad = NC == 1 && !ONE ? MEPGL_MINB_STRIP_GRAD_SWEEP : MEPGL_MINB_STRIP_GRAD,
                         fused = MEPGL_MINB_STRIP_FUSED,
                         dir = NC == 1 && !ONE ? MEPGL_MINB_STRIP_DIR_SWEEP : MEPGL_MINB_STRIP_DIR;
};
// Fused steps only for batches of at most this many waves of the pass kernels
// (beyond that the boundaries cost little; FP32 pass kernels hold more warps)
#ifndef MEPGL_FUSE_WAVES
#define MEPGL_FUSE_WAVES 4
#endif
#ifndef MEPGL_FUSE_WAVES_F64
#define MEPGL_FUSE_WAVES_F64 16
#endif

int fuse_waves(int precision) { return precision == 1 ? MEPGL_FUSE_WAVES_F64 : MEPGL_FUSE_WAVES; }

// Rows per strip.  A strip walks its rows one after the other, so a string
// with fewer strips than the GPU holds warps waits on a few long walks: ten
// FP32 steps of 67 x 61 x 9 sites took 865 us with 40-row strips (54 of
// them), 300 us with 2-row ones.  A long strip reads its two halo rows less
// often; past 40 rows (FP32) the fused launch's per-image waits cost more
// than that saves, and past 16 (FP64) nothing is gained, the passes being
// bound by arithmetic.  So the rows shrink from the cap in proportion once a
// batch has fewer strips than FILL per cent of the resident warps (ten steps
// of 128 x 128 x 24 sites, one / two components, at 50, 100, 150, 200, 300 %:
// FP32 389 / 508, 341 / 392, 316 / 347, 360 / 354, 359 / 403 us; FP64 3431 /
// 6027, 2407 / 4279, 2329 / 4143, 2341 / 4154, 2397 / 4216 us; FP32 256 x
// 256 x 40 loses 3 % from 150 on), down to the fewest rows that still gain.
// Float-float strips are bound by issue, and a second wave of them costs more
// than long ones: four steps of 128 x 128 x 24 take 447 / 845 us at 80 % (one
// wave of 12 rows), 613 / 1029 at 110 %, 522 / 903 at 150 %.  So a string of
// one to one and a half waves of the most rows takes up to half as many more and
// is one wave (ten steps, two components: 200 x 160 x 24 4.2 -> 3.4 ms, 40 x 1000
// x 10 3.1 -> 2.2).
#ifndef MEPGL_STRIP_ROWS_F32
#define MEPGL_STRIP_ROWS_F32 40
#endif
#ifndef MEPGL_STRIP_ROWS_F64
#define MEPGL_STRIP_ROWS_F64 16
#endif
#ifndef MEPGL_STRIP_FILL_F32
#define MEPGL_STRIP_FILL_F32 125
#endif
#ifndef MEPGL_STRIP_FILL_F64
#define MEPGL_STRIP_FILL_F64 150
#endif
#ifndef MEPGL_STRIP_ROWS_FF
#define MEPGL_STRIP_ROWS_FF 16
#endif
#ifndef MEPGL_STRIP_FILL_FF
#define MEPGL_STRIP_FILL_FF 80
#endif
int strip_rows_cap(int precision, int paired)
{
    return precision == 0 ? MEPGL_STRIP_ROWS_F32 : paired ? MEPGL_STRIP_ROWS_FF : MEPGL_STRIP_ROWS_F64;
}

// ny rows in strips of equal height: `cap` rows, fewer (`least` at least) where
// `tiles` strips of cap rows are fewer than `want`
static int equal_rows(int ny, int cap, int least, long tiles, long want)
{
    long rows = tiles < want ? cap * tiles / want : cap;
    if (rows < least) rows = least;
    const long k = (ny + rows - 1) / rows;
    return (int)((ny + k - 1) / k);
}

int strip_rows(int precision, int paired, int ny, long columns, long tiles, int slots)
{
    const int cap = strip_rows_cap(precision, paired);
    if (paired && tiles > slots && 2 * tiles <= 3L * slots) {
        const long k = std::max(1L, slots / columns), rows = (ny + k - 1) / k;   // k strips a column: one wave
        if (k * columns <= slots && 2 * rows <= 3 * cap) return (int)rows;
        return equal_rows(ny, cap, 1, tiles, 3L * slots / 2);
    }
    const int fill = precision == 0 ? MEPGL_STRIP_FILL_F32 : paired ? MEPGL_STRIP_FILL_FF : MEPGL_STRIP_FILL_F64;
    return equal_rows(ny, cap, precision == 0 ? 2 : 1, tiles, (long)slots * fill / 100);
}

#ifndef MEPGL_WALK_ROWS_F32
#define MEPGL_WALK_ROWS_F32 8
#endif
#ifndef MEPGL_WALK_ROWS_F64
#define MEPGL_WALK_ROWS_F64 8
#endif
static_assert(MEPGL_WALK_ROWS_F32 <= 8, "a lane adds up its rows in float");
int walk_rows(int precision, int ny, long columns, int sms)
{
    const int cap = precision == 0 ? MEPGL_WALK_ROWS_F32 : MEPGL_WALK_ROWS_F64;
    return equal_rows(ny, cap, precision == 0 ? 2 : 1, columns * ((ny + cap - 1) / cap), (long)sms * 16);
}

cudaError_t upload_mask_tables()
{
    static MaskTable<float> f;
    static MaskTable<double> d;
    build_mask_table(f);
    build_mask_table(d);
    cudaError_t e = cudaMemcpyToSymbol(c_mask_f, &f, sizeof(f));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_mask_d, &d, sizeof(d));
    return e;
}

namespace {

// Asynchronous copy of one element to shared memory, zero-filled where it is
// not valid.
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src, bool valid)
{
    const int n = valid ? BYTES : 0;
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(n)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES),
                     "r"(n)
                     : "memory");
}

// Per-site strings: the fields at the four neighbours of site s = (i, j).  FP32
// loads them ahead of the site's parameters (PackParams::load_site); the wider types
// where they are used (held over the divisions they cost FP64 gradients 5 %).
template <class T>
struct FieldSites {
    T u, d, r, l;
    static constexpr bool ahead = std::is_same<T, float>::value;
    template <class At>
    __device__ __forceinline__ void take(const StringDesc &S, int i, int j, int s, const At &at)
    {
        u = at(j + 1 < S.ny ? s + S.nx : s);
        d = at(j > 0 ? s - S.nx : s);
        r = at(i + 1 < S.nx ? s + 1 : s);
        l = at(i > 0 ? s - 1 : s);
    }
    __device__ __forceinline__ void load(const StringDesc &S, int i, int j, int s)
    {
        if constexpr (ahead) take(S, i, j, s, [&](int n) { return static_cast<const T *>(S.ph)[n]; });
    }
};

// (h + h_neighbour) dx of the four neighbours of site s = (i, j), near loaded.
// PAIRS: of a float-float pass; PS: the string may have per-site parameters.
template <class T, int NC, bool PAIRS = false, bool PS = true>
__device__ __forceinline__ FieldSums<T> field_sums(const StringDesc &S, const PackParams<T, NC> &pp, FieldSites<T> near, int i,
                                                   int j, int s)
{
    const T hs = pp.hd + pp.hd;
    FieldSums<T> f{hs, hs, hs, hs};
    if (PS && S.per_site) {
        if constexpr (!FieldSites<T>::ahead) near.take(S, i, j, s, [&](int n) {
            if constexpr (PAIRS && std::is_same<T, ff>::value) return pair_site(S.pairs.h, n);
            else return from_store<T>(static_cast<const store_t<T> *>(S.ph)[n]);
        });
        const T dx = S.template u<T>().dx;
        f.u = pp.hd + near.u * dx;
        f.d = pp.hd + near.d * dx;
        f.r = pp.hd + near.r * dx;
        f.l = pp.hd + near.l * dx;
    }
    return f;
}

// --------------------------------------------------------------- line search
// Quartic A + B x + C x^2 + D x^3 + E x^4 evaluated in round-to-nearest
// double without contraction, in the oracle's order.
__device__ __forceinline__ double quartic_rn(const double *c, double x)
{
    const double x2 = __dmul_rn(x, x);
    double f = __dmul_rn(c[4], __dmul_rn(x2, x2));
    f = __dadd_rn(f, __dmul_rn(__dmul_rn(__dmul_rn(c[3], x), x), x));
    f = __dadd_rn(f, __dmul_rn(__dmul_rn(c[2], x), x));
    f = __dadd_rn(f, __dmul_rn(c[1], x));
    return __dadd_rn(f, c[0]);
}

// lineSearch (nlcg.cu:1398-1445) by one warp: first p in 1..2000 with
// f(x_p) > f(x_{p-1}) (else 2000); alpha = x_p / m in the working precision.
//
// Every FP64 instruction of a lone warp takes 64 clocks here whatever its
// lanes do, and the grid starts at 1e-10, some 800 points below a usual
// step: a scan from its start is 26 rounds of 32 points, 10 us.  So the
// scan starts at the last multiple of 64 up to which the slope stays below
// B / 2 (|B| at least twice the other terms of the derivative): there the
// polynomial part falls by more than 1 % of |B| x from point to point, its
// rounding is 1e-15 of that, and adding the energy rounds monotonically, so
// no f(x_p) > f(x_{p-1}) is passed over.
template <class T>
__device__ double line_search_scan(const double *c, const double *xt)
{
    const int lane = threadIdx.x & 31;
    int p0 = 0;
    {
        const double x = xt[64 * lane];
        const bool falls = c[1] <= -1e-200 && x * (4 * fabs(c[2]) + x * (6 * fabs(c[3]) + x * 8 * fabs(c[4]))) <= -c[1];
        const unsigned bal = ~__ballot_sync(0xffffffffu, falls);
        const int n = bal ? __ffs(bal) - 1 : 32;   // leading points that fall
        if (n > 0) p0 = 64 * (n - 1);
    }
    double f_prev = quartic_rn(c, xt[p0]);
    int found = 0;
    for (int base = p0 + 1; base <= 2000; base += 32) {
        const int p = base + lane;
        const double fp = p <= 2000 ? quartic_rn(c, xt[p]) : 0.0;
        double fl = __shfl_up_sync(0xffffffffu, fp, 1);
        if (lane == 0) fl = f_prev;
        const unsigned bal = __ballot_sync(0xffffffffu, p <= 2000 && fp > fl);
        if (bal) { found = base + __ffs(bal) - 1; break; }
        f_prev = __shfl_sync(0xffffffffu, fp, 31);
    }
    const int j = found ? found : 2000;
    const T m = (T)1.025f;
    return (double)((T)xt[j] / m);
}

// Smallest positive root of the quartic's derivative f = a0 + a1 x + a2 x^2 +
// a3 x^3 with a0 < 0 < a3 (its first local minimum: f crosses zero upwards
// there).  Newton's method in float, x and f in units (powers of two) that
// make the constant about -1 and every other coefficient 1 at most, from a
// point from which it converges monotonically: f has its turning points at c1
// <= c2 where D = a2^2 - 3 a1 a3 > 0 and its inflection at cm.  Left of cm it
// is concave: if f rises from 0 to its root there, Newton from 0 stays left of
// it.  Right of cm it is convex: Newton from a bound above the root stays right
// of it.  Then steps in double with that slope, each of which gains about five
// digits.  False where a case is out of the ordinary (far out of float's range,
// a turning point that float cannot tell from a root, steps that shrink by less
// than 1000); the caller then takes the closed form.
__device__ bool first_minimum(double a0, double a1, double a2, double a3, double &root)
{
    if (!(a0 < 0.0)) return false;
    if (a3 == 0.0 && a2 == 0.0) {
        root = -a0 / a1;
        return a1 > 0.0;
    }
    if (!(a3 > 0.0)) return false;
    auto exponent = [](double v) { return ((__double2hiint(v) >> 20) & 0x7ff) - 1023; };
    auto pow2 = [](int k) { return __hiloint2double((k + 1023) << 20, 0); };
    const int e0 = exponent(a0), k1 = e0 - exponent(a1), k2 = (e0 - exponent(a2)) >> 1, k3 = (e0 - exponent(a3)) / 3 - 1;
    const int ex = min(k1, min(k2, k3));
    if (abs(e0) > 300 || abs(ex) > 200) return false;
    const float A0 = (float)(a0 * pow2(-e0)), A1 = (float)(a1 * pow2(ex - e0)), A2 = (float)(a2 * pow2(2 * ex - e0)),
                A3 = (float)(a3 * pow2(3 * ex - e0));
    const float b2 = 2.0f * A2, b3 = 3.0f * A3;
    float x = 0.0f;
    if (k1 == ex && A1 > 0.0f && fabsf(A2) <= 0x1p-8f && A3 <= 0x1p-8f) {
        x = -A0 / A1;   // nearly linear: 1 <= A1 < 2, so that f rises from 0 to 4 by more than |A0| < 2
    } else {
        const float p = A2 * A2, q = A1 * b3, D = p - q;
        if (!(b3 > 1e-25f)) return false;
        const float cm = -A2 / b3, fm = A0 + cm * (A1 + cm * (A2 + cm * A3));
        const float noise = 1e-6f * (fabsf(A0) + fabsf(cm) * (fabsf(A1) + fabsf(cm) * (fabsf(A2) + fabsf(cm) * A3)));
        if (fabsf(D) <= 1e-6f * (p + fabsf(q)) && !(fabsf(fm) > noise)) return false;
        bool right = fm < 0.0f;   // monotone f: right of the inflection if it is still negative there
        if (D > 0.0f) {
            // c1 > 0 needs a2 < 0 (else it is the negative one of two roots, or both are negative)
            const float c1 = A2 < 0.0f ? A1 / (sqrtf(D) - A2) : -1.0f;
            const float f1 = A0 + c1 * (A1 + c1 * (A2 + c1 * A3));
            if (c1 > 0.0f && !(fabsf(f1) > 1e-6f * (fabsf(A0) + c1 * (fabsf(A1) + c1 * (fabsf(A2) + c1 * A3))))) return false;
            right = !(c1 > 0.0f && f1 > 0.0f);
        } else if (!right && !(A1 > 0.0f)) {
            return false;
        }
        if (right) {
            // x - cm <= max(sqrt(2 |P|), cbrt(2 |Q|)) of the depressed cubic z^3 + P z + Q
            const float z = 1.0001f * fmaxf(sqrtf(2.0f * fabsf(D) / (b3 * A3)), cbrtf(2.0f * fabsf(fm) / A3));
            if (!(z > 1e-30f && z < 1e30f)) return false;
            x = cm + z;
            if (!(x > 0.0f)) return false;
        }
    }
    float r = 0.0f;   // 1 / slope
    for (int it = 0; it < 24; ++it) {
        const float f = A0 + x * (A1 + x * (A2 + x * A3)), d = A1 + x * (b2 + x * b3);
        if (!(d > 1e-30f && d < 1e30f)) return false;
        r = 1.0f / d;
        const float dx = f * r;
        x -= dx;
        if (fabsf(dx) <= 1e-4f * fabsf(x)) break;
    }
    const double rs = pow2(ex - e0) * (double)r;
    double y = (double)x * pow2(ex), last = fabs(y);
    for (int it = 0; it < 8; ++it) {
        const double dy = (a0 + y * (a1 + y * (a2 + y * a3))) * rs, ay = fabs(dy);
        y -= dy;
        if (ay <= 1e-13 * fabs(y)) {
            root = y;
            return y > 0.0;
        }
        if (!(ay <= 1e-3 * last)) return false;
        last = ay;
    }
    return false;
}

// Exact version of the reference's scan: the first local minimum of the
// quartic downhill from alpha = 0, i.e. the smallest positive root of the
// cubic derivative with positive curvature (closed-form roots, two Newton
// steps each); `fallback` (the scan's answer) when p'(0) >= 0 or none exists.
__device__ double line_search_exact(const double *c, double fallback)
{
    const double a3 = 4 * c[4], a2 = 3 * c[3], a1 = 2 * c[2], a0 = c[1];
    double roots[3];
    int nr = 0;
    if (fabs(a0) + fabs(a1) + fabs(a2) + fabs(a3) == 0) return fallback;
    if (fabs(a3) > 1e-300) {
        const double A2 = a2 / a3, A1 = a1 / a3, A0 = a0 / a3;
        const double Q = (3 * A1 - A2 * A2) / 9, R = (9 * A2 * A1 - 27 * A0 - 2 * A2 * A2 * A2) / 54;
        const double disc = Q * Q * Q + R * R;
        if (disc >= 0) {
            const double sd = sqrt(disc);
            roots[nr++] = -A2 / 3 + cbrt(R + sd) + cbrt(R - sd);
        } else {
            const double th = acos(R / sqrt(-Q * Q * Q)), r = 2 * sqrt(-Q);
            roots[nr++] = r * cos(th / 3) - A2 / 3;
            roots[nr++] = r * cos((th + 2 * M_PI) / 3) - A2 / 3;
            roots[nr++] = r * cos((th + 4 * M_PI) / 3) - A2 / 3;
        }
    } else if (fabs(a2) > 1e-300) {
        const double disc = a1 * a1 - 4 * a2 * a0;
        if (disc >= 0) {
            const double sq = sqrt(disc), qq = -0.5 * (a1 + (a1 >= 0 ? sq : -sq));
            if (qq != 0) { roots[nr++] = qq / a2; roots[nr++] = a0 / qq; }
        }
    } else if (a1 != 0) {
        roots[nr++] = -a0 / a1;
    }
    // the scan stops at the first increase: not a descent direction -> its answer
    if (!(a0 < 0)) return fallback;
    double best = -1;
    for (int t = 0; t < nr; ++t) {
        double r = roots[t];
        for (int it = 0; it < 2; ++it) {
            const double dp = a0 + r * (a1 + r * (a2 + r * a3)), ddp = a1 + r * (2 * a2 + r * 3 * a3);
            if (ddp != 0) r -= dp / ddp;
        }
        const double ddp = a1 + r * (2 * a2 + r * 3 * a3);
        if (!(r > 0) || !(ddp > 0)) continue;
        if (best < 0 || r < best) best = r;   // first local minimum downhill from 0
    }
    return best < 0 ? fallback : best;
}

// The step of one image from its quartic, by one warp: the scan's answer, or
// the exact first minimum (the scan's where there is none).  T: stored
// precision, whose grid and rounding the scan follows.
template <class T>
__device__ double line_search(const double *coef, const Scalars &sc, int exact)
{
    if (exact) {
        double x;
        if (first_minimum(coef[1], 2 * coef[2], 3 * coef[3], 4 * coef[4], x)) return x;
    }
    const double alpha = line_search_scan<T>(coef, sizeof(T) == 8 ? sc.xtab_d : sc.xtab_f);
    return exact ? line_search_exact(coef, alpha) : alpha;
}

// ------------------------------------------------------------------ kernels
#include "strip.cuh"

#include "walk.cuh"

// x += alpha_pend[image] d over every string of a batch: block (chunk, image
// of the batch, field).  W: the compute type of the NLCG passes that wrote d
// (ff: d holds float-float pairs, the update runs in double on their values).
template <class T, class W, bool ONE>
__global__ void __launch_bounds__(NT) k_apply_update(const __grid_constant__ batch_t<ONE> bt, const double *alpha_pend,
                                                     int img0, int xbuf, int dbuf)
{
    const int img = img0 + blockIdx.y;
    int si = 0;
    if (!ONE)
        for (int k = 1; k < bt.n; ++k)
            if (img >= bt.s[k].img_base) si = k;
    const StringDesc &S = bt.s[si];
    const T a = (T)alpha_pend[img];
    if (a == (T)0) return;
    const long M = (long)S.nx * S.ny, off = (long)(img - S.img_base) * M;
    vec2_t<T> *x = static_cast<vec2_t<T> *>(S.x[xbuf][blockIdx.z]) + off;
    const vec2_t<T> *d = static_cast<const vec2_t<T> *>(S.d[dbuf][blockIdx.z]) + off;
    for (long p = blockIdx.x * (long)NT + threadIdx.x; p < M; p += (long)gridDim.x * NT) {
        vec2_t<T> v = x[p];
        vec2_t<T> dd;
        if constexpr (std::is_same<W, ff>::value) {
            const ff2 w = loadw<ff>(d + p);
            dd.x = to_double(w.x);
            dd.y = to_double(w.y);
        } else {
            dd = d[p];
        }
        v.x = v.x + a * dd.x;
        v.y = v.y + a * dd.y;
        x[p] = v;
    }
}

// NLCG history of every image: |g|^2 = infinity (the next beta is 0, and the
// passes then read neither the old gradient nor the old direction, whose
// contents no longer matter), no step pending, scalars zero.
__global__ void k_reset_history(Scalars sc, int n_images)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= n_images) return;
    sc.gn0[n] = sc.gn1[n] = INFINITY;
    sc.gdg[n] = sc.beta[n] = sc.alpha[n] = sc.alpha_pend[n] = sc.fenergy[n] = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) sc.poly[4 * n + k] = 0.0;
}

// |g|^2 = infinity for images [first, last).
__global__ void k_restart_cg(Scalars sc, int first, int last)
{
    const int n = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (n < last) sc.gn0[n] = sc.gn1[n] = INFINITY;
}

// PairSites' arrays of one component, or (a alone) of the field.
__global__ void __launch_bounds__(NT) k_pair_sites(const double *a, const double *b, const double *mx, const double *my, float2 *out,
                                                   long M)
{
    const long i = blockIdx.x * (long)NT + threadIdx.x;
    if (i >= M) return;
    auto put = [&](int k, double v) {
        const ff w = to_ff(v);
        out[k * M + i] = make_float2(w.hi, w.lo);
    };
    put(0, a[i]);
    if (!b) return;
    put(1, b[i]);
    put(2, 0.5 / mx[i]);
    put(3, 0.5 / my[i]);
    put(4, a[i] / b[i]);
}

// Fields x between double pairs and float-float pairs, in place (an ff2
// fills the 16 bytes of a double2).  A double holds a float-float pair that
// the passes wrote exactly, so a round trip returns the same doubles.
template <bool TO_PAIRS>
__global__ void __launch_bounds__(NT) k_x_format(double2 *x, long n)
{
    for (long i = blockIdx.x * (long)NT + threadIdx.x; i < n; i += (long)gridDim.x * NT) {
        if (TO_PAIRS) {
            const double2 v = x[i];
            ff2 w;
            w.x = to_ff(v.x);
            w.y = to_ff(v.y);
            storew<ff>(x + i, w);
        } else {
            const ff2 w = loadw<ff>(x + i);
            x[i] = make_double2(to_double(w.x), to_double(w.y));
        }
    }
}

// Arc length from stored arrays: squared image-to-image distance over every
// site (no mask, no dx^2; interpolation.cu:39-92).  Block (bx, n) covers sites
// [bx * NT * ARC_SPT, ...) of image n against image n - 1: each thread issues
// all its loads of both images, then adds them in the fixed order (site,
// field, component), so each (image, site block) partial is the same sum
// one walk through the images would give.
constexpr int ARC_SPT = 4;

template <class T>
__global__ void __launch_bounds__(NT) k_arc_partial(const T *__restrict__ f0, const T *__restrict__ f1,
                                                    const T *__restrict__ f2, int w0, int w1, int w2, long sites,
                                                    double *part)
{
    __shared__ double red[NT / 32];
    const T *fs[3] = {f0, f1, f2};
    const int ws[3] = {w0, w1, w2};
    const int n = blockIdx.y;
    const long base = (long)blockIdx.x * NT * ARC_SPT + threadIdx.x;
    T acc = 0;
    if (n > 0) {
        T cur[3][ARC_SPT][2], prv[3][ARC_SPT][2];
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int q = 0; q < ARC_SPT; ++q) {
                const long s = base + (long)q * NT;
                cur[f][q][0] = cur[f][q][1] = prv[f][q][0] = prv[f][q][1] = 0;
                if (!fs[f] || s >= sites) continue;
                if (ws[f] == 2) {   // one vector load per site and image
                    const vec2_t<T> *v = reinterpret_cast<const vec2_t<T> *>(fs[f]);
                    const vec2_t<T> c = v[(long)n * sites + s], p = v[(long)(n - 1) * sites + s];
                    cur[f][q][0] = c.x;
                    cur[f][q][1] = c.y;
                    prv[f][q][0] = p.x;
                    prv[f][q][1] = p.y;
                } else {
                    cur[f][q][0] = fs[f][(long)n * sites + s];
                    prv[f][q][0] = fs[f][(long)(n - 1) * sites + s];
                }
            }
#pragma unroll
        for (int q = 0; q < ARC_SPT; ++q) {
            if (base + (long)q * NT >= sites) continue;
            T d2 = 0;
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                if (!fs[f]) continue;
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    if (w >= ws[f]) continue;
                    d2 += (cur[f][q][w] - prv[f][q][w]) * (cur[f][q][w] - prv[f][q][w]);
                }
            }
            acc += d2;
        }
    }
    const T vv[1] = {acc};
    double tot[1];
    block_sum<1>(vv, tot, red);
    if (threadIdx.x == 0) part[(size_t)n * gridDim.x + blockIdx.x] = tot[0];
}

// ------------------------------------------------------- initial strings
// Counter-based Gaussian noise: Philox4x32-10 (Salmon, Moraes, Dror and
// Shaw, "Parallel random numbers: as easy as 1, 2, 3", SC 2011) keyed by the
// seed and counted by (image, site, component), then Box-Muller.  Each site
// draws the same numbers whatever the launch shape.
__device__ __forceinline__ void philox_round(uint32_t (&c)[4], uint32_t (&k)[2])
{
    const uint64_t p0 = (uint64_t)0xD2511F53u * c[0], p1 = (uint64_t)0xCD9E8D57u * c[2];
    const uint32_t h0 = (uint32_t)(p0 >> 32), l0 = (uint32_t)p0, h1 = (uint32_t)(p1 >> 32), l1 = (uint32_t)p1;
    c[0] = h1 ^ c[1] ^ k[0];
    c[1] = l1;
    c[2] = h0 ^ c[3] ^ k[1];
    c[3] = l0;
    k[0] += 0x9E3779B9u;
    k[1] += 0xBB67AE85u;
}

__device__ __forceinline__ void philox4x32_10(uint32_t (&c)[4], uint64_t seed)
{
    uint32_t k[2] = {(uint32_t)seed, (uint32_t)(seed >> 32)};
#pragma unroll
    for (int r = 0; r < 10; ++r) philox_round(c, k);
}

// two standard normals from the counter (n, s, component)
__device__ __forceinline__ void normal_pair(uint64_t seed, int n, long s, int comp, double &z0, double &z1)
{
    uint32_t c[4] = {(uint32_t)s, (uint32_t)((unsigned long long)s >> 32), (uint32_t)n, (uint32_t)comp};
    philox4x32_10(c, seed);
    // 53-bit uniforms in (0, 1]
    const double u1 = ((double)(((uint64_t)c[0] << 21) ^ (c[1] >> 11)) + 1.0) * 0x1.0p-53;
    const double u2 = (double)(((uint64_t)c[2] << 21) ^ (c[3] >> 11)) * 0x1.0p-53;
    const double r = sqrt(-2.0 * log(u1));
    double sn, cs;
    sincospi(2.0 * u2, &sn, &cs);
    z0 = r * cs;
    z1 = r * sn;
}

// The initial guess of the reference's StringBuilder (builder.py:107-189)
// for every image at once: per component |psi| = psi_abs * prod_v f(r_v),
// theta = sum_v w_v atan2(y - y_v, x - x_v) over the vortex tracks with a
// nonzero winding in that image, plus N(0, noise^2) on Re and Im, times the
// superconducting domain; A from the gauge of B_z times the computational
// domain.  f = tanh(-r^2) (the builder's profile) or tanh(r / sqrt 2).
// tracks: n_tracks x F x {x, y, winding, component} doubles.
template <class T>
__global__ void k_generate(vec2_t<T> *a, vec2_t<T> *p1, vec2_t<T> *p2, int nx, int ny, int F, int ncomp,
                           const int32_t *comp, const int32_t *sc, const double *tracks, int n_tracks, GuessParams g)
{
    const long M = (long)nx * ny;
    for (long e = blockIdx.x * (long)NT + threadIdx.x; e < M * F; e += (long)gridDim.x * NT) {
        const int n = (int)(e / M);
        const long s = e - (long)n * M;
        const int i = (int)(s % nx), j = (int)(s / nx);
        const double x = g.x0 + i * g.dx, y = g.y0 + j * g.dx;
        const double cm = comp[s] ? 1.0 : 0.0, scm = sc[s] ? 1.0 : 0.0;
        vec2_t<T> av;
        double ax = 0.0, ay = 0.0;
        if (g.gauge == 1) ax = -g.b_z * y;
        else if (g.gauge == 2) ay = g.b_z * x;
        else if (g.gauge == 3) { ax = -0.5 * g.b_z * y; ay = 0.5 * g.b_z * x; }
        av.x = (T)(ax * cm);
        av.y = (T)(ay * cm);
        a[e] = av;
        for (int c = 0; c < ncomp; ++c) {
            double mag = c == 0 ? g.psi_abs_1 : g.psi_abs_2, th = 0.0;
            for (int v = 0; v < n_tracks; ++v) {
                const double *t = tracks + ((size_t)v * F + n) * 4;
                if ((int)t[3] != c + 1 || t[2] == 0.0) continue;
                const double dxv = x - t[0], dyv = y - t[1], r2 = dxv * dxv + dyv * dyv;
                mag *= g.profile == 0 ? tanh(-r2) : tanh(sqrt(r2) * 0.70710678118654752440);
                th += t[2] * atan2(dyv, dxv);
            }
            double z0 = 0.0, z1 = 0.0;
            if (g.noise != 0.0) normal_pair(g.seed, n, s, c, z0, z1);
            double sn, cs;
            sincos(th, &sn, &cs);
            vec2_t<T> pv;
            pv.x = (T)((mag * cs + g.noise * z0) * scm);
            pv.y = (T)((mag * sn + g.noise * z1) * scm);
            (c == 0 ? p1 : p2)[e] = pv;
        }
    }
}

// Winding sum of one field per image (compute_winding, gl_utils.py:10-41):
// around the rectangle `inset` sites inside the lattice edge, counter-
// clockwise from the lower-left corner, sum of the linearised phase steps
// (u dv - v du) / (u^2 + v^2) taken at the start of each step (2 pi per
// vortex enclosed, approximately).  The loop visits (W - 1) steps along
// each horizontal side and (H - 1) along each vertical side.
template <class T>
__global__ void k_winding(const vec2_t<T> *__restrict__ psi, int nx, int ny, int F, int inset, double *out)
{
    __shared__ double red[NT / 32];
    const int W = nx - 2 * inset, H = ny - 2 * inset, i0 = inset, j0 = inset, i1 = nx - 1 - inset,
              j1 = ny - 1 - inset;
    const int L = 2 * (W - 1) + 2 * (H - 1);
    for (int n = blockIdx.x; n < F; n += gridDim.x) {
        const vec2_t<T> *pn = psi + (size_t)n * nx * ny;
        double v[1] = {0.0};
        for (int t = threadIdx.x; t < L; t += NT) {
            int ia, ja, ib, jb;
            if (t < W - 1) {
                ia = i0 + t; ja = j0; ib = ia + 1; jb = ja;
            } else if (t < (W - 1) + (H - 1)) {
                const int k = t - (W - 1);
                ia = i1; ja = j0 + k; ib = ia; jb = ja + 1;
            } else if (t < 2 * (W - 1) + (H - 1)) {
                const int k = t - (W - 1) - (H - 1);
                ia = i1 - k; ja = j1; ib = ia - 1; jb = ja;
            } else {
                const int k = t - 2 * (W - 1) - (H - 1);
                ia = i0; ja = j1 - k; ib = ia; jb = ja - 1;
            }
            const vec2_t<T> a = pn[ia + (size_t)nx * ja], b = pn[ib + (size_t)nx * jb];
            const double u = a.x, w = a.y, du = (double)b.x - u, dv = (double)b.y - w;
            v[0] += (u * dv - w * du) / (u * u + w * w);
        }
        double tot[1];
        block_sum<1>(v, tot, red);
        if (threadIdx.x == 0) out[n] = tot[0];
    }
}

// computeArcLength (interpolation.cu:126-140), first half: block (n, metric)
// adds image n's partials.
__global__ void k_arc_sum(const double *part_f, const double *part_jb, int nblocks, double *s_f, double *s_jb)
{
    __shared__ double red[NT / 32];
    const int n = blockIdx.x;
    const double *part = blockIdx.y ? part_jb : part_f;
    double v = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += NT) v += part[(size_t)n * nblocks + b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < NT / 32; ++k) v += red[k];
        (blockIdx.y ? s_jb : s_f)[n] = v;
    }
}

// Second half: cumulative sqrt, normalised so that s[F-1] = 1.  The square
// roots and the divisions (slow in FP64 here) run across the block; one
// thread adds in image order.  Strings of more than ARC_CUM_MAX images run
// it all in one thread.
//
// A string of zero or non-finite length (all images equal, or a non-finite
// field) has no arc length: the reference divides 0 by 0 there
// (interpolation.cu:126-140).  Here *bad is set and s becomes the uniform
// n / (F - 1), computed as the resample plan computes its output positions,
// so that a linear resample onto as many images copies every image exactly;
// the host reports the flag as an error.
constexpr int ARC_CUM_MAX = 4096;

__device__ __forceinline__ bool arc_total_ok(double t) { return t > 0.0 && t <= 1.7976931348623157e308; }

// By a whole block, for one or two metrics (s[1] null: one), whose additions
// run at the same time in the first threads of two warps; r: 2 F doubles of
// shared memory, or null (then everything in those threads).
__device__ void arc_cumulate(int F, double *const (&s)[2], int *bad, double *r)
{
    __shared__ double total[2];
    const int metrics = s[1] ? 2 : 1;
    if (F == 1) {     // a single image has no length to normalise
        if (threadIdx.x == 0)
            for (int m = 0; m < metrics; ++m) s[m][0] = 0.0;
        return;
    }
    if (r)
        for (int m = 0; m < metrics; ++m)
            for (int n = threadIdx.x; n < F; n += blockDim.x) r[m * F + n] = n == 0 ? 0.0 : sqrt(s[m][n]);
    __syncthreads();
    const int m = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0 && m < metrics) {
        double acc = 0.0;
        if (r) {
            for (int n = 1; n < F; ++n) {
                acc += r[m * F + n];
                r[m * F + n] = acc;
            }
        } else {
            s[m][0] = 0.0;
            for (int n = 1; n < F; ++n) {
                acc += sqrt(s[m][n]);
                s[m][n] = acc;
            }
        }
        total[m] = acc;
        if (!arc_total_ok(acc)) atomicExch(bad, 1);
    }
    __syncthreads();
    for (int k = 0; k < metrics; ++k) {
        const bool ok = arc_total_ok(total[k]);
        const double *from = r ? r + k * F : s[k];
        for (int n = threadIdx.x; n < F; n += blockDim.x) s[k][n] = ok ? from[n] / total[k] : (double)n / (double)(F - 1);
    }
}

__global__ void k_arc_cumulate(int F, double *s, int *bad, int use_smem)
{
    extern __shared__ double cum_sm[];
    double *const one[2] = {s, nullptr};
    arc_cumulate(F, one, bad, use_smem ? cum_sm : nullptr);
}

// Finiteness of the per-image scalars after a call's NLCG steps: the energy
// (constant term of the last line polynomial) and |g|^2 of the slot the
// last step wrote.  A NaN or infinite value (from non-finite fields, or a
// step that overflowed) counts into status[1]; status[2] keeps the first
// such image + 1.  The host reports them at its next synchronising call.
__global__ void k_check_scalars(const double *fenergy, const double *gn, int n_images, int *status)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= n_images) return;
    const double e = fenergy[n], g = gn[n];
    const double big = 1.7976931348623157e308;
    if (!(fabs(e) <= big) || !(g <= big)) {
        atomicAdd(status + 1, 1);
        atomicCAS(status + 2, 0, n + 1);
    }
}

// Redistribution plan: segment and weight per output image, and for the
// cubic spline the Forsythe-Malcolm-Moler matrix (buildHMatrix,
// interpolation.cu:252-290) factorised once by Gaussian elimination with
// partial pivoting (the LAPACK gtsv algorithm) for every site's system.  One
// block.
//
// What bounds it is the chain of dependent FP64 operations: an addition takes
// tens of clocks here, a division hundreds.  So the segments are found by
// bisection, one thread per output image, and the elimination's pivots come
// from the continuants p_q = d_q p_{q-1} - dl_q du_{q-1} p_{q-2} (a multiply-add
// per image; d'_q = p_q / p_{q-1} are then independent divisions), polished by
// two sweeps of d'_q = d_q - dl_q du_{q-1} / d'_{q-1}, each of which shrinks an
// error by dl_q du_{q-1} / d'_{q-1}^2: at most 1/4, except 1 at q = 1, where the
// first sweep leaves d'_0 = d_0 exact and the second d'_1.  Hence two.  If a pivot would have been exchanged, or one is not
// a normal number, the elimination runs as written.  With both
// cumulations before it, 32 images, cubic: 45 us -> 26; 64 images, linear: 34 us
// -> 14.  The arrays live in shared memory when they fit, else in the plan's
// global arrays (elimination by one thread).

// Shared-memory bytes of the plan kernel: s, h, dl, d, du, du2 and two more
// [F or F+1] as doubles; ipiv [F] and the segments [F_new] as ints.
__host__ __device__ inline size_t redist_plan_smem(int F, int F_new)
{
    return (size_t)(8 * F + 1) * sizeof(double) + (size_t)(F + F_new) * sizeof(int);
}

// Weight of the segment's end image.  A segment of zero length (two equal
// adjacent images, where the reference divides 0 by 0) takes its end image:
// both ends are the same state.
__device__ __forceinline__ double redist_weight(double num, double len) { return len != 0.0 ? num / len : 1.0; }

// Smallest k in [1, last] with e[k] >= x, else last (e does not decrease).
__device__ __forceinline__ int first_not_below(const double *e, double x, int last)
{
    int lo = 1, hi = last;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (e[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// gtsv's elimination, in place, by one thread.
__device__ void eliminate(int F, double *dl, double *d, double *du, double *du2, int *ipiv)
{
    for (int q = 0; q < F - 1; ++q) {
        const double sub = dl[q + 1];
        if (fabs(d[q]) >= fabs(sub)) {
            if (d[q] != 0) {
                const double l = sub / d[q];
                dl[q + 1] = l;
                d[q + 1] = d[q + 1] - l * du[q];
            } else {
                dl[q + 1] = 0;
            }
        } else {
            const double l = d[q] / sub;
            d[q] = sub;
            dl[q + 1] = l;
            const double tmp = du[q];
            du[q] = d[q + 1];
            d[q + 1] = tmp - l * d[q + 1];
            if (q < F - 2) {
                du2[q] = du[q + 1];
                du[q + 1] = -l * du[q + 1];
            }
            ipiv[q] = 1;
        }
    }
}

// s_f and s_jb hold squared distances, which become arc lengths first (the
// plan is made on s_use, one of the two).
__global__ void k_redist_plan(double *s_f, double *s_jb, const double *s_use, int *status, int F, int F_new, int cubic,
                              int spline, RedistPlan p, int use_smem)
{
    extern __shared__ double plan_sm[];
    const int t = threadIdx.x, nt = blockDim.x;
    double *const both[2] = {s_f, s_jb};
    arc_cumulate(F, both, status + STATUS_ARC, use_smem ? plan_sm : nullptr);
    __syncthreads();
    const double *s = s_use;
    double *h = p.h, *dl = p.dl, *d = p.d, *du = p.du, *du2 = p.du2, *w1 = nullptr, *w2 = nullptr;
    int *ipiv = p.ipiv, *kk = p.k;
    if (use_smem) {
        double *ss = plan_sm;
        h = ss + F;
        dl = h + F + 1;
        d = dl + F;
        du = d + F;
        du2 = du + F;
        w1 = du2 + F;
        w2 = w1 + F;
        ipiv = reinterpret_cast<int *>(w2 + F);
        kk = ipiv + F;
        for (int n = t; n < F; n += nt) ss[n] = s_use[n];
        s = ss;
        __syncthreads();
    }
    // h[n] = s[n] - s[n-1]; output positions n / (F_new - 1)
    for (int n = t; n <= F; n += nt) h[n] = n == 0 ? 0.0 : (n == F ? INFINITY : s[n] - s[n - 1]);
    __syncthreads();
    // Segment k ends at s[k].  The reference's cubic walks by running sums of h
    // (interpolation.cu:380-386), which are s again up to rounding; where theirs
    // ends below 1 it reads past its array, and the last image comes from the
    // wrong segment.  s itself ends at 1.
    for (int n = t; n < F_new; n += nt) {
        const double s_new = (double)n / (double)(F_new - 1);
        const int k = first_not_below(s, s_new, F - 1);
        const double start = k > 1 ? s[k - 1] : 0.0;
        kk[n] = k;
        p.k[n] = k;
        p.w[n] = redist_weight(s_new - start, cubic ? h[k] : (s[k] - s[k - 1]));
    }
    __syncthreads();
    if (!cubic) {
        if (use_smem)
            for (int n = t; n <= F; n += nt) p.h[n] = h[n];
        return;
    }
    for (int n = t; n < F; n += nt) {
        const bool ends = n == 0 || n == F - 1;
        dl[n] = n == 0 ? 0.0 : h[n];
        d[n] = n == 0 ? -h[1] : (n == F - 1 ? -h[F - 1] : 2 * (h[n] + h[n + 1]));
        du[n] = n == 0 ? h[1] : (ends ? 0.0 : h[n + 1]);
        du2[n] = 0.0;
        ipiv[n] = 0;
    }
    __syncthreads();
    bool done = false;
    if (use_smem) {
        // continuants p_q of the matrix times F: w1 = p_q, w2 = p_{q-1} (rescaled together)
        const double sc = (double)F;
        for (int q = t; q < F; q += nt) {
            w1[q] = d[q] * sc;
            w2[q] = q > 0 ? -(dl[q] * sc) * (du[q - 1] * sc) : 0.0;
        }
        __syncthreads();
        if (t == 0) {
            double pm = 1.0, pq = w1[0];
            w2[0] = 1.0;
            for (int q = 1; q < F; ++q) {
                const double pn = fma(w1[q], pq, w2[q] * pm);
                pm = pq;
                pq = pn;
                w1[q] = pq;
                w2[q] = pm;
                const int ex = (__double2hiint(pq) >> 20) & 0x7ff;
                if (ex > 1023 + 400 || ex < 1023 - 400) {   // out of 10^+-120: bring both back
                    const double r = ex > 1023 ? 1e-120 : 1e120;
                    pq *= r;
                    pm *= r;
                }
            }
        }
        __syncthreads();
        int good = 1;
        for (int q = t; q < F; q += nt) w1[q] = w1[q] / (w2[q] * (double)F);
        __syncthreads();
        for (int it = 0; it < 2; ++it) {
            for (int q = t; q < F; q += nt) w2[q] = q == 0 ? d[0] : d[q] - (dl[q] * du[q - 1]) / w1[q - 1];
            __syncthreads();
            for (int q = t; q < F; q += nt) w1[q] = w2[q];
            __syncthreads();
        }
        // no exchange and every pivot a normal number, except that the last may be anything
        for (int q = t; q < F - 1; q += nt)
            if (!(fabs(w1[q]) >= fabs(dl[q + 1])) || !(fabs(w1[q]) > 1e-280) || !(fabs(w1[q]) < 1e280)) good = 0;
        done = __syncthreads_and(good);
        if (done) {
            for (int q = t; q < F; q += nt) d[q] = w1[q];
            for (int q = t; q < F; q += nt)
                if (q > 0) dl[q] = dl[q] / w1[q - 1];
        }
    }
    if (!done && t == 0) eliminate(F, dl, d, du, du2, ipiv);
    __syncthreads();
    for (int q = t; q < F; q += nt)
        if (d[q] == 0) status[STATUS_SPLINE] = 1;
    // factors out (from shared memory), and the cubic resample's uniform coefficients
    double *rh = p.aux, *rd = rh + F, *ev = rd + F, *ends = ev + 4 * F_new;
    for (int n = t; n <= F; n += nt) {
        if (use_smem) p.h[n] = h[n];
        if (n == F) continue;
        if (use_smem) {
            p.dl[n] = dl[n];
            p.d[n] = d[n];
            p.du[n] = du[n];
            p.du2[n] = du2[n];
            p.ipiv[n] = ipiv[n];
        }
        rh[n] = n > 0 ? 1.0 / h[n] : 0.0;
        rd[n] = 1.0 / d[n];
    }
    for (int n = t; n < F_new; n += nt) {
        const int k = kk[n];
        const double w = p.w[n], wm = spline == 0 ? (w - 1) : (1 - w), hk2 = h[k] * h[k];
        ev[4 * n] = w;
        ev[4 * n + 1] = 1 - w;
        ev[4 * n + 2] = hk2 * (w * w * w - w);
        ev[4 * n + 3] = hk2 * (wm * wm * wm - wm);
    }
    if (t == 0) {   // end conditions: third divided differences at both ends
        ends[0] = 1.0 / (h[3] + h[2]);
        ends[1] = 1.0 / (h[2] + h[1]);
        ends[2] = 1.0 / (h[3] + h[2] + h[1]);
        ends[3] = h[1] * h[1];
    } else if (t == 32) {
        ends[4] = 1.0 / (h[F - 1] + h[F - 2]);
        ends[5] = 1.0 / (h[F - 2] + h[F - 3]);
        ends[6] = 1.0 / (h[F - 1] + h[F - 2] + h[F - 3]);
        ends[7] = -(h[F - 1] * h[F - 1]);
    }
}

// Linear resample: block row blockIdx.y is output image n, the blocks of the
// row stride over its reals, V of them per access (V = 4 for float fields
// whose image size allows 16-byte vectors, 2 for double, else 1).
template <class T, int V>
__global__ void __launch_bounds__(NT) k_redist_linear(const T *f, T *fnew, long reals, const int *kk, const double *ww)
{
    using Vec = typename std::conditional<V == 4, float4, typename std::conditional<V == 2, double2, T>::type>::type;
    const int n = blockIdx.y;
    const int k = kk[n];
    const T w = (T)ww[n];
    const Vec *a = reinterpret_cast<const Vec *>(f + (long)k * reals);
    const Vec *b = reinterpret_cast<const Vec *>(f + (long)(k - 1) * reals);
    Vec *o = reinterpret_cast<Vec *>(fnew + (long)n * reals);
    const long nv = reals / V;
    for (long i = blockIdx.x * (long)NT + threadIdx.x; i < nv; i += (long)gridDim.x * NT) {
        const Vec va = a[i], vb = b[i];
        const T *pa = reinterpret_cast<const T *>(&va), *pb = reinterpret_cast<const T *>(&vb);
        Vec vo;
        T *po = reinterpret_cast<T *>(&vo);
#pragma unroll
        for (int c = 0; c < V; ++c) po[c] = w * pa[c] + (1 - w) * pb[c];
        o[i] = vo;
    }
}

// Cubic resample (computeDeltaX/Y + gtsv + generateNewFramesCubic,
// interpolation.cu:292-402), one thread per real of a site: builds the
// right-hand side, solves with the shared factors, evaluates the new
// images.  The arithmetic type C is that of the fields: float for FP32
// fields, as the reference's FP32 build computes its spline, and double for
// FP64 ones.  Every division is a product with a reciprocal the plan made
// once, and the per-image evaluation weights come from the plan too, so a
// real costs about ten multiply-adds per image.  SG(n), the thread's column
// of the solution, lives in shared memory ([n][thread]) or, for strings too
// long for that, in the strided global scratch.

// Uniform data of one resample in type C, staged in shared memory per block.
template <class C>
struct CubicUniform {
    C *rh, *rd, *dl, *du, *du2, *ev, *ends;
    int *ipiv, *kk;
};

template <class C>
__host__ __device__ inline size_t cubic_uniform_bytes(int F, int F_new)
{
    return ((size_t)(5 * F + 4 * F_new + 8) * sizeof(C) + (size_t)(F + F_new) * sizeof(int) + 15) & ~(size_t)15;
}

template <class C>
__device__ __forceinline__ CubicUniform<C> stage_cubic_uniform(const RedistPlan &p, int F, int F_new, char *sm)
{
    CubicUniform<C> u;
    u.rh = reinterpret_cast<C *>(sm);
    u.rd = u.rh + F;
    u.dl = u.rd + F;
    u.du = u.dl + F;
    u.du2 = u.du + F;
    u.ev = u.du2 + F;
    u.ends = u.ev + 4 * F_new;
    u.ipiv = reinterpret_cast<int *>(u.ends + 8);
    u.kk = u.ipiv + F;
    const double *rh = p.aux, *rd = rh + F, *ev = rd + F, *ends = ev + 4 * F_new;
    for (int n = threadIdx.x; n < F; n += blockDim.x) {
        u.rh[n] = (C)rh[n];
        u.rd[n] = (C)rd[n];
        u.dl[n] = (C)p.dl[n];
        u.du[n] = (C)p.du[n];
        u.du2[n] = (C)p.du2[n];
        u.ipiv[n] = p.ipiv[n];
    }
    for (int n = threadIdx.x; n < 4 * F_new; n += blockDim.x) u.ev[n] = (C)ev[n];
    for (int n = threadIdx.x; n < F_new; n += blockDim.x) u.kk[n] = p.k[n];
    if (threadIdx.x < 8) u.ends[threadIdx.x] = (C)ends[threadIdx.x];
    __syncthreads();
    return u;
}

template <class T, class C, bool SMEM>
__device__ __forceinline__ void redist_cubic_real(const T *__restrict__ f, T *__restrict__ fnew, C *sig, long reals,
                                                  long e, int F, int F_new, const CubicUniform<C> &u)
{
#define FV(n) ((C)f[(long)(n) * reals + e])
#define SG(n) (SMEM ? sig[(n) * (int)blockDim.x + (int)threadIdx.x] : sig[(long)(n) * reals + e])
    // the column of f into the solution's storage, eight loads in flight at a time
    {
        int n = 0;
        for (; n + 8 <= F; n += 8) {
            C v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = FV(n + i);
#pragma unroll
            for (int i = 0; i < 8; ++i) SG(n + i) = v[i];
        }
        for (; n < F; ++n) SG(n) = FV(n);
    }
    // first divided differences D[n] = (f_n - f_{n-1}) / h_n, n >= 1; the
    // right-hand side overwrites f in place (f_n is carried in fp)
    const C D1 = (SG(1) - SG(0)) * u.rh[1], D2 = (SG(2) - SG(1)) * u.rh[2], D3 = (SG(3) - SG(2)) * u.rh[3];
    const C Dm1 = (SG(F - 1) - SG(F - 2)) * u.rh[F - 1], Dm2 = (SG(F - 2) - SG(F - 3)) * u.rh[F - 2];
    const C Dm3 = (SG(F - 3) - SG(F - 4)) * u.rh[F - 3];
    const C d3s = ((D3 - D2) * u.ends[0] - (D2 - D1) * u.ends[1]) * u.ends[2];
    const C d3e = ((Dm1 - Dm2) * u.ends[4] - (Dm2 - Dm3) * u.ends[5]) * u.ends[6];
    C Dn = D1, fp = SG(1);
    for (int n = 1; n < F - 1; ++n) {
        const C fn1 = SG(n + 1);
        const C Dn1 = (fn1 - fp) * u.rh[n + 1];
        SG(n) = Dn1 - Dn;
        Dn = Dn1;
        fp = fn1;
    }
    SG(0) = u.ends[3] * d3s;
    SG(F - 1) = u.ends[7] * d3e;
    // forward elimination with the recorded pivots
    for (int q = 0; q < F - 1; ++q) {
        const C bk = SG(q), bk1 = SG(q + 1);
        if (u.ipiv[q]) {
            SG(q) = bk1;
            SG(q + 1) = bk - u.dl[q + 1] * bk1;
        } else {
            SG(q + 1) = bk1 - u.dl[q + 1] * bk;
        }
    }
    SG(F - 1) = SG(F - 1) * u.rd[F - 1];
    SG(F - 2) = (SG(F - 2) - u.du[F - 2] * SG(F - 1)) * u.rd[F - 2];
    for (int q = F - 3; q >= 0; --q) SG(q) = (SG(q) - u.du[q] * SG(q + 1) - u.du2[q] * SG(q + 2)) * u.rd[q];
    // new images: f re-read (from L2), four outputs' loads in flight at a time
    int n = 0;
    for (; n + 4 <= F_new; n += 4) {
        C a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = u.kk[n + i];
            a[i] = FV(k);
            b[i] = FV(k - 1);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = u.kk[n + i];
            const C *c = u.ev + 4 * (n + i);
            fnew[(long)(n + i) * reals + e] = (T)(c[0] * a[i] + c[1] * b[i] + c[2] * SG(k) + c[3] * SG(k - 1));
        }
    }
    for (; n < F_new; ++n) {
        const int k = u.kk[n];
        const C *c = u.ev + 4 * n;
        fnew[(long)n * reals + e] = (T)(c[0] * FV(k) + c[1] * FV(k - 1) + c[2] * SG(k) + c[3] * SG(k - 1));
    }
#undef FV
#undef SG
}

// Arithmetic type of the cubic resample for fields of type T.
template <class T> using cubic_t = T;

template <class T>
__global__ void __launch_bounds__(NT) k_redist_cubic(const T *f, T *fnew, cubic_t<T> *sig, long reals, int F,
                                                     int F_new, RedistPlan p)
{
    extern __shared__ __align__(16) char cubic_sm[];
    const CubicUniform<cubic_t<T>> u = stage_cubic_uniform<cubic_t<T>>(p, F, F_new, cubic_sm);
    for (long e = blockIdx.x * (long)NT + threadIdx.x; e < reals; e += (long)gridDim.x * NT)
        redist_cubic_real<T, cubic_t<T>, false>(f, fnew, sig, reals, e, F, F_new, u);
}

// Shared-memory columns: after the uniform data, F * blockDim.x values;
// each thread owns one column, so no barrier is needed after the staging.
template <class T>
__global__ void __launch_bounds__(128) k_redist_cubic_s(const T *f, T *fnew, long reals, int F, int F_new,
                                                        RedistPlan p)
{
    extern __shared__ __align__(16) char cubic_sm[];
    const CubicUniform<cubic_t<T>> u = stage_cubic_uniform<cubic_t<T>>(p, F, F_new, cubic_sm);
    cubic_t<T> *cols = reinterpret_cast<cubic_t<T> *>(cubic_sm + cubic_uniform_bytes<cubic_t<T>>(F, F_new));
    for (long e0 = blockIdx.x * (long)blockDim.x; e0 < reals; e0 += (long)gridDim.x * blockDim.x) {
        const long e = e0 + threadIdx.x;
        if (e < reals) redist_cubic_real<T, cubic_t<T>, true>(f, fnew, cols, reals, e, F, F_new, u);
    }
}

template <class S, class D>
__global__ void k_convert(const S *src, D *dst, long n)
{
    for (long e = blockIdx.x * (long)NT + threadIdx.x; e < n; e += (long)gridDim.x * NT) dst[e] = (D)src[e];
}

inline int grid_for(long n, int cap = 152 * 16)
{
    long b = (n + NT - 1) / NT;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

// ----------------------------------------------------------------- launchers
// One operation over every strip of the launch's string.
template <class T, class Op>
static cudaError_t walk(const Launch &L, const Scalars &sc, int xbuf, const Op &op)
{
    if (L.ncomp == 2) k_walk<T, 2, Op><<<L.n_tiles, NTS, 0, L.stream>>>(*L.str, sc, xbuf, op);
    else k_walk<T, 1, Op><<<L.n_tiles, NTS, 0, L.stream>>>(*L.str, sc, xbuf, op);
    return cudaGetLastError();
}

template <class Op>
static cudaError_t walk(const Launch &L, const Scalars &sc, int xbuf, const Op &op)
{
    return L.precision == 1 ? walk<double>(L, sc, xbuf, op) : walk<float>(L, sc, xbuf, op);
}

// NLCG passes: one single-warp block per strip; launches of one string take
// the kernels that read its descriptor at fixed offsets, and in float-float, where
// the registers run out, those without per-site parameters have no code for them
// (256 x 256 x 64, four steps: 5.65 ms with it, 5.32 without).
#define DISPATCH_STRIP_T(L, KERNEL, T, ...)                                                         \
    do {                                                                                            \
        if (strip_one(L)) {                                                                         \
            const batch_t<true> one = only_string(L);                                               \
            if ((L).ncomp == 2) KERNEL<T, 2, true><<<(L).n_stiles, NTS, 0, (L).stream>>>(one, __VA_ARGS__); \
            else KERNEL<T, 1, true><<<(L).n_stiles, NTS, 0, (L).stream>>>(one, __VA_ARGS__);        \
        } else {                                                                                    \
            if ((L).ncomp == 2) KERNEL<T, 2, false><<<(L).n_stiles, NTS, 0, (L).stream>>>(*(L).batch, __VA_ARGS__); \
            else KERNEL<T, 1, false><<<(L).n_stiles, NTS, 0, (L).stream>>>(*(L).batch, __VA_ARGS__); \
        }                                                                                           \
    } while (0)
#define DISPATCH_STRIP(L, KERNEL, ...)                                                              \
    do {                                                                                            \
        if ((L).precision == 0) DISPATCH_STRIP_T(L, KERNEL, float, __VA_ARGS__);                    \
        else if ((L).paired && strip_one(L) && !(L).batch->s[0].per_site) {                         \
            const batch_t<true> one = only_string(L);                                               \
            if ((L).ncomp == 2) KERNEL<ff, 2, true, false><<<(L).n_stiles, NTS, 0, (L).stream>>>(one, __VA_ARGS__); \
            else KERNEL<ff, 1, true, false><<<(L).n_stiles, NTS, 0, (L).stream>>>(one, __VA_ARGS__); \
        } else if ((L).paired) DISPATCH_STRIP_T(L, KERNEL, ff, __VA_ARGS__);                        \
        else DISPATCH_STRIP_T(L, KERNEL, double, __VA_ARGS__);                                      \
    } while (0)

static inline bool strip_one(const Launch &L) { return L.batch->n == 1; }
static inline batch_t<true> only_string(const Launch &L)
{
    batch_t<true> b;
    b.n = 1;
    b.s[0] = L.batch->s[0];
    return b;
}

cudaError_t launch_grad(const Launch &L, const Scalars &sc, const StepFlags &f)
{
    DISPATCH_STRIP(L, k_grad_s, L.stile0, sc, f);
    return cudaGetLastError();
}

cudaError_t launch_dir_poly(const Launch &L, const Scalars &sc, const StepFlags &f)
{
    DISPATCH_STRIP(L, k_dir_poly_s, L.stile0, sc, f);
    return cudaGetLastError();
}

// Resident blocks of one strip kernel on the current device.
template <class K>
static int resident(K kernel)
{
    int dev = 0, sms = 0, nb = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, NTS, 0) != cudaSuccess)
        return 0;
    return nb * sms;
}

// Constants and not what the compiler's register counts happen to give: the
// rows of a strip, and with them the order of an image's sums, follow from it.
// One component in FP32: 96 registers, five warps in each quarter of the SM.
int strip_pass_slots(int precision, int ncomp, int sms) { return sms * (precision == 1 ? 8 : ncomp == 2 ? 16 : 20); }

template <class T>
static cudaError_t nlcg_fused_launch(const Launch &L, const Scalars &sc, const StepPlan &plan, int steps,
                                     unsigned long long *queue, unsigned *stage, unsigned max_polls)
{
    static int slots[4] = {0, 0, 0, 0};
    const int ci = (L.ncomp == 2 ? 1 : 0) + (strip_one(L) ? 2 : 0);
    if (slots[ci] == 0) {
        slots[ci] = ci == 0   ? resident(k_nlcg_s<T, 1, false>)
                    : ci == 1 ? resident(k_nlcg_s<T, 2, false>)
                    : ci == 2 ? resident(k_nlcg_s<T, 1, true>)
                              : resident(k_nlcg_s<T, 2, true>);
        if (slots[ci] == 0) {
            const cudaError_t e = cudaGetLastError();
            return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
        }
    }
    const int grid = L.n_stiles < slots[ci] ? L.n_stiles : slots[ci];
#define FUSED_ARGS L.stile0, L.n_stiles, steps, plan, sc, queue, stage, max_polls
    switch (ci) {
    case 0: k_nlcg_s<T, 1, false><<<grid, NTS, 0, L.stream>>>(*L.batch, FUSED_ARGS); break;
    case 1: k_nlcg_s<T, 2, false><<<grid, NTS, 0, L.stream>>>(*L.batch, FUSED_ARGS); break;
    case 2: k_nlcg_s<T, 1, true><<<grid, NTS, 0, L.stream>>>(only_string(L), FUSED_ARGS); break;
    default: k_nlcg_s<T, 2, true><<<grid, NTS, 0, L.stream>>>(only_string(L), FUSED_ARGS); break;
    }
#undef FUSED_ARGS
    return cudaGetLastError();
}

cudaError_t launch_nlcg_fused(const Launch &L, const Scalars &sc, const StepFlags &f0, int it0, int steps,
                              unsigned long long *queue, unsigned *stage, int n_stage, unsigned long long first_item,
                              unsigned max_polls)
{
    StepPlan plan;
    plan.xi0 = f0.xin;
    plan.di0 = f0.din;
    plan.it0 = it0;
    plan.base = f0;
    // the counter and the stages lie in one piece of memory
    char *const end = reinterpret_cast<char *>(stage + (size_t)n_stage * STAGE_STRIDE);
    cudaError_t e = cudaMemsetAsync(queue, 0, end - reinterpret_cast<char *>(queue), L.stream);
    if (e == cudaSuccess && first_item) {
        e = cudaMemcpyAsync(queue, &first_item, sizeof(first_item), cudaMemcpyHostToDevice, L.stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(L.stream);   // first_item is a host local
    }
    if (e != cudaSuccess) return e;
    return L.precision == 0 ? nlcg_fused_launch<float>(L, sc, plan, steps, queue, stage, max_polls)
           : L.paired       ? nlcg_fused_launch<ff>(L, sc, plan, steps, queue, stage, max_polls)
                            : nlcg_fused_launch<double>(L, sc, plan, steps, queue, stage, max_polls);
}

cudaError_t launch_energy(const Launch &L, const Scalars &sc, int xbuf, double *out)
{
    return walk(L, sc, xbuf, EnergyOp{out});
}

// FP64 launches with L.paired compute in float-float on the double fields
// (about 48 bits) and store double gradients; the link discretisation has
// no float-float form and stays IEEE double.
cudaError_t launch_gradient_only(const Launch &L, const Scalars &sc, int xbuf, FieldPtrs out, int maxwell,
                                 const double *weights, double *adjoint)
{
    if (adjoint)
        return walk(L, sc, xbuf, GradientOp<true>{{out.p[0], out.p[1], out.p[2]}, maxwell, weights, adjoint});
    const GradientOp<false> op{{out.p[0], out.p[1], out.p[2]}, maxwell, weights, nullptr};
    if (L.paired && L.precision == 1 && !L.str->disc) return walk<ff>(L, sc, xbuf, op);
    return walk(L, sc, xbuf, op);
}

cudaError_t launch_param_adjoint(const Launch &L, const Scalars &sc, int xbuf, double *out)
{
    return walk(L, sc, xbuf, AdjointOp{out});
}

cudaError_t launch_jb(const Launch &L, const Scalars &sc, int xbuf, void *b, void *j1, void *j2)
{
    return walk(L, sc, xbuf, JbOp{b, j1, j2});
}

cudaError_t launch_flux(const Launch &L, const Scalars &sc, int xbuf, double *out)
{
    return walk(L, sc, xbuf, FluxOp{out});
}

template <class T, class W>
static void apply_update(const Launch &L, const Scalars &sc, int xbuf, int dbuf)
{
    const Batch &B = *L.batch;
    long M = 0;
    for (int k = 0; k < B.n; ++k) M = M > (long)B.s[k].nx * B.s[k].ny ? M : (long)B.s[k].nx * B.s[k].ny;
    const int img0 = B.s[0].img_base, images = B.s[B.n - 1].img_base + B.s[B.n - 1].F - img0;
    const long chunks = (M + NT - 1) / NT;
    constexpr int MOST = 65535;   // images per launch (grid y)
    for (int i = 0; i < images; i += MOST) {
        const int n = images - i < MOST ? images - i : MOST;
        const dim3 grid((unsigned)(chunks < 64 ? chunks : 64), (unsigned)n, (unsigned)(1 + L.ncomp));
        if (strip_one(L)) k_apply_update<T, W, true><<<grid, NT, 0, L.stream>>>(only_string(L), sc.alpha_pend, img0 + i, xbuf, dbuf);
        else k_apply_update<T, W, false><<<grid, NT, 0, L.stream>>>(B, sc.alpha_pend, img0 + i, xbuf, dbuf);
    }
}

cudaError_t launch_apply_update(const Launch &L, const Scalars &sc, int xbuf, int dbuf)
{
    if (L.precision == 0) apply_update<float, float>(L, sc, xbuf, dbuf);
    else if (L.paired) apply_update<double, ff>(L, sc, xbuf, dbuf);   // d holds float-float pairs (paired passes)
    else apply_update<double, double>(L, sc, xbuf, dbuf);
    return cudaGetLastError();
}

cudaError_t launch_reset_history(const Scalars &sc, int n_images, cudaStream_t st)
{
    k_reset_history<<<(n_images + NT - 1) / NT, NT, 0, st>>>(sc, n_images);
    return cudaGetLastError();
}

cudaError_t launch_restart_cg(const Scalars &sc, int first, int last, cudaStream_t st)
{
    k_restart_cg<<<(last - first + NT - 1) / NT, NT, 0, st>>>(sc, first, last);
    return cudaGetLastError();
}

cudaError_t launch_check_scalars(const Scalars &sc, int n_images, int slot, cudaStream_t st)
{
    k_check_scalars<<<(n_images + NT - 1) / NT, NT, 0, st>>>(sc.fenergy, slot ? sc.gn1 : sc.gn0, n_images, sc.status);
    return cudaGetLastError();
}

// Distances by one walk (k_arc_walk) or from stored B and J.  The walk reads
// each image once but forms B and J of every chunk's first image again and has
// few, long blocks: it pays in FP32, which is bound by memory, once there are
// blocks for every SM (256 x 256 x 64: 77 us against 104; 64 x 64 x 16 in FP64:
// 97 us against 24).
static bool arc_by_walk(const Launch &L, int metrics, int sms)
{
    const StringDesc &S = *L.str;
    return L.precision == 0 && metrics == 3 && (long)S.tiles_x * ((S.ny + ARC_ROWS - 1) / ARC_ROWS) * S.F >= 64L * sms;
}

size_t arc_blocks(const StringDesc &S)
{
    const size_t walk = (size_t)S.tiles_x * ((S.ny + ARC_ROWS - 1) / ARC_ROWS);
    const size_t flat = ((size_t)S.nx * S.ny + NT * ARC_SPT - 1) / (NT * ARC_SPT);
    return walk > flat ? walk : flat;
}

template <int NC>
static void arc_walk(const Launch &L, int xbuf, int nb, int sms, double *part_f, double *part_jb)
{
    const StringDesc &S = *L.str;
    // images per block: long enough to spare the image read twice at a chunk's
    // start, short enough that there is a wave of blocks
    int chunk = (int)((long)nb * S.F / ((long)sms * 16));
    chunk = chunk < 4 ? 4 : (chunk > 32 ? 32 : chunk);
    const dim3 grid((unsigned)nb, (unsigned)((S.F + chunk - 1) / chunk));
    k_arc_walk<NC><<<grid, NTS, 0, L.stream>>>(S, xbuf, chunk, part_f, part_jb);
}

template <class T>
static void arc_flat(const Launch &L, const void *const *f, int w0, int nb, double *part)
{
    const StringDesc &S = *L.str;
    k_arc_partial<T><<<dim3(nb, S.F), NT, 0, L.stream>>>((const T *)f[0], (const T *)f[1], L.ncomp == 2 ? (const T *)f[2] : nullptr,
                                                         w0, 2, 2, (long)S.nx * S.ny, part);
}

cudaError_t launch_arc_distances(const Launch &L, const Scalars &sc, int xbuf, int metrics, int sms, void *const *spare,
                                 double *s_f, double *s_jb)
{
    const StringDesc &S = *L.str;
    double *part = sc.part, *part_jb = part + (metrics == 3 ? arc_blocks(S) * S.F : 0);
    int nb;
    if (arc_by_walk(L, metrics, sms)) {
        nb = S.tiles_x * ((S.ny + ARC_ROWS - 1) / ARC_ROWS);
        if (L.ncomp == 2) arc_walk<2>(L, xbuf, nb, sms, part, part_jb);
        else arc_walk<1>(L, xbuf, nb, sms, part, part_jb);
    } else {
        nb = (int)(((long)S.nx * S.ny + NT * ARC_SPT - 1) / (NT * ARC_SPT));
        if (metrics & 2) {
            const cudaError_t e = launch_jb(L, sc, xbuf, spare[0], spare[1], spare[2]);
            if (e != cudaSuccess) return e;
            if (L.precision == 1) arc_flat<double>(L, spare, 1, nb, part_jb);
            else arc_flat<float>(L, spare, 1, nb, part_jb);
        }
        if (metrics & 1) {
            if (L.precision == 1) arc_flat<double>(L, S.x[xbuf], 2, nb, part);
            else arc_flat<float>(L, S.x[xbuf], 2, nb, part);
        }
    }
    const double *pf = metrics & 1 ? part : part_jb;
    double *sf = metrics & 1 ? s_f : s_jb;
    k_arc_sum<<<dim3(S.F, metrics == 3 ? 2 : 1), NT, 0, L.stream>>>(pf, part_jb, nb, sf, s_jb);
    return cudaGetLastError();
}

cudaError_t launch_arc_cumulate(int F, double *s, int *bad, cudaStream_t st)
{
    const int smem = F <= ARC_CUM_MAX;
    k_arc_cumulate<<<1, NT, smem ? F * sizeof(double) : 0, st>>>(F, s, bad, smem);
    return cudaGetLastError();
}

cudaError_t launch_generate(int precision, void *a, void *p1, void *p2, int nx, int ny, int F, int ncomp,
                            const int32_t *comp, const int32_t *sc, const double *tracks, int n_tracks,
                            const GuessParams &g, cudaStream_t st)
{
    const long n = (long)nx * ny * F;
    long b = (n + NT - 1) / NT;
    const int grid = (int)(b < 1 ? 1 : (b > 152 * 32 ? 152 * 32 : b));
    if (precision == 1)
        k_generate<double><<<grid, NT, 0, st>>>((double2 *)a, (double2 *)p1, (double2 *)p2, nx, ny, F, ncomp, comp, sc,
                                                tracks, n_tracks, g);
    else
        k_generate<float><<<grid, NT, 0, st>>>((float2 *)a, (float2 *)p1, (float2 *)p2, nx, ny, F, ncomp, comp, sc,
                                               tracks, n_tracks, g);
    return cudaGetLastError();
}

cudaError_t launch_winding(int precision, const void *psi, int nx, int ny, int F, int inset, double *out,
                           cudaStream_t st)
{
    const int grid = F < 152 * 4 ? F : 152 * 4;
    if (precision == 1) k_winding<double><<<grid, NT, 0, st>>>((const double2 *)psi, nx, ny, F, inset, out);
    else k_winding<float><<<grid, NT, 0, st>>>((const float2 *)psi, nx, ny, F, inset, out);
    return cudaGetLastError();
}

// Dynamic shared memory of a reparametrization kernel, at most.  A kernel's limit
// is one setting for the whole process, so every launch that needs more than the
// default sets this, and none lowers what another thread's launch counts on.
constexpr size_t REDIST_SMEM = 200 * 1024;

template <class K>
static cudaError_t allow_smem(K kernel, size_t need)
{
    if (need <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)REDIST_SMEM);
}

cudaError_t launch_redist_plan(double *s_f, double *s_jb, const double *s_use, int *status, int F, int F_new, int cubic,
                               int spline, const RedistPlan &p, cudaStream_t st)
{
    const size_t sm = redist_plan_smem(F, F_new);
    const int use_smem = sm <= REDIST_SMEM;   // about 2,300 images
    const cudaError_t e = allow_smem(k_redist_plan, use_smem ? sm : 0);
    if (e != cudaSuccess) return e;
    k_redist_plan<<<1, 128, use_smem ? sm : 0, st>>>(s_f, s_jb, s_use, status, F, F_new, cubic, spline, p, use_smem);
    return cudaGetLastError();
}

cudaError_t launch_redist_linear(int precision, const void *f, void *fnew, long pairs, int F_new, const RedistPlan &p,
                                 cudaStream_t st)
{
    const long reals = 2 * pairs;
    // blocks per output image: about four waves of the GPU in all
    auto grid = [&](long nv) {
        long bx = (nv + NT - 1) / NT, cap = (152L * 8 * 4 + F_new - 1) / F_new;
        bx = bx < cap ? bx : cap;
        return dim3((unsigned)(bx < 1 ? 1 : bx), (unsigned)F_new);
    };
    if (precision == 1) {
        k_redist_linear<double, 2><<<grid(reals / 2), NT, 0, st>>>((const double *)f, (double *)fnew, reals, p.k, p.w);
    } else if (reals % 4 == 0) {
        k_redist_linear<float, 4><<<grid(reals / 4), NT, 0, st>>>((const float *)f, (float *)fnew, reals, p.k, p.w);
    } else {
        k_redist_linear<float, 1><<<grid(reals), NT, 0, st>>>((const float *)f, (float *)fnew, reals, p.k, p.w);
    }
    return cudaGetLastError();
}

// Shape of a cubic resample launch: threads per block and dynamic shared
// memory of the shared-memory form (32 KB of columns per block where F
// allows: 128 threads, 64 or 32; up to 200 KB in all at 32 threads), or
// sm = 0 when the string is too long for it and the global scratch is used.
static void cubic_shape(int precision, int F, int F_new, int *tpb_out, size_t *sm_out)
{
    const size_t cs = precision == 1 ? sizeof(double) : sizeof(float);
    const size_t ub = precision == 1 ? cubic_uniform_bytes<double>(F, F_new) : cubic_uniform_bytes<float>(F, F_new);
    int tpb = 128;
    while (tpb > 32 && (size_t)tpb * F * cs > 32 * 1024) tpb >>= 1;
    const size_t sm = ub + (size_t)tpb * F * cs;
    *tpb_out = tpb;
    *sm_out = sm <= REDIST_SMEM ? sm : 0;
}

size_t redist_cubic_scratch_bytes(int precision, long pairs, int F, int F_new)
{
    int tpb;
    size_t sm;
    cubic_shape(precision, F, F_new, &tpb, &sm);
    return sm ? 0 : (size_t)2 * pairs * F * (precision == 1 ? sizeof(double) : sizeof(float));
}

cudaError_t launch_redist_cubic(int precision, const void *f, void *fnew, void *sigma, long pairs, int F, int F_new,
                                int spline, const RedistPlan &p, cudaStream_t st)
{
    (void)spline;   // folded into the plan's evaluation weights
    const long reals = 2 * pairs;
    const size_t ub = precision == 1 ? cubic_uniform_bytes<double>(F, F_new) : cubic_uniform_bytes<float>(F, F_new);
    int tpb;
    size_t sm;
    cubic_shape(precision, F, F_new, &tpb, &sm);
    cudaError_t e = cudaSuccess;
    if (sm) {
        const long blocks = (reals + tpb - 1) / tpb;
        const int grid = (int)(blocks < 152 * 32 ? blocks : 152 * 32);
        if (precision == 1) {
            e = allow_smem(k_redist_cubic_s<double>, sm);
            if (e != cudaSuccess) return e;
            k_redist_cubic_s<double><<<grid, tpb, sm, st>>>((const double *)f, (double *)fnew, reals, F, F_new, p);
        } else {
            e = allow_smem(k_redist_cubic_s<float>, sm);
            if (e != cudaSuccess) return e;
            k_redist_cubic_s<float><<<grid, tpb, sm, st>>>((const float *)f, (float *)fnew, reals, F, F_new, p);
        }
        return cudaGetLastError();
    }
    if (ub > REDIST_SMEM || !sigma) return cudaErrorInvalidValue;   // more than about 2,800 images
    e = precision == 1 ? allow_smem(k_redist_cubic<double>, ub) : allow_smem(k_redist_cubic<float>, ub);
    if (e != cudaSuccess) return e;
    if (precision == 1)
        k_redist_cubic<double><<<grid_for(reals), NT, ub, st>>>((const double *)f, (double *)fnew, (double *)sigma,
                                                                reals, F, F_new, p);
    else
        k_redist_cubic<float><<<grid_for(reals), NT, ub, st>>>((const float *)f, (float *)fnew, (float *)sigma, reals,
                                                               F, F_new, p);
    return cudaGetLastError();
}

cudaError_t launch_pair_sites(void *const *p, int ncomp, void *out, long M)
{
    // behind the parameters' own copies, and done when the context's stream may read them
    const unsigned grid = (unsigned)((M + NT - 1) / NT);
    const double *const *q = reinterpret_cast<const double *const *>(p);
    float2 *o = static_cast<float2 *>(out);
    for (int k = 0; k < ncomp; ++k) k_pair_sites<<<grid, NT, 0, cudaStreamLegacy>>>(q[4 * k], q[4 * k + 1], q[4 * k + 2], q[4 * k + 3], o + 5 * k * M, M);
    k_pair_sites<<<grid, NT, 0, cudaStreamLegacy>>>(q[8], nullptr, nullptr, nullptr, o + 5 * ncomp * M, M);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e : cudaStreamSynchronize(cudaStreamLegacy);
}

cudaError_t launch_x_format(void *x, long pairs, int to_pairs, cudaStream_t st)
{
    if (to_pairs) k_x_format<true><<<grid_for(pairs), NT, 0, st>>>((double2 *)x, pairs);
    else k_x_format<false><<<grid_for(pairs), NT, 0, st>>>((double2 *)x, pairs);
    return cudaGetLastError();
}

cudaError_t launch_convert(const void *src, int src_prec, void *dst, int dst_prec, long n, cudaStream_t st)
{
    if (src_prec == 0 && dst_prec == 1)
        k_convert<float, double><<<grid_for(n), NT, 0, st>>>((const float *)src, (double *)dst, n);
    else if (src_prec == 1 && dst_prec == 0)
        k_convert<double, float><<<grid_for(n), NT, 0, st>>>((const double *)src, (float *)dst, n);
    else
        return cudaMemcpyAsync(dst, src, n * (src_prec ? 8 : 4), cudaMemcpyDeviceToDevice, st);
    return cudaGetLastError();
}

}  // namespace mepgl

// ===================================================== allocation-free energy
//
// Some callers cannot allocate device memory: embedded solvers that own a
// fixed device arena and hand out only pre-allocated buffers, host
// frameworks whose memory pool owns the whole device, or plugins whose host
// process forbids cudaMalloc after start-up (an allocation there can
// synchronise the device in the middle of its pipelined work).  mepgl_free_energy_noalloc serves them: it
// evaluates the per-image free energy of caller-owned device arrays without
// creating a context and without any allocation.  The per-tile partial sums
// and per-image tickets of the deterministic reduction live in the fixed
// arrays below, which every GPU that loads this library holds until the
// process exits (4 MiB + 16 KiB per device).
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/mepgl.h"

namespace {

constexpr int NOALLOC_MAX_TILES = 65536;     // images x ceil(nx/32) x ceil(ny/8)
constexpr int NOALLOC_MAX_IMAGES = 4096;
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) double g_noalloc_part[NOALLOC_MAX_TILES * 8];
static __device__ __align__(256) unsigned g_noalloc_ticket[NOALLOC_MAX_IMAGES];

struct NoallocScratch {
    bool ready;
    double *part;
    unsigned *ticket;
};
std::mutex g_noalloc_mu;
NoallocScratch g_noalloc[NOALLOC_MAX_DEVICES];
thread_local std::string g_noalloc_err;

// Device addresses of the scratch arrays, resolved once per device with that
// device current (a host-side reference to the array names is not a device
// address).  Also uploads the constant neighbour-code tables.  Both are kept
// for the life of the process: a device reset (cudaDeviceReset, or a reset
// of the primary context by the host framework) is not supported, since the
// cached addresses and the constant tables would then be stale.
cudaError_t noalloc_setup(int dev, NoallocScratch *out)
{
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    NoallocScratch &s = g_noalloc[dev];
    if (!s.ready) {
        cudaError_t e = cudaGetSymbolAddress((void **)&s.part, g_noalloc_part);
        if (e != cudaSuccess) return e;
        e = cudaGetSymbolAddress((void **)&s.ticket, g_noalloc_ticket);
        if (e != cudaSuccess) return e;
        e = mepgl::upload_mask_tables();
        if (e != cudaSuccess) return e;
        s.ready = true;
    }
    *out = s;
    return cudaSuccess;
}

mepgl_status noalloc_fail(mepgl_status st, const std::string &m)
{
    g_noalloc_err = m;
    return st;
}

}  // namespace

extern "C" const char *mepgl_noalloc_last_error(void) { return g_noalloc_err.c_str(); }

extern "C" mepgl_status mepgl_free_energy_noalloc(int nx, int ny, int n_images, int multicomponent, int thin_film,
                                                  double dx, const int32_t *comp_code, const int32_t *sc_code,
                                                  const double *a_1, const double *b_1, const double *m_xx_1,
                                                  const double *m_yy_1, const double *a_2, const double *b_2,
                                                  const double *m_xx_2, const double *m_yy_2, const double *h,
                                                  double q_1, double q_2, double eta, double gamma, double delta,
                                                  const void *a, const void *psi_1, const void *psi_2,
                                                  double *fenergy, void *stream)
{
    using namespace mepgl;
    constexpr int rows = 8;   // per strip
    if (nx < 2 || ny < 2 || n_images < 1 || !(dx > 0))
        return noalloc_fail(MEPGL_ERR_INVALID_ARG, "need nx, ny >= 2, n_images >= 1, dx > 0");
    if (!comp_code || !sc_code || !a_1 || !b_1 || !m_xx_1 || !m_yy_1 || !h || !a || !psi_1 || !fenergy ||
        (multicomponent && (!a_2 || !b_2 || !m_xx_2 || !m_yy_2 || !psi_2)))
        return noalloc_fail(MEPGL_ERR_INVALID_ARG, "null device pointer");
    const long tiles_x = (nx + TX - 1) / TX, tiles_y = (ny + rows - 1) / rows;
    const long n_tiles = tiles_x * tiles_y * n_images;
    // the lattice limits of mepgl_create
    if (nx > 32767 * TX || ny > 32767 * rows || (long)nx * ny >= (1L << 31))
        return noalloc_fail(MEPGL_ERR_INVALID_ARG, "lattice too large: need nx <= 32767*32, ny <= 32767*8 "
                                                   "and nx * ny < 2^31");
    if (n_images > NOALLOC_MAX_IMAGES || n_tiles > NOALLOC_MAX_TILES)
        return noalloc_fail(MEPGL_ERR_INVALID_ARG,
                            "string too large for the fixed scratch: need n_images <= 4096 and "
                            "n_images * ceil(nx/32) * ceil(ny/8) <= 65536");
    for (const void *p : {a, psi_1, multicomponent ? psi_2 : a})   // read as whole pairs
        if (reinterpret_cast<uintptr_t>(p) % (2 * sizeof(double)))
            return noalloc_fail(MEPGL_ERR_INVALID_ARG, "fields not aligned to a pair of doubles");
    // An error left pending by the caller's own earlier work is reported as
    // such and left in place, not taken for a failure of this call.
    cudaError_t pend = cudaPeekAtLastError();
    if (pend != cudaSuccess)
        return noalloc_fail(MEPGL_ERR_CUDA, std::string("error pending before this call (left for the caller): ") +
                                                cudaGetErrorString(pend));
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES)
        return noalloc_fail(MEPGL_ERR_CUDA, "no usable current device");
    NoallocScratch scr;
    cudaError_t e = noalloc_setup(dev, &scr);
    if (e != cudaSuccess) return noalloc_fail(MEPGL_ERR_CUDA, std::string("scratch setup: ") + cudaGetErrorString(e));

    StringDesc S;
    memset(&S, 0, sizeof(S));
    S.nx = nx;
    S.ny = ny;
    S.F = n_images;
    S.ncomp = multicomponent ? 2 : 1;
    S.tiles_x = (int)tiles_x;
    S.wtiles_y = (int)tiles_y;
    S.wrows = rows;
    S.thin_film = thin_film ? 1 : 0;
    S.per_site = 1;
    const double *pa[2] = {a_1, multicomponent ? a_2 : a_1}, *pb[2] = {b_1, multicomponent ? b_2 : b_1};
    const double *px[2] = {m_xx_1, multicomponent ? m_xx_2 : m_xx_1}, *py[2] = {m_yy_1, multicomponent ? m_yy_2 : m_yy_1};
    for (int c = 0; c < 2; ++c) {
        S.pa[c] = pa[c];
        S.pb[c] = pb[c];
        S.pmxx[c] = px[c];
        S.pmyy[c] = py[c];
    }
    S.ph = h;
    S.ud.q[0] = q_1;
    S.ud.q[1] = q_2;
    S.ud.eta = eta;
    S.ud.gamma = gamma;
    S.ud.delta = delta;
    S.ud.idx = 1.0 / dx;
    S.ud.dx2 = dx * dx;
    S.ud.dx = dx;
    fold_spacing(S.ud);
    S.code_comp = comp_code;
    S.code_sc = sc_code;
    S.x[0][0] = const_cast<void *>(a);
    S.x[0][1] = const_cast<void *>(psi_1);
    S.x[0][2] = multicomponent ? const_cast<void *>(psi_2) : nullptr;
    Scalars sc;
    memset(&sc, 0, sizeof(sc));
    sc.part = scr.part;
    sc.ticket = scr.ticket;
    cudaStream_t st = (cudaStream_t)stream;
    // the tickets must start at zero; the array keeps the previous call's contents
    e = cudaMemsetAsync(scr.ticket, 0, sizeof(unsigned) * n_images, st);
    if (e != cudaSuccess) return noalloc_fail(MEPGL_ERR_CUDA, std::string("ticket reset: ") + cudaGetErrorString(e));
    if (multicomponent)
        k_walk<double, 2, EnergyOp><<<(unsigned)n_tiles, NTS, 0, st>>>(S, sc, 0, EnergyOp{fenergy});
    else
        k_walk<double, 1, EnergyOp><<<(unsigned)n_tiles, NTS, 0, st>>>(S, sc, 0, EnergyOp{fenergy});
    e = cudaGetLastError();
    if (e != cudaSuccess) return noalloc_fail(MEPGL_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    return MEPGL_OK;
}
