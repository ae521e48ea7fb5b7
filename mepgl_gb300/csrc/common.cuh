// common.cuh -- shared device-side definitions of libmepgl_gb300.
//
// Work decomposition.  Every kernel over the lattice shares a string out as
// strips of TX columns x some rows of one image, one warp each; a launch of
// the NLCG passes covers every image of up to MAX_STRINGS strings (strings
// may differ in size and image count).  Per-image reductions are
// deterministic: each strip writes one partial per quantity, and the last
// strip of an image to finish (atomic ticket per image) sums that image's
// partials in a fixed order.
//
// Precision.  Fields are float or double (T).  Sums are formed in T inside
// a warp (fixed shuffle trees), then in double across groups of rows and
// images.  GB300's FP64 pipe is a small fraction of its FP32
// rate, so FP32 kernels avoid any per-site double arithmetic or conversion.
#pragma once

#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "pair_float.cuh"

namespace mepgl {

constexpr int TX = 32;        // strip width: a warp
constexpr int NT = 256;       // threads per block for the lattice kernels
constexpr int MAX_STRINGS = 16;   // strings per launch (descriptors travel as a kernel parameter)

template <class T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };
template <> struct Vec2<ff> { using type = ff2; };
template <class T> using vec2_t = typename Vec2<T>::type;

// Storage type of a compute type: float-float arithmetic works on double
// fields (the paired FP64 mode); float and double are stored as computed.
template <class T> struct Store { using type = T; };
template <> struct Store<ff> { using type = double; };
template <class T> using store_t = typename Store<T>::type;

template <class T> __device__ __forceinline__ T from_store(store_t<T> v) { return v; }
template <> __device__ __forceinline__ ff from_store<ff>(double v) { return to_ff(v); }
template <class T> __device__ __forceinline__ store_t<T> to_store(T v) { return v; }
template <> __device__ __forceinline__ double to_store<ff>(ff v) { return to_double(v); }

template <class T> __device__ __forceinline__ vec2_t<T> load2(const vec2_t<store_t<T>> *p) { return *p; }
template <> __device__ __forceinline__ ff2 load2<ff>(const double2 *p)
{
    const double2 d = *p;
    ff2 r;
    r.x = to_ff(d.x);
    r.y = to_ff(d.y);
    return r;
}
template <class T> __device__ __forceinline__ void store2(vec2_t<store_t<T>> *p, vec2_t<T> v) { *p = v; }
template <> __device__ __forceinline__ void store2<ff>(double2 *p, ff2 v)
{
    *p = make_double2(to_double(v.x), to_double(v.y));
}

// Storage of the NLCG work arrays (gradient g and direction d): the compute
// type itself for float and double; float-float pairs in the paired FP64 mode
// (ff2 fills the same 16 bytes as double2), so the paired passes move them
// without conversions.  The arrays are internal to the NLCG passes and the
// pending-step update.  A restart does not clear them: after one, no pass uses what
// they hold (beta is 0 and |g|^2 infinite; what a pass has loaded ahead is dropped)
// before it has written them, in its own format.
template <class T> __device__ __forceinline__ vec2_t<T> loadw(const vec2_t<store_t<T>> *p) { return load2<T>(p); }
template <> __device__ __forceinline__ ff2 loadw<ff>(const double2 *p)
{
    const float4 q = *reinterpret_cast<const float4 *>(p);
    ff2 r;
    r.x = ff(q.x, q.y);
    r.y = ff(q.z, q.w);
    return r;
}
template <class T> __device__ __forceinline__ void storew(vec2_t<store_t<T>> *p, vec2_t<T> v) { store2<T>(p, v); }
template <> __device__ __forceinline__ void storew<ff>(double2 *p, ff2 v)
{
    *reinterpret_cast<float4 *>(p) = make_float4(v.x.hi, v.x.lo, v.y.hi, v.y.lo);
}

// Uniform GL parameters in one precision (hm* = 0.5 / m, aob = a / b).
template <class T>
struct Uniform {
    T a[2], b[2], hmx[2], hmy[2], aob[2], q[2];
    T eta, gamma, delta, h, idx, dx2, dx;
    // the same with the spacing folded in, as the stencils of site_pack.cuh
    // use them: q dx, +- half of it, (q + 1) dx, q / dx; -2 hm*, hm* / dx^2, half
    // of that; hm* q / dx; 2 a dx^2, 2 b dx^2; couplings times dx^2; h dx;
    // 1 / (4 dx), 1 / (8 dx^2)
    T qd[2], hqd[2], nhqd[2], kq[2], qi[2], n2hmx[2], n2hmy[2], hmxi[2], hmyi[2], hhmx[2], hhmy[2], jmx[2], jmy[2],
        a2[2], b2[2];
    T etad, gammad, deltad, hd, idx4, idx8;
    T hl;   // what rounding h to float left out, times dx (float only)
};

// The folded parameters from the plain ones (host, in double).
inline void fold_spacing(Uniform<double> &U)
{
    for (int c = 0; c < 2; ++c) {
        U.qd[c] = U.q[c] * U.dx;
        U.hqd[c] = 0.5 * U.qd[c];
        U.nhqd[c] = -U.hqd[c];
        U.kq[c] = (U.q[c] + 1.0) * U.dx;
        U.qi[c] = U.q[c] * U.idx;
        U.n2hmx[c] = -2.0 * U.hmx[c];
        U.n2hmy[c] = -2.0 * U.hmy[c];
        U.hmxi[c] = U.hmx[c] * U.idx * U.idx;
        U.hmyi[c] = U.hmy[c] * U.idx * U.idx;
        U.hhmx[c] = 0.5 * U.hmxi[c];
        U.hhmy[c] = 0.5 * U.hmyi[c];
        U.jmx[c] = U.hmx[c] * U.qi[c];
        U.jmy[c] = U.hmy[c] * U.qi[c];
        U.a2[c] = 2.0 * U.a[c] * U.dx2;
        U.b2[c] = 2.0 * U.b[c] * U.dx2;
    }
    U.idx4 = 0.25 * U.idx;
    U.idx8 = 0.125 * U.idx * U.idx;
    U.etad = U.eta * U.dx2;
    U.gammad = U.gamma * U.dx2;
    U.deltad = U.delta * U.dx2;
    U.hd = U.h * U.dx;
    U.hl = 0.0;
}

// Rounded once from double: to float, or split into a float pair.
template <class T>
inline void round_uniform(Uniform<T> &r, const Uniform<double> &U)
{
    for (int c = 0; c < 2; ++c) {
        r.a[c] = T(U.a[c]);
        r.b[c] = T(U.b[c]);
        r.hmx[c] = T(U.hmx[c]);
        r.hmy[c] = T(U.hmy[c]);
        r.aob[c] = T(U.aob[c]);
        r.q[c] = T(U.q[c]);
        r.qd[c] = T(U.qd[c]);
        r.hqd[c] = T(U.hqd[c]);
        r.nhqd[c] = T(U.nhqd[c]);
        r.kq[c] = T(U.kq[c]);
        r.qi[c] = T(U.qi[c]);
        r.n2hmx[c] = T(U.n2hmx[c]);
        r.n2hmy[c] = T(U.n2hmy[c]);
        r.hmxi[c] = T(U.hmxi[c]);
        r.hmyi[c] = T(U.hmyi[c]);
        r.hhmx[c] = T(U.hhmx[c]);
        r.hhmy[c] = T(U.hhmy[c]);
        r.jmx[c] = T(U.jmx[c]);
        r.jmy[c] = T(U.jmy[c]);
        r.a2[c] = T(U.a2[c]);
        r.b2[c] = T(U.b2[c]);
    }
    r.eta = T(U.eta);
    r.gamma = T(U.gamma);
    r.delta = T(U.delta);
    r.h = T(U.h);
    r.idx = T(U.idx);
    r.dx2 = T(U.dx2);
    r.dx = T(U.dx);
    r.etad = T(U.etad);
    r.gammad = T(U.gammad);
    r.deltad = T(U.deltad);
    r.hd = T(U.hd);
    r.hl = T(std::is_same<T, float>::value ? (U.h - (double)(float)U.h) * U.dx : 0.0);
    r.idx4 = T(U.idx4);
    r.idx8 = T(U.idx8);
}

// Per-site parameters as float pairs, with what a site's stencils divide formed
// once: a, b, 1 / (2 m_xx), 1 / (2 m_yy), a / b, and h.  Ten FP64 divisions and the
// conversions of fifteen doubles per site and pass made ten float-float steps of 200
// x 160 x 24, two components, 6.1 ms; they take 3.2 this way (5.5 as tiles).
struct PairSites {
    const void *a[2], *b[2], *hmx[2], *hmy[2], *aob[2], *h;
};

// One string (one lattice, F images) as seen by the kernels.  Field buffers
// hold three arrays each (A, psi_1, psi_2) of F*nx*ny pairs; psi_2 is null
// for one component.  Buffers: x (state, ping-pong), g (gradient, two
// slots), d (direction, ping-pong).
struct StringDesc {
    int nx, ny, F, ncomp;
    int tiles_x;              // strips across an image
    int img_base;             // first global image index of this string
    int rows;                 // rows per warp strip of the NLCG passes
    int grows, gper;          // rows per group of their sums, groups per strip
    int groups, part_base;    // groups of an image (all columns); first global group index
    int stiles_y, stile_base; // strips down an image; first global strip index
    int wrows, wtiles_y;      // the same of the walks over one string (walk.cuh)
    int thin_film;
    int disc;                 // 0: the reference's linearised differences, 1: gauge links
    int per_site;             // 1: parameters read from the arrays below
    Uniform<float> uf;
    Uniform<double> ud;
    Uniform<ff> uff;          // ud split into float pairs (paired FP64 mode)
    const void *pa[2], *pb[2], *pmxx[2], *pmyy[2], *ph;  // per-site (type T)
    PairSites pairs;          // the same as the float-float passes read them
    const uint16_t *mask;     // per site: comp code | sc code << 8
    const int32_t *code_comp, *code_sc;   // used when mask is null: int32 codes per site
    void *x[2][3], *g[2][3], *d[2][3];

    template <class T> __host__ __device__ const Uniform<T> &u() const;
};
template <> __host__ __device__ inline const Uniform<float> &StringDesc::u<float>() const { return uf; }
template <> __host__ __device__ inline const Uniform<double> &StringDesc::u<double>() const { return ud; }
template <> __host__ __device__ inline const Uniform<ff> &StringDesc::u<ff>() const { return uff; }

// Descriptors of the strings covered by one launch; passed by value as a
// __grid_constant__ kernel parameter, i.e. read through the constant cache.
// Launches of a single string pass only its own: every launch copies its
// parameters, and sixteen descriptors are 20 KB of them.
template <int N>
struct BatchOf {
    int n;
    StringDesc s[N];
};
using Batch = BatchOf<MAX_STRINGS>;
template <bool ONE> using batch_t = BatchOf<ONE ? 1 : MAX_STRINGS>;

struct StripRef {
    int s;        // string within the batch
    int ty, tx;   // strip row and column
    int n;        // image
};

// Per-image scalars of the whole context (index = img_base + n).
struct Scalars {
    double *gn0, *gn1;    // |g|^2, two slots (nlcgSteps' g_norm2 / g_norm2_old)
    double *gdg;          // g . (g - g_prev)
    double *beta;         // Polak-Ribiere coefficient of the last step
    double *alpha;        // step of the last line search (reported)
    double *alpha_pend;   // step not yet applied to x (0 = nothing pending)
    double *fenergy;      // energy (polynomial constant term)
    double *poly;         // [img][4] = B, C, D, E
    double *part;         // partial sums, [group of rows of a strip][8]
    unsigned *ticket;     // per-image arrival counters
    double *xtab_f, *xtab_d;   // line-search grid x_p, p = 0..2000, rounded to float / double
    int *status;          // device-side error flags
};

__device__ __forceinline__ unsigned bit(unsigned c, int n) { return (c >> n) & 1u; }

// Block-wide sum of NV values; a pairwise tree in T inside each warp, then
// across the warps in float (FP32 fields) or double (the others).  Result
// (double) valid in thread 0.
template <int NV, class T>
__device__ __forceinline__ void block_sum(const T (&v)[NV], double (&out)[NV], double *smem /* NT/32*NV */)
{
    T w[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        w[k] = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w[k] += shfl_down(w[k], o);
    }
    const int wi = threadIdx.x >> 5, l = threadIdx.x & 31;
    if constexpr (std::is_same<T, float>::value) {
        // FP32 fields: the eight warp sums are added in float too (the FP64
        // pipe is scarce; one conversion per quantity and block)
        float *fs = reinterpret_cast<float *>(smem);
        if (l == 0)
#pragma unroll
            for (int k = 0; k < NV; ++k) fs[wi * NV + k] = w[k];
        __syncthreads();
        if (threadIdx.x < 32) {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                float t = (l < NT / 32) ? fs[l * NV + k] : 0.0f;
#pragma unroll
                for (int o = NT / 64; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
                out[k] = (double)t;
            }
        }
    } else {
        if (l == 0)
#pragma unroll
            for (int k = 0; k < NV; ++k) smem[wi * NV + k] = (double)w[k];
        __syncthreads();
        if (threadIdx.x < 32) {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                double t = (l < NT / 32) ? smem[l * NV + k] : 0.0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
                out[k] = t;
            }
        }
    }
    __syncthreads();
}

}  // namespace mepgl
