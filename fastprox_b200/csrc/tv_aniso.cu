// Anisotropic image TV on sm_100a: the reference's own method, replayed per
// image on the device.
//
// Two active axes: the accelerated dual block proximal gradient method
// (ADBPG) of TVAniso::adbpg (src/ops/tv_aniso.cpp:429-530): per iteration an
// exact 1D TV prox of every fibre along the axis of smaller stride (a1) and
// then along the other (a2), the dual update with extrapolation, the gradient
// restart every 4 iterations (Restart, :357-367), gap checks on the adaptive
// CheckSchedule (:396-414), and the polish on the PolishSchedule (:382-391)
// that reads the flat regions off the dual and solves on them exactly
// (try_polish, :886-953). Three active axes: FDPG for three terms
// (TVAniso::fdpg3, :534-616). One active axis: a single exact pass.
//
// Each image carries a stage (iterate, check, polish, final, done); every
// kernel acts only on the images in its stage, and the last block of an
// image (a ticket per image) advances the stage with the scalar logic of the
// reference in FP64. The host issues the same round of launches until no
// image is live. The 1D steps are Condat's algorithm, several lanes per fibre
// (tv1d.cuh). Components of the polish are found by union-find with atomic
// hooking of the larger root to the smaller (so every root is the smallest
// index of its component, whatever the order), and region sums use 64-bit
// fixed point, so every result is the same bit for bit on every run.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "aniso.h"
#include "common.cuh"
#include "tv1d.cuh"

namespace fpb {
namespace {

constexpr int kCheck = 4;               // tv_aniso.cpp:76
constexpr double kPolishDrop = 0.1;     // :78
constexpr double kPolishEta = 1e-9;     // :81, for FP64 duals
// FP32 duals carry rounding near 1e-7 of the bound: the margin of the
// reference's own device path for float32, max(1e-9, 64 eps)
// (bindings/python/fastprox/_tv_torch.py dual_eta).
template <class T>
__device__ __forceinline__ double polish_eta() {
    return sizeof(T) == 4 ? 64.0 * 1.1920928955078125e-07 : kPolishEta;
}
constexpr double kPolishRatio = 0.01;   // :86
constexpr int kThreads = 256;

template <class T>
__device__ __forceinline__ T ldexp_t(T v, int e);
template <>
__device__ __forceinline__ float ldexp_t<float>(float v, int e) { return ldexpf(v, e); }
template <>
__device__ __forceinline__ double ldexp_t<double>(double v, int e) { return ldexp(v, e); }

struct Fib {
    int64_t s, L, nfib;
    __device__ __forceinline__ int64_t base(int64_t f) const { return (f / s) * L * s + (f % s); }
};

__device__ __forceinline__ Fib fibers(const AnGeom &g, int a) {
    Fib f;
    f.s = g.S[a];
    f.L = g.L[a];
    f.nfib = g.N / g.L[a];
    return f;
}

// The image of launch slot z in a round (-1: none, the live list is shorter).
__device__ __forceinline__ int round_image(const AnBuffers &bf, unsigned z) {
    if (!bf.lmap) return (int)z;
    return (int)z < *bf.lcnt ? bf.lmap[z] : -1;
}

// The live images in order (one block).
__global__ void __launch_bounds__(1024) an_live_list(const AnState *st, int64_t B, int *lmap, int *lcnt) {
    __shared__ int wsum[32];
    __shared__ int base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int64_t c0 = 0; c0 < B; c0 += blockDim.x) {
        const int64_t i = c0 + threadIdx.x;
        const int f = (i < B && st[i].status == kLive) ? 1 : 0;
        int x = f;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int w = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            wsum[lane] = w;
        }
        __syncthreads();
        const int before = base + (wid > 0 ? wsum[wid - 1] : 0) + x - f;
        if (f) lmap[before] = (int)i;
        __syncthreads();
        if (threadIdx.x == 0) base += wsum[(blockDim.x >> 5) - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) *lcnt = base;
}

__device__ __forceinline__ double *img_part(const AnBuffers &bf, int b) { return bf.part + (int64_t)b * bf.max_part * 2; }

// Ends a per-image reduction: block partial (two sums) to part, and in the
// last block of the image the totals. Returns true in thread 0 of that block.
__device__ __forceinline__ bool reduce2(const AnBuffers &bf, int b, unsigned blk, unsigned nblk, double a0,
                                        double a1, double *sh, int *flag, double &t0, double &t1) {
    const double s0 = block_sum(a0, sh);
    const double s1 = block_sum(a1, sh);
    double *part = img_part(bf, b);
    if (threadIdx.x == 0) {
        part[blk * 2 + 0] = s0;
        part[blk * 2 + 1] = s1;
    }
    if (!arrive_last(bf.ticket + b, nblk, flag)) return false;
    t0 = sum_partials(part, nblk, 2, 0, sh);
    t1 = sum_partials(part, nblk, 2, 1, sh);
    if (threadIdx.x != 0) return false;
    bf.ticket[b] = 0;
    return true;
}

// The same over a partition of an image's pixels into nch chunks (chunk q: the
// pixels q T + t + j nch T of thread t of T) that does not depend on the grid:
// each block takes chunks in turn, acc(p) summed over a thread's pixels of the
// chunk. Batches launch few blocks per image, so that a launch whose images are
// all in other stages costs little (64 x 512^2: 16384 blocks that return at
// once took 35 us, 2368 take 5).
template <class F>
__device__ __forceinline__ bool reduce_chunks(const AnBuffers &bf, int b, int64_t N, int nch, const F &term, double *sh,
                                              int *flag, double &total) {
    double *part = img_part(bf, b);
    for (int q = blockIdx.x; q < nch; q += gridDim.x) {
        double acc = 0.0;
        for (int64_t p = (int64_t)q * blockDim.x + threadIdx.x; p < N; p += (int64_t)nch * blockDim.x) acc += term((int)p);
        const double s0 = block_sum(acc, sh);
        if (threadIdx.x == 0) part[q * 2] = s0;
    }
    if (!arrive_last(bf.ticket + b, gridDim.x, flag)) return false;
    total = sum_partials(part, nch, 2, 0, sh);
    if (threadIdx.x != 0) return false;
    bf.ticket[b] = 0;
    return true;
}

// Chunks of an image (blocks of a launch over one image), at most 256.
__host__ __device__ __forceinline__ int pixel_chunks(int64_t N) {
    const int64_t nb = (N + kThreads * 4 - 1) / (kThreads * 4);
    return (int)(nb < 1 ? 1 : (nb > 256 ? 256 : nb));
}

// The coordinates of pixel p (axis 0 slowest).
__device__ __forceinline__ void coords(const AnGeom &g, int p, int co[3]) {
    unsigned q = (unsigned)p;
#pragma unroll
    for (int a = 2; a >= 0; --a) {
        co[a] = 0;
        if (a >= g.k) continue;
        if (a == 0) {
            co[0] = (int)q;
        } else {
            const unsigned L = (unsigned)g.L[a], t = q / L;
            co[a] = (int)(q - t * L);
            q = t;
        }
    }
}

// ---------------------------------------------------------------------------
// Set-up (tv_aniso.cpp:260-340)
// ---------------------------------------------------------------------------

template <class T>
__global__ void __launch_bounds__(kThreads) an_scan1(const T *__restrict__ x, AnGeom g, AnCall c, AnBuffers bf) {
    __shared__ double sh[32];
    __shared__ int flag;
    const int b = blockIdx.y;
    const int64_t N = g.N;
    const T *xb = x + (int64_t)b * N;
    T *db = static_cast<T *>(bf.d) + (int64_t)b * N;
    double m = 0.0;
    int fl = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
        const T v = xb[i];
        if (xb != db) db[i] = v;
        const double a = fabs((double)v);
        if (isnan(a)) fl |= 1;
        else if (isinf(a)) fl |= 2;
        else m = fmax(m, a);
    }
    const double mb = block_max(m, sh);
    const double f1 = block_max((double)(fl & 1), sh);
    const double f2 = block_max((double)((fl >> 1) & 1), sh);
    double *part = img_part(bf, b);
    if (threadIdx.x == 0) {
        part[blockIdx.x * 2 + 0] = mb;
        part[blockIdx.x * 2 + 1] = f1 + 2.0 * f2;
    }
    if (!arrive_last(bf.ticket + b, gridDim.x, &flag)) return;
    const double mx = max_partials(part, gridDim.x, 2, 0, sh);
    double o1 = 0.0, o2 = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
        const int code = (int)__ldcg(part + i * 2 + 1);
        o1 = fmax(o1, (double)(code & 1));
        o2 = fmax(o2, (double)((code >> 1) & 1));
    }
    o1 = block_max(o1, sh);
    o2 = block_max(o2, sh);
    if (threadIdx.x != 0) return;
    bf.ticket[b] = 0;
    AnImage im{};
    im.gamma_in = bf.gammas[b];
    im.maxabs = mx;
    im.flags = (o1 > 0.0 ? 1 : 0) | (o2 > 0.0 ? 2 : 0);
    int na = 0;
    for (int a = 0; a < 3; ++a) {
        im.lam[a] = 0.0;
        if (a < g.k) {
            const double l = im.gamma_in * c.w[a];
            if (l > 0.0 && g.L[a] > 1) {
                im.lam[a] = l;
                ++na;
            }
        }
    }
    im.na = na;
    if (im.flags & 2) im.mode = kAnInf;
    else if (im.flags & 1) im.mode = kAnNan;
    else if (na == 0) im.mode = kAnIdentity;
    else if (na == 1) im.mode = kAnSingle;
    else im.mode = na == 2 ? kAnAdbpg : kAnFdpg3;
    int e = 0;
    if (na > 0 && mx > 0.0) {  // rescale_exponent (src/ops/image_util.hpp:56-65)
        const double gamma = im.gamma_in;
        e = ilogb(mx);
        if (e >= -64 && e <= 64) {
            e = 0;
        } else {
            const double top = fmax(gamma, gamma * c.step_scale);
            if (e < 0 && top > 0.0) e = min(0, max(e, ilogb(top) + 1 - 960));
        }
        for (int a = 0; a < 3 && e; ++a)
            if (im.lam[a] > 0.0 && !(ldexp(im.lam[a], -e) > 0.0)) e = 0;
    }
    im.e = e;
    for (int a = 0; a < 3; ++a) im.lam[a] = e ? ldexp(im.lam[a], -e) : im.lam[a];
    // the active axes of ADBPG: a1 of the smaller stride (tv_aniso.cpp:432-433)
    int act[3], n = 0;
    for (int a = 0; a < g.k; ++a)
        if (im.lam[a] > 0.0) act[n++] = a;
    im.a1 = n >= 2 ? (g.S[act[0]] < g.S[act[1]] ? act[0] : act[1]) : (n ? act[0] : 0);
    im.a2 = n >= 2 ? (im.a1 == act[0] ? act[1] : act[0]) : 0;
    // the fixed-point scale of the polish's region sums: |zp| <= max|d| + 2 k lam_max beta_max
    double lmax = 0.0;
    for (int a = 0; a < 3; ++a) lmax = fmax(lmax, im.lam[a]);
    const double zb = ldexp(mx, -e) + 2.0 * g.k * lmax * c.beta_max + 1e-300;
    int lgN = 0;
    while ((1LL << lgN) <= g.N) ++lgN;
    im.fx_shift = 61 - lgN - (ilogb(zb) + 1);
    bf.img[b] = im;
    AnState st{};
    st.status = (im.mode == kAnAdbpg || im.mode == kAnFdpg3) ? kLive : kFinished;
    st.stage = kStIter;
    st.tn = fista_t(1.0);
    st.beta = 0.0;
    st.gp = CUDART_INF;
    st.chk_next = 1;
    st.chk_prev_it = -1;
    st.pol_next = CUDART_INF;
    bf.st[b] = st;
    if (st.status == kLive) atomicAdd(bf.live, 1);
}

// d *= 2^-e, |d|^2 -> target (tv_aniso.cpp:329-337)
template <class T>
__global__ void __launch_bounds__(kThreads) an_scan2(AnGeom g, AnCall c, AnBuffers bf) {
    __shared__ double sh[32];
    __shared__ int flag;
    const int b = blockIdx.y;
    const int mode = bf.img[b].mode;
    if (mode == kAnNan || mode == kAnInf) return;
    const int e = bf.img[b].e;
    T *db = static_cast<T *>(bf.d) + (int64_t)b * g.N;
    double s2 = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.N; i += (int64_t)gridDim.x * blockDim.x) {
        T v = db[i];
        if (e) {
            v = ldexp_t(v, -e);
            db[i] = v;
        }
        s2 += (double)v * (double)v;
    }
    double t0, t1;
    if (!reduce2(bf, b, blockIdx.x, gridDim.x, s2, 0.0, sh, &flag, t0, t1)) return;
    bf.img[b].dd = t0;
    bf.img[b].target = c.tol * 0.5 * t0;
}

// ---------------------------------------------------------------------------
// Fibre passes of the iteration
// ---------------------------------------------------------------------------

// Edge weight of the edge (o, o + S[a]) times nothing (beta), or 1.
template <class T>
struct BetaW {
    const T *p;
    int64_t s;
    __device__ __forceinline__ double operator()(int64_t i) const { return (double)p[i * s]; }
};

// One exact 1D TV prox on fibre f of axis a of image b: in(i) -> out(i, v).
template <class T, class In, class Out>
__device__ __forceinline__ void fibre_prox(const AnCall &c, const AnBuffers &bf, int a, int64_t base, const Fib &fb,
                                           double lam, const In &in, const Out &out) {
    if (c.has_beta) {
        const T *bw = static_cast<const T *>(bf.beta) + (int64_t)a * c.N + base;
        tv1d_fiber<T>(in, out, (int)fb.L, lam, true, BetaW<T>{bw, fb.s}, DivRecip<T>{});
    } else {
        tv1d_fiber<T>(in, out, (int)fb.L, lam, false, NoWeight{}, DivRecip<T>{});
    }
}

// ADBPG first block step: u = prox_{g1}(d + w) along a1 (tv_aniso.cpp:459-460).
template <class T>
__global__ void __launch_bounds__(128) an_pass1(AnGeom g, AnCall c, AnBuffers bf) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || (st.stage != kStIter && st.stage != kStWarm)) return;
    const AnImage &im = bf.img[b];
    if (im.mode != kAnAdbpg) return;
    const int a = im.a1;
    const Fib fb = fibers(g, a);
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= fb.nfib) return;
    const int64_t N = g.N, base = fb.base(f), s = fb.s;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N + base;
    const T *Wv = static_cast<const T *>(bf.wv) + (int64_t)b * g.k * N + base;
    T *U = static_cast<T *>(bf.u) + (int64_t)b * N + base;
    auto in = [D, Wv, s](int64_t i) -> double { return (double)(D[i * s] + Wv[i * s]); };
    auto out = [U, s](int64_t i, double v) { U[i * s] = (T)v; };
    fibre_prox<T>(c, bf, a, base, fb, im.lam[a], in, out);
}

// ADBPG second block step along a2 with the dual update and extrapolation
// (tv_aniso.cpp:461-80); the last block runs the restart test, advances the
// iteration and decides whether a gap check is due.
template <class T>
__global__ void __launch_bounds__(128) an_pass2(AnGeom g, AnCall c, AnBuffers bf) {
    __shared__ double sh[32];
    __shared__ int flag;
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState st = bf.st[b];
    if (st.status != kLive || st.stage != kStIter) return;
    const AnImage &im = bf.img[b];
    if (im.mode != kAnAdbpg) return;
    const int a = im.a2;
    const Fib fb = fibers(g, a);
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t N = g.N;
    const bool test = st.it % kCheck == 0;
    const T beta = (T)st.beta;
    double up = 0.0;
    if (f < fb.nfib) {
        const int64_t base = fb.base(f), s = fb.s;
        const T *U = static_cast<const T *>(bf.u) + (int64_t)b * N + base;
        T *Wv = static_cast<T *>(bf.wv) + (int64_t)b * g.k * N + base;
        T *Y = static_cast<T *>(bf.y) + (int64_t)b * g.k * N + base;
        T *Z = static_cast<T *>(bf.z) + (int64_t)b * N + base;
        auto in = [U, Wv, s](int64_t i) -> double { return (double)(U[i * s] - Wv[i * s]); };
        auto out = [Z, s](int64_t i, double v) { Z[i * s] = (T)v; };
        fibre_prox<T>(c, bf, a, base, fb, im.lam[a], in, out);
        for (int64_t i = 0; i < fb.L; ++i) {
            const int64_t o = i * s;
            const T v = U[o] - Wv[o];
            const T yn = Z[o] - v;
            const T y = Y[o], w = Wv[o];
            if (test) up += (double)((w - yn) * (yn - y));
            Wv[o] = yn + beta * (yn - y);
            Y[o] = yn;
        }
    }
    double dot, unused;
    if (!reduce2(bf, b, blockIdx.x, gridDim.x, test ? up : 0.0, 0.0, sh, &flag, dot, unused)) return;
    AnState s2 = st;
    // Restart (tv_aniso.cpp:357-367): ++since; restart when test && up > 0 && since >= last
    s2.since += 1;
    double t = s2.tn;
    if (test && dot > 0.0 && s2.since >= s2.last) {
        s2.last = s2.since;
        s2.since = 0;
        s2.restart = 1;
        t = 1.0;
    } else {
        s2.restart = 0;
    }
    s2.it += 1;
    const double tn = fista_t(t);
    s2.beta = (t - 1.0) / tn;
    s2.tn = tn;
    if (s2.it == s2.chk_next || s2.it == c.max_iter) s2.stage = kStCheck;
    bf.st[b] = s2;
}

// ---------------------------------------------------------------------------
// Fibre tiles in shared memory
// ---------------------------------------------------------------------------
//
// A thread walking one fibre through global memory waits a memory latency at
// every step of Condat's scan (each step depends on the last), and a batch has
// only as many fibres as rows or columns: the passes above run latency-bound
// at a few percent of the memory bandwidth. The tiled passes copy the inputs of
// fb fibres (and their edge weights) into shared memory first, with loads
// that do not depend on one another and are coalesced (along the fibre when
// fibres are contiguous, across fibres otherwise), run the scans out of shared
// memory (the result overwrites the input: Condat never reads back an entry it
// has written), and store the results the same way. A tile is L x (fb + 1)
// entries (the odd row length keeps both copy directions free of bank
// conflicts; thread t of the scan always reads bank t + i mod 32). The values
// and their order of operations are those of the untiled passes.

struct TileCfg {
    int fb[3];  // fibres per block along each axis (0: the axis does not fit)
};

template <class T>
struct TileIn {
    const T *s;
    int P, t;
    __device__ __forceinline__ T operator()(int i) const { return s[i * P + t]; }
};
// A segment writes its value at its last entry and marks it (one bit per
// entry, word i / 32 of the fibre's column); finish fills each segment's
// other entries from its end, backwards, and clears the marks.
template <class T>
struct TileSink {
    T *s;
    unsigned *m;
    int P, t;
    __device__ __forceinline__ void segment(int, int k1, double v) const {
        s[k1 * P + t] = (T)v;
        m[(k1 >> 5) * P + t] |= 1u << (k1 & 31);
    }
    __device__ __forceinline__ void finish(int n) const {
        T v = T(0);
        for (int w = (n - 1) >> 5; w >= 0; --w) {
            const unsigned bits = m[w * P + t];
            m[w * P + t] = 0u;
            const int top = (w << 5) + 31 < n - 1 ? (w << 5) + 31 : n - 1;
            for (int i = top; i >= (w << 5); --i) {
                const int j = i * P + t;
                if (bits & (1u << (i & 31))) v = s[j];
                else s[j] = v;
            }
        }
    }
};

// tile[i][r] = ld(o) for the block's nv fibres, o the entry's offset in the image
template <class T, class Ld>
__device__ __forceinline__ void tile_load(T *tile, int P, const Fib &fb, int64_t f0, int nv, const Ld &ld) {
    const int L = (int)fb.L, n = nv * L;
    if (fb.s == 1) {
        for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
            const int r = idx / L, i = idx - r * L;
            tile[i * P + r] = ld(fb.base(f0 + r) + i);
        }
    } else {
        for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
            const int i = idx / nv, r = idx - i * nv;
            tile[i * P + r] = ld(fb.base(f0 + r) + (int64_t)i * fb.s);
        }
    }
}

// st(o, tile[i][r]) for the block's nv fibres, in the order of tile_load
template <class T, class St>
__device__ __forceinline__ void tile_store(const T *tile, int P, const Fib &fb, int64_t f0, int nv, const St &st) {
    const int L = (int)fb.L, n = nv * L;
    if (fb.s == 1) {
        for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
            const int r = idx / L, i = idx - r * L;
            st(fb.base(f0 + r) + i, tile[i * P + r]);
        }
    } else {
        for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
            const int i = idx / nv, r = idx - i * nv;
            st(fb.base(f0 + r) + (int64_t)i * fb.s, tile[i * P + r]);
        }
    }
}

// The tiles of a block in shared memory: the fibres' inputs (then results),
// their edge weights when there are any, one mark bit per entry, and the
// reciprocals 1/m (m <= L) of the scans.
template <class T>
struct Tiles {
    T *in, *w, *rc;
    unsigned *mk;
    __device__ __forceinline__ Tiles(unsigned char *smem, const AnCall &c, int L, int P) {
        in = reinterpret_cast<T *>(smem);
        w = in + L * P;
        mk = reinterpret_cast<unsigned *>(in + (c.has_beta ? 2 : 1) * L * P);
        const int nw = ((L + 31) >> 5) * P;
        rc = reinterpret_cast<T *>(mk + ((nw + 1) & ~1));
        for (int i = threadIdx.x; i < nw; i += blockDim.x) mk[i] = 0u;
        const DivRecip<T> div;
        for (int m = threadIdx.x; m <= L; m += blockDim.x) rc[m] = m ? div(m) : T(0);
    }
};

// Shared-memory bytes of a tile of fb fibres of L entries.
__host__ __device__ __forceinline__ size_t tile_bytes(int L, int fb, int nbuf, size_t tsize) {
    const size_t P = (size_t)fb + 1;
    const size_t nw = (((size_t)L + 31) / 32) * P;
    return (size_t)nbuf * tsize * (size_t)L * P + 4 * ((nw + 1) & ~(size_t)1) + tsize * ((size_t)L + 1);
}

// The scans of a loaded tile (edge weights in the second tile when present),
// by the block's first warp, lane t on fibre t, in lockstep (tv1d_warp).
template <class T>
__device__ __forceinline__ void tile_scan(const AnCall &c, const Tiles<T> &tl, int P, int nv, int L, double lam) {
    const int t = threadIdx.x;
    if (t >= 32) return;
    const TileIn<T> in{tl.in, P, t};
    const TileSink<T> out{tl.in, tl.mk, P, t};
    if (c.has_beta) tv1d_warp<T>(in, out, L, lam, true, TileIn<T>{tl.w, P, t}, TableRecip<T>{tl.rc}, t < nv);
    else tv1d_warp<T>(in, out, L, lam, false, NoWeight{}, TableRecip<T>{tl.rc}, t < nv);
}

// Threads of a tile block: all copy the tiles in and out, the first warp scans.
constexpr int kTileThreads = 128;

// an_pass1 on tiles
template <class T>
__global__ void __launch_bounds__(kTileThreads) an_pass1_tile(AnGeom g, AnCall c, AnBuffers bf, TileCfg tc) {
    extern __shared__ __align__(16) unsigned char an_smem[];
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || (st.stage != kStIter && st.stage != kStWarm)) return;
    const AnImage &im = bf.img[b];
    if (im.mode != kAnAdbpg) return;
    const int a = im.a1;
    const Fib fb = fibers(g, a);
    const int FB = tc.fb[a];
    const int64_t f0 = (int64_t)blockIdx.x * FB;
    if (f0 >= fb.nfib) return;
    const int nv = (int)(fb.nfib - f0 < FB ? fb.nfib - f0 : FB), P = FB + 1;
    const Tiles<T> tl(an_smem, c, (int)fb.L, P);
    const int64_t N = g.N;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N;
    const T *Wv = static_cast<const T *>(bf.wv) + (int64_t)b * g.k * N;
    tile_load(tl.in, P, fb, f0, nv, [D, Wv](int64_t o) { return (T)(D[o] + Wv[o]); });
    if (c.has_beta) {
        const T *bw = static_cast<const T *>(bf.beta) + (int64_t)a * c.N;
        tile_load(tl.w, P, fb, f0, nv, [bw](int64_t o) { return bw[o]; });
    }
    __syncthreads();
    tile_scan(c, tl, P, nv, (int)fb.L, im.lam[a]);
    __syncthreads();
    T *U = static_cast<T *>(bf.u) + (int64_t)b * N;
    tile_store(tl.in, P, fb, f0, nv, [U](int64_t o, T v) { U[o] = v; });
}

// an_pass2 on tiles, with the dual update, the extrapolation and the restart
// logic of an_pass2
template <class T>
__global__ void __launch_bounds__(kTileThreads) an_pass2_tile(AnGeom g, AnCall c, AnBuffers bf, TileCfg tc) {
    extern __shared__ __align__(16) unsigned char an_smem[];
    __shared__ double sh[32];
    __shared__ int flag;
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState st = bf.st[b];
    if (st.status != kLive || st.stage != kStIter) return;
    const AnImage &im = bf.img[b];
    if (im.mode != kAnAdbpg) return;
    const int a = im.a2;
    const Fib fb = fibers(g, a);
    const int FB = tc.fb[a];
    const int64_t f0 = (int64_t)blockIdx.x * FB;
    const int64_t N = g.N;
    const bool test = st.it % kCheck == 0;
    const T beta = (T)st.beta;
    double up = 0.0;
    if (f0 < fb.nfib) {
        const int nv = (int)(fb.nfib - f0 < FB ? fb.nfib - f0 : FB), P = FB + 1;
        const Tiles<T> tl(an_smem, c, (int)fb.L, P);
        const T *U = static_cast<const T *>(bf.u) + (int64_t)b * N;
        T *Wv = static_cast<T *>(bf.wv) + (int64_t)b * g.k * N;
        T *Y = static_cast<T *>(bf.y) + (int64_t)b * g.k * N;
        T *Z = static_cast<T *>(bf.z) + (int64_t)b * N;
        tile_load(tl.in, P, fb, f0, nv, [U, Wv](int64_t o) { return (T)(U[o] - Wv[o]); });
        if (c.has_beta) {
            const T *bw = static_cast<const T *>(bf.beta) + (int64_t)a * c.N;
            tile_load(tl.w, P, fb, f0, nv, [bw](int64_t o) { return bw[o]; });
        }
        __syncthreads();
        tile_scan(c, tl, P, nv, (int)fb.L, im.lam[a]);
        __syncthreads();
        tile_store(tl.in, P, fb, f0, nv, [&](int64_t o, T z) {
            const T v = U[o] - Wv[o];
            const T yn = z - v;
            const T y = Y[o], w = Wv[o];
            if (test) up += (double)((w - yn) * (yn - y));
            Wv[o] = yn + beta * (yn - y);
            Y[o] = yn;
            Z[o] = z;
        });
    }
    double dot, unused;
    if (!reduce2(bf, b, blockIdx.x, gridDim.x, test ? up : 0.0, 0.0, sh, &flag, dot, unused)) return;
    AnState s2 = st;
    s2.since += 1;
    double t = s2.tn;
    if (test && dot > 0.0 && s2.since >= s2.last) {
        s2.last = s2.since;
        s2.since = 0;
        s2.restart = 1;
        t = 1.0;
    } else {
        s2.restart = 0;
    }
    s2.it += 1;
    const double tn = fista_t(t);
    s2.beta = (t - 1.0) / tn;
    s2.tn = tn;
    if (s2.it == s2.chk_next || s2.it == c.max_iter) s2.stage = kStCheck;
    bf.st[b] = s2;
}

// an_fdpg3_pass on tiles (blockIdx.y = axis)
template <class T>
__global__ void __launch_bounds__(kTileThreads) an_fdpg3_tile(AnGeom g, AnCall c, AnBuffers bf, TileCfg tc) {
    extern __shared__ __align__(16) unsigned char an_smem[];
    __shared__ double sh[32];
    __shared__ int flag;
    const int b = round_image(bf, blockIdx.z);
    if (b < 0) return;
    const AnState st = bf.st[b];
    if (st.status != kLive || st.stage != kStIter) return;
    const AnImage &im = bf.img[b];
    if (im.mode != kAnFdpg3) return;
    const int64_t N = g.N;
    const bool test = st.it % kCheck == 0;
    const T beta = (T)st.beta;
    double up = 0.0;
    const int a = blockIdx.y;
    const Fib fb = fibers(g, a);
    const int FB = tc.fb[a];
    const int64_t f0 = (int64_t)blockIdx.x * FB;
    if (f0 < fb.nfib) {
        const int nv = (int)(fb.nfib - f0 < FB ? fb.nfib - f0 : FB), P = FB + 1;
        const Tiles<T> tl(an_smem, c, (int)fb.L, P);
        const T *U = static_cast<const T *>(bf.u) + (int64_t)b * N;
        T *Wa = static_cast<T *>(bf.wv) + ((int64_t)b * 3 + a) * N;
        T *Ya = static_cast<T *>(bf.y) + ((int64_t)b * 3 + a) * N;
        // the three axes write disjoint scratch: zp (a = 0), z (a = 1), dual slot (a = 2)
        T *Za = static_cast<T *>(bf.zp) + (int64_t)b * N;
        if (a == 1) Za = static_cast<T *>(bf.z) + (int64_t)b * N;
        if (a == 2) Za = static_cast<T *>(bf.scratch) + (int64_t)b * N;
        tile_load(tl.in, P, fb, f0, nv, [U, Wa](int64_t o) { return (T)(U[o] - T(3) * Wa[o]); });
        if (c.has_beta) {
            const T *bw = static_cast<const T *>(bf.beta) + (int64_t)a * c.N;
            tile_load(tl.w, P, fb, f0, nv, [bw](int64_t o) { return bw[o]; });
        }
        __syncthreads();
        tile_scan(c, tl, P, nv, (int)fb.L, 3.0 * im.lam[a]);
        __syncthreads();
        tile_store(tl.in, P, fb, f0, nv, [&](int64_t o, T z) {
            const T v = U[o] - T(3) * Wa[o];
            const T yn = (z - v) / T(3);
            const T y = Ya[o], w = Wa[o];
            if (test) up += (double)((w - yn) * (yn - y));
            Wa[o] = yn + beta * (yn - y);
            Ya[o] = yn;
            Za[o] = z;
        });
    }
    double dot, unused;
    const unsigned nblk = gridDim.x * gridDim.y;
    const unsigned blk = blockIdx.y * gridDim.x + blockIdx.x;
    if (!reduce2(bf, b, blk, nblk, test ? up : 0.0, 0.0, sh, &flag, dot, unused)) return;
    AnState s2 = st;
    s2.since += 1;
    double t = s2.tn;
    if (test && dot > 0.0 && s2.since >= s2.last) {
        s2.last = s2.since;
        s2.since = 0;
        s2.restart = 1;
        t = 1.0;
    } else {
        s2.restart = 0;
    }
    s2.it += 1;
    const double tn = fista_t(t);
    s2.beta = (t - 1.0) / tn;
    s2.tn = tn;
    if (s2.it % kCheck == 0 || s2.it == c.max_iter) s2.stage = kStCheck;
    bf.st[b] = s2;
}

// ---------------------------------------------------------------------------
// Fibre passes by pieces
// ---------------------------------------------------------------------------
//
// One kernel per pass of ADBPG: a block stages the inputs of its fibres (and
// their radii) in shared memory, coalesced along the fibre when fibres are
// contiguous and across fibres otherwise, scans every fibre by P pieces at
// once (tv1d.cuh, PieceScan: a lane per piece), fills the fibres' entries from
// the segments found, and ends with the pass's epilogue (u, or z with the dual
// update and the restart test's sums). Each array of the pass is read from HBM
// once and written once.
//
// What bounds a pass is the scan: a chain of dependent steps, two to three
// per entry. A lane per fibre leaves 1400 chains of 3000 steps for one 1400^2
// image and lets a block of 512^2 images fill a quarter of each warp; pieces
// make the chains P times shorter and fill the warps. Measured, ms a solve, a
// lane per fibre over fibre-major copies in global memory (three kernels a
// pass), then this: 64 x 512^2 with edge weights 284, 173; 1400^2 67.8, 14.4;
// 90^2 3.24, 2.16. With pieces of 64 entries (P = 8) a warp takes 37 trips of 8
// steps for 4 fibres of 512 entries and 1200 steps each; an SM holds 10 warps
// by shared memory (40 weighted fibres) and issues 0.37 instructions per
// scheduler and cycle, so latency and occupancy bound it, not HBM (36 B per
// pixel and iteration, 92 of about 870 us).
// The segments' values go to global scratch (segv, at their last entry) and
// their ends to a byte per entry in shared memory, so that a fibre takes 5
// bytes per entry there (9 with weights) and an SM holds many.

constexpr int kFibList = 6;      // segments a lane may hold beyond its piece before it scans them twice
constexpr int kFibThreads = 256; // most threads of a block
template <class T>
constexpr int kFibVec = 16 / (int)sizeof(T);

struct FibCfg {
    int nf;     // fibres per block
    int P;      // pieces (lanes) per fibre, a power of two up to 32
    int len;    // entries per piece (odd, so that a fibre's pieces start in different banks)
    int pitch;  // entries between fibres in shared memory (odd)
};

// Shared memory of a block: 1/m, the fibres (y, or (y, r) pairs), a lane's
// list (values, ends), the end marks. (The scan's trips read a few entries past
// a fibre's last and 1/m past m = L: the next array's, unused.)
template <class T>
__host__ __device__ __forceinline__ size_t fib_smem(const FibCfg &c, int L, bool w) {
    const size_t nt = (size_t)c.nf * c.P;
    size_t b = sizeof(T) * ((size_t)(w ? 2 : 1) * c.nf * c.pitch + nt * kFibList + (size_t)(L + 1));
    b += sizeof(int) * nt * kFibList;
    return b + (size_t)c.nf * ((c.pitch + 3) / 4 * 4);
}

// The scalars of an ADBPG iteration after its second pass (tv_aniso.cpp:357-367, 461-480).
__device__ __forceinline__ void adbpg_advance(AnState s2, const AnCall &c, bool test, double dot, AnState *out) {
    s2.since += 1;
    double t = s2.tn;
    if (test && dot > 0.0 && s2.since >= s2.last) {
        s2.last = s2.since;
        s2.since = 0;
        s2.restart = 1;
        t = 1.0;
    } else {
        s2.restart = 0;
    }
    s2.it += 1;
    const double tn = fista_t(t);
    s2.beta = (t - 1.0) / tn;
    s2.tn = tn;
    if (s2.it == s2.chk_next || s2.it == c.max_iter) s2.stage = kStCheck;
    *out = s2;
}

// Whether pass PASS of a round acts on image b (the stages of an_pass1 / an_pass2).
template <int PASS>
__device__ __forceinline__ bool fib_active(const AnState &st, const AnImage &im) {
    if (st.status != kLive || im.mode != kAnAdbpg) return false;
    return PASS == 1 ? (st.stage == kStIter || st.stage == kStWarm) : st.stage == kStIter;
}

// A segment's end and value at its last entry.
template <class T>
struct MarkSink {
    T *val;
    unsigned char *mark;
    __device__ __forceinline__ void segment(int, int k1, double v) const {
        val[k1] = (T)v;
        mark[k1] = kMarkFinal;
    }
    __device__ __forceinline__ void finish(int) const {}
};

// V: fibres of a strided axis per load (16 bytes where the rows allow, else 1).
template <class T, int PASS, bool WT, int V>
__global__ void __launch_bounds__(kFibThreads, sizeof(T) == 4 ? 4 : 2)
an_fib_pass(AnGeom g, AnCall c, AnBuffers bf, FibCfg fc) {
    extern __shared__ __align__(16) unsigned char an_fib_smem[];
    __shared__ double sh[32];
    __shared__ int flag;
    constexpr int E = WT ? 2 : 1;
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    const AnImage &im = bf.img[b];
    if (!fib_active<PASS>(st, im)) return;
    const int a = PASS == 1 ? im.a1 : im.a2;
    const Fib fb = fibers(g, a);
    const int n = (int)fb.L, nt = blockDim.x, tid = threadIdx.x, lane = tid & 31;
    const int64_t N = g.N, f0 = (int64_t)blockIdx.x * fc.nf;
    const int s = (int)fb.s;  // N < 2^31
    const int nfb = (int)(fb.nfib - f0 < fc.nf ? fb.nfib - f0 : fc.nf);
    T *yr = reinterpret_cast<T *>(an_fib_smem);
    T *lv = yr + (size_t)E * fc.nf * fc.pitch;
    T *rc = lv + (size_t)nt * kFibList;
    int *le = reinterpret_cast<int *>(rc + n + 1);
    unsigned char *marks = reinterpret_cast<unsigned char *>(le + nt * kFibList);
    const int mpitch = (fc.pitch + 3) / 4 * 4;
    {
        const DivRecip<T> div;
        for (int m = tid; m <= n; m += nt) rc[m] = m ? div(m) : T(0);
        int *mw = reinterpret_cast<int *>(marks);
        for (int i = tid; i < fc.nf * mpitch / 4; i += nt) mw[i] = 0;
    }
    const T *Bw = WT ? static_cast<const T *>(bf.beta) + (int64_t)a * N : nullptr;
    const T lam = (T)im.lam[a];
    // staging: y of the block's fibres and their radii (entry n - 1: 0)
    const int ng = fc.nf / V, tx = tid % ng, ty = tid / ng, rows = nt / ng;
    const int64_t ob = tx * V < nfb ? fb.base(f0 + tx * V) : 0;
    {
        const T *P0 = static_cast<const T *>(PASS == 1 ? bf.d : bf.u) + (int64_t)b * N;
        // after a restart the extrapolated dual is y itself (tv_aniso.cpp:474-477)
        const T *Wv = static_cast<const T *>(st.restart ? bf.y : bf.wv) + (int64_t)b * g.k * N;
        auto put = [&](T *q, int i, T p0, T w, T bw) {
            q[i * E] = PASS == 1 ? p0 + w : p0 - w;
            if (WT) q[i * E + 1] = i < n - 1 ? lam * bw : T(0);
        };
        if (s == 1) {
            for (int f = tid >> 5; f < nfb; f += nt >> 5) {
                const int64_t o = (f0 + f) * n;
                const T *p0 = P0 + o, *wv = Wv + o, *bw = WT ? Bw + o : nullptr;
                T *q = yr + (size_t)f * fc.pitch * E;
#pragma unroll 8
                for (int i = lane; i < n; i += 32) put(q, i, p0[i], wv[i], WT ? bw[i] : T(0));
            }
        } else if (tx * V < nfb) {
            const T *p0 = P0 + ob, *wv = Wv + ob, *bw = WT ? Bw + ob : nullptr;
            T *q = yr + (size_t)tx * V * fc.pitch * E;
#pragma unroll 4
            for (int i = ty; i < n; i += rows) {
                T p[V], w[V], r[V];
                load_pack<T, V>(p0 + i * s, p);
                load_pack<T, V>(wv + i * s, w);
                if (WT) load_pack<T, V>(bw + i * s, r);
#pragma unroll
                for (int j = 0; j < V; ++j) put(q + j * fc.pitch * E, i, p[j], w[j], WT ? r[j] : T(0));
            }
        }
    }
    __syncthreads();
    // the scan: lane `sub` of a fibre's P lanes takes piece sub
    const int fib = tid / fc.P, sub = tid & (fc.P - 1);
    const bool act = fib < nfb;
    T *q = yr + (size_t)fib * fc.pitch * E;
    unsigned char *mark = marks + fib * mpitch;
    T *val = static_cast<T *>(bf.segv) + (int64_t)b * N + (act ? (f0 + fib) * n : 0);
    const int c0 = sub * fc.len < n ? sub * fc.len : n, c1 = c0 + fc.len < n ? c0 + fc.len : n;
    bool live = false, zero = false;
    T l = lam;
    // whether edge e has zero weight (not merely a radius that underflowed)
    const T *bw = WT && act ? Bw + fb.base(f0 + fib) : nullptr;
    auto cut = [&](int e) { return WT && q[e * E + 1] == T(0) && bw[e * s] == T(0); };
    {
        // the fibre's range, its largest radius and whether an edge has zero weight (fiber_range)
        T lo = Num<T>::inf(), hi = -Num<T>::inf(), rmax = T(0);
        if (act) {
#pragma unroll 4
            for (int i = c0; i < c1; ++i) {
                T v, r = T(0);
                if (WT) {
                    const Pair<T> yp = reinterpret_cast<const Pair<T> *>(q)[i];
                    v = yp.y;
                    r = yp.r;
                } else {
                    v = q[i];
                }
                lo = v < lo ? v : lo;
                hi = v > hi ? v : hi;
                if (WT) {
                    zero = zero || (r == T(0) && i < n - 1);
                    rmax = r > rmax ? r : rmax;
                }
            }
        }
        for (int o = fc.P >> 1; o > 0; o >>= 1) {
            const T lo2 = __shfl_xor_sync(0xffffffffu, lo, o), hi2 = __shfl_xor_sync(0xffffffffu, hi, o);
            lo = lo2 < lo ? lo2 : lo;
            hi = hi2 > hi ? hi2 : hi;
            if (WT) {
                const T r2 = __shfl_xor_sync(0xffffffffu, rmax, o);
                rmax = r2 > rmax ? r2 : rmax;
                zero = __shfl_xor_sync(0xffffffffu, (int)zero, o) || zero;
            }
        }
        if (WT && __any_sync(0xffffffffu, zero)) {  // some radius is zero: by its weight?
            bool z = false;
            if (zero)
                for (int i = c0; i < c1 && i < n - 1; ++i) z = z || cut(i);
            zero = z;
            for (int o = fc.P >> 1; o > 0; o >>= 1) zero = __shfl_xor_sync(0xffffffffu, (int)zero, o) || zero;
        }
        const T range = hi - lo;
        if (act) {
            if (n == 1 || lam == T(0) || range == T(0)) {  // the fibre is its own prox
                for (int i = c0; i < c1; ++i) {
                    val[i] = q[i * E];
                    mark[i] = kMarkFinal;
                }
            } else if (!WT && lam >= (T)(n / 2) * range) {  // no edge can be active: the mean
                if (sub == 0) fiber_mean([&](int i) { return q[i * E]; }, MarkSink<T>{val, mark}, n);
            } else if (WT && zero && rmax > T(2) * range) {
                // radii clamped between the cuts: each part between two cuts by the lane in whose piece it begins
                for (int i = c0; i < c1; ++i) {
                    if (i > 0 && !cut(i - 1)) continue;
                    int e = i;
                    while (e < n - 1 && !cut(e)) ++e;
                    const int m = e - i + 1;
                    auto rad = [&](int j) -> T {
                        if (j >= m - 1) return T(0);
                        const T r = q[(i + j) * E + 1];
                        const int jj = j + 1 < m - 1 - j ? j + 1 : m - 1 - j;
                        const T cap = T(2) * (T)(jj > 0 ? jj : 1) * range;
                        return r < cap ? r : cap;
                    };
                    const MarkSink<T> out{val, mark};
                    condat_piece<T>([&](int j) { return q[(i + j) * E]; }, ShiftedSink<MarkSink<T>>{out, i}, m, rad,
                                    TableRecip<T>{rc});
                }
            } else {
                live = true;
                if (!WT) {
                    const T cap = T(2) * (T)((n / 2) > 0 ? (n / 2) : 1) * range;
                    l = lam < cap ? lam : cap;
                } else if (rmax > T(2) * range) {  // radii clamped as in tv1d_fiber_sink (below 2 range none is)
                    for (int i = c0; i < c1; ++i) {
                        const T r = q[i * E + 1];
                        const int jj = i + 1 < n - 1 - i ? i + 1 : n - 1 - i;
                        const T cap = T(2) * (T)(jj > 0 ? jj : 1) * range;
                        q[i * E + 1] = r < cap ? r : cap;
                    }
                }
            }
        }
    }
    __syncwarp();
    // Warps with cut fibres on a path of their own: looking for the next cut costs
    // the others nothing. One lane scanning a cut fibre, part after part, took 420 ms
    // on 64 x 512^2 with one cut near each border and 817 with 1 % of the edges cut;
    // the pieces take 151 and 174 (128 without cuts; 93 and 24 on one 1400^2 image).
    auto scan = [&](auto cuts) {
        tv1d_pieces<T, WT, decltype(cuts)::value>(q, rc, l, n, fc.P, fc.len, sub, live, mark, val, le + tid * kFibList,
                                                  lv + tid * kFibList, kFibList, cut, bf.err);
    };
    if constexpr (WT) {
        if (__any_sync(0xffffffffu, live && zero)) scan(std::true_type{});
        else scan(std::false_type{});
    } else {
        scan(std::false_type{});
    }
    __syncwarp();
    // fill: a warp takes its fibres in turn, from their ends; entry i's value
    // is that of the first valid segment end at or after it
    {
        const int per = 32 / fc.P, wf = (tid >> 5) * per;
        T *U = static_cast<T *>(bf.u) + (int64_t)b * N;
        for (int f = wf; f < wf + per && f < nfb; ++f) {
            const unsigned char *mk = marks + f * mpitch;
            const T *vl = static_cast<const T *>(bf.segv) + (int64_t)b * N + (f0 + f) * n;
            T *z = yr + (size_t)f * fc.pitch * E;
            int carry = -1;
            constexpr int kC = 4;  // chunks of 32 entries whose values are read together
            for (int cb = (n - 1) >> 5; cb >= 0; cb -= kC) {
                int idx[kC];
#pragma unroll
                for (int u = 0; u < kC; ++u) {
                    const int i = (cb - u) * 32 + lane;
                    const bool in = cb - u >= 0 && i < n;
                    const unsigned w = __ballot_sync(0xffffffffu, in && mk[i] != 0);
                    const unsigned up = w >> lane;
                    idx[u] = in ? (up ? i + __ffs(up) - 1 : carry) : -1;
                    carry = w ? (cb - u) * 32 + __ffs(w) - 1 : carry;
                }
                T v[kC];
#pragma unroll
                for (int u = 0; u < kC; ++u) v[u] = idx[u] >= 0 ? vl[idx[u]] : T(0);
#pragma unroll
                for (int u = 0; u < kC; ++u) {
                    const int i = (cb - u) * 32 + lane;
                    if (cb - u < 0 || i >= n) continue;
                    if (idx[u] < 0) atomicExch(bf.err, 4);  // no end after i: a broken scan
                    if (PASS == 1 && s == 1) U[(f0 + f) * n + i] = v[u];
                    else z[i * E] = v[u];
                }
            }
        }
        if (PASS == 1 && s == 1) return;
    }
    __syncthreads();
    // epilogue
    const bool test = st.it % kCheck == 0;
    double up = 0.0;
    if (tx * V < nfb) {
        const T beta = (T)st.beta;
        T *U = static_cast<T *>(bf.u) + (int64_t)b * N + ob;
        T *Wv = static_cast<T *>(bf.wv) + (int64_t)b * g.k * N + ob;
        T *Yd = static_cast<T *>(bf.y) + (int64_t)b * g.k * N + ob;
        T *Z = static_cast<T *>(bf.z) + (int64_t)b * N + ob;
        const T *Ws = st.restart ? Yd : Wv;
        const T *zs = yr + (size_t)tx * V * fc.pitch * E;
        constexpr int kU = V > 1 ? 2 : 4;  // rows whose loads are in flight together
        for (int i = ty; i < n; i += kU * rows) {
            T u4[kU][V], w4[kU][V], y4[kU][V];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int o = (i + u * rows < n ? i + u * rows : i) * s;
                if (PASS == 2) {
                    load_pack<T, V>(U + o, u4[u]);
                    load_pack<T, V>(Ws + o, w4[u]);
                    load_pack<T, V>(Yd + o, y4[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int ii = i + u * rows;
                if (ii >= n) break;
                T z[V];
#pragma unroll
                for (int j = 0; j < V; ++j) z[j] = zs[(j * fc.pitch + ii) * E];
                if (PASS == 1) {
                    store_pack<T, V>(U + ii * s, z);
                } else {
#pragma unroll
                    for (int j = 0; j < V; ++j) {
                        const T w = w4[u][j], y = y4[u][j];
                        const T v = u4[u][j] - w;
                        const T yn = z[j] - v;
                        if (test) up += (double)((w - yn) * (yn - y));
                        w4[u][j] = yn + beta * (yn - y);
                        y4[u][j] = yn;
                    }
                    store_pack<T, V>(Wv + ii * s, w4[u]);
                    store_pack<T, V>(Yd + ii * s, y4[u]);
                    store_pack<T, V>(Z + ii * s, z);
                }
            }
        }
    }
    if (PASS == 1) return;
    double dot, unused;
    if (!reduce2(bf, b, blockIdx.x, gridDim.x, test ? up : 0.0, 0.0, sh, &flag, dot, unused)) return;
    adbpg_advance(bf.st[b], c, test, dot, bf.st + b);
}

// ---------------------------------------------------------------------------
// Warm starts (tv_aniso.cpp:316-320, 436-486, 539-543, 630-684)
// ---------------------------------------------------------------------------

// feasible_dual along axis a, one thread per fibre: q_a at the solved scale
// (zero on an inactive axis); a fibre whose running sums -p_e stay within
// their bounds and end at 0 up to rounding is kept, any other rebuilt from
// its running sums clipped to [-lam_e, lam_e] (non-finite ones 0).
template <class T>
__global__ void __launch_bounds__(128) an_warm_feasible(AnGeom g, AnCall c, AnBuffers bf, int a) {
    const int b = blockIdx.y;
    const AnImage &im = bf.img[b];
    if (bf.st[b].status != kLive || (im.mode != kAnAdbpg && im.mode != kAnFdpg3)) return;
    const Fib fb = fibers(g, a);
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= fb.nfib) return;
    const int64_t N = g.N, B = g.B, base = fb.base(f), s = fb.s, L = fb.L;
    T *Q = static_cast<T *>(bf.dual) + ((int64_t)a * B + b) * N + base;
    const double lam = im.lam[a];
    const T *bw = c.has_beta ? static_cast<const T *>(bf.beta) + (int64_t)a * c.N + base : nullptr;
    if (!(lam > 0.0)) {
        for (int64_t l = 0; l < L; ++l) Q[l * s] = T(0);
        return;
    }
    double acc = 0.0, mass = 0.0, peak = -lam;
    for (int64_t l = 0; l < L; ++l) {
        const double q = im.e ? ldexp((double)Q[l * s], -im.e) : (double)Q[l * s];
        Q[l * s] = (T)q;
        acc += q;
        mass += fabs(q);
        const double e = l + 1 < L ? fabs(acc) - (bw ? lam * (double)bw[l * s] : lam) : -lam;
        peak = (e > peak || e != e) ? e : peak;
    }
    const double eps = sizeof(T) == 4 ? 1.1920928955078125e-07 : DBL_EPSILON;
    const double tol = 1e-10 * lam + 16.0 * eps * mass;
    if (isfinite(mass) && peak <= tol && fabs(acc) <= tol) return;
    double run = 0.0, prev = 0.0;
    for (int64_t l = 0; l < L; ++l) {
        const double qi = (double)Q[l * s];
        run += qi;
        double pe = 0.0;
        const double lb = (l + 1 < L && bw) ? lam * (double)bw[l * s] : lam;
        if (l + 1 < L && isfinite(run)) pe = fmin(fmax(-run, -lb), lb);
        Q[l * s] = (T)(prev - pe);
        prev = pe;
    }
}

// y = -q2 and z = d - q1 - q2 (ADBPG), y_a = -q_a (FDPG-3); w = y
template <class T>
__global__ void an_warm_init(AnGeom g, AnBuffers bf) {
    const int b = blockIdx.y;
    const AnImage &im = bf.img[b];
    if (bf.st[b].status != kLive || (im.mode != kAnAdbpg && im.mode != kAnFdpg3)) return;
    const int64_t N = g.N, B = g.B;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N;
    const T *Q = static_cast<const T *>(bf.dual);
    T *Y = static_cast<T *>(bf.y) + (int64_t)b * g.k * N;
    T *Wv = static_cast<T *>(bf.wv) + (int64_t)b * g.k * N;
    T *Z = static_cast<T *>(bf.z) + (int64_t)b * N;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x) {
        if (im.mode == kAnAdbpg) {
            const T q1 = Q[((int64_t)im.a1 * B + b) * N + p], q2 = Q[((int64_t)im.a2 * B + b) * N + p];
            Y[p] = -q2;
            Wv[p] = -q2;
            Z[p] = D[p] - q1 - q2;
        } else {
            for (int a = 0; a < 3; ++a) {
                const T q = Q[((int64_t)a * B + b) * N + p];
                Y[(int64_t)a * N + p] = -q;
                Wv[(int64_t)a * N + p] = -q;
            }
        }
    }
}

// the first check at iteration 0
__global__ void an_warm_state(AnGeom g, AnBuffers bf) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= g.B) return;
    AnState &st = bf.st[b];
    const int mode = bf.img[b].mode;
    if (st.status != kLive || (mode != kAnAdbpg && mode != kAnFdpg3)) return;
    st.warm = 1;
    st.stage = kStCheck;
    st.wphase = mode == kAnAdbpg ? 1 : 0;
}

// The warm pass's dual (tv_aniso.cpp:443-449): q1 = d + y - u, q2 = -y and
// z = d - q1 - q2, for the second check.
template <class T>
__global__ void an_warm_z(AnGeom g, AnBuffers bf) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || st.stage != kStWarm) return;
    const int64_t N = g.N;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N;
    const T *Y = static_cast<const T *>(bf.y) + (int64_t)b * g.k * N;
    const T *U = static_cast<const T *>(bf.u) + (int64_t)b * N;
    T *Z = static_cast<T *>(bf.z) + (int64_t)b * N;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x) {
        const T q1 = D[p] + Y[p] - U[p], q2 = -Y[p];
        Z[p] = D[p] - q1 - q2;
    }
}

__global__ void an_warm_next(AnGeom g, AnBuffers bf) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= g.B) return;
    AnState &st = bf.st[b];
    if (st.status == kLive && st.stage == kStWarm) st.stage = kStCheck;
}

// After a restart the extrapolated dual restarts from y (tv_aniso.cpp:474-477).
template <class T>
__global__ void an_restart_copy(AnGeom g, AnBuffers bf) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || !st.restart) return;
    const int64_t n = (int64_t)g.k * g.N;
    const T *Y = static_cast<const T *>(bf.y) + (int64_t)b * n;
    T *Wv = static_cast<T *>(bf.wv) + (int64_t)b * n;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        Wv[i] = Y[i];
}

// FDPG-3 (tv_aniso.cpp:534-616): u = d + w0 + w1 + w2, then for each axis a
// y_a+ = (prox_{3 g_a}(u - 3 w_a) - (u - 3 w_a)) / 3 and the extrapolation.
template <class T>
__global__ void an_fdpg3_u(AnGeom g, AnBuffers bf) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || st.stage != kStIter || bf.img[b].mode != kAnFdpg3) return;
    const int64_t N = g.N;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N;
    const T *Wv = static_cast<const T *>(bf.wv) + (int64_t)b * 3 * N;
    T *U = static_cast<T *>(bf.u) + (int64_t)b * N;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
        U[i] = D[i] + Wv[i] + Wv[N + i] + Wv[2 * N + i];
}

template <class T>
__global__ void __launch_bounds__(128) an_fdpg3_pass(AnGeom g, AnCall c, AnBuffers bf) {
    __shared__ double sh[32];
    __shared__ int flag;
    const int b = round_image(bf, blockIdx.z);
    if (b < 0) return;
    const AnState st = bf.st[b];
    if (st.status != kLive || st.stage != kStIter) return;
    const AnImage &im = bf.img[b];
    if (im.mode != kAnFdpg3) return;
    const int64_t N = g.N;
    const bool test = st.it % kCheck == 0;
    const T beta = (T)st.beta;
    double up = 0.0;
    // blockIdx.y = axis; the fibres of all three axes in one launch
    const int a = blockIdx.y;
    const Fib fb = fibers(g, a);
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f < fb.nfib) {
        const int64_t base = fb.base(f), s = fb.s;
        const T *U = static_cast<const T *>(bf.u) + (int64_t)b * N + base;
        T *Wa = static_cast<T *>(bf.wv) + ((int64_t)b * 3 + a) * N + base;
        T *Ya = static_cast<T *>(bf.y) + ((int64_t)b * 3 + a) * N + base;
        T *Zs = static_cast<T *>(bf.zp) + (int64_t)b * N;  // scratch: z of this axis' fibres
        T *Za = Zs + base;
        // the three axes write disjoint scratch: zp (a = 0), z (a = 1), dual slot (a = 2)
        if (a == 1) Za = static_cast<T *>(bf.z) + (int64_t)b * N + base;
        if (a == 2) Za = static_cast<T *>(bf.scratch) + (int64_t)b * N + base;
        auto in = [U, Wa, s](int64_t i) -> double { return (double)(U[i * s] - T(3) * Wa[i * s]); };
        auto out = [Za, s](int64_t i, double v) { Za[i * s] = (T)v; };
        fibre_prox<T>(c, bf, a, base, fb, 3.0 * im.lam[a], in, out);
        for (int64_t i = 0; i < fb.L; ++i) {
            const int64_t o = i * s;
            const T v = U[o] - T(3) * Wa[o];
            const T yn = (Za[o] - v) / T(3);
            const T y = Ya[o], w = Wa[o];
            if (test) up += (double)((w - yn) * (yn - y));
            Wa[o] = yn + beta * (yn - y);
            Ya[o] = yn;
        }
    }
    double dot, unused;
    const unsigned nblk = gridDim.x * gridDim.y;
    const unsigned blk = blockIdx.y * gridDim.x + blockIdx.x;
    if (!reduce2(bf, b, blk, nblk, test ? up : 0.0, 0.0, sh, &flag, dot, unused)) return;
    AnState s2 = st;
    s2.since += 1;
    double t = s2.tn;
    if (test && dot > 0.0 && s2.since >= s2.last) {
        s2.last = s2.since;
        s2.since = 0;
        s2.restart = 1;
        t = 1.0;
    } else {
        s2.restart = 0;
    }
    s2.it += 1;
    const double tn = fista_t(t);
    s2.beta = (t - 1.0) / tn;
    s2.tn = tn;
    if (s2.it % kCheck == 0 || s2.it == c.max_iter) s2.stage = kStCheck;
    bf.st[b] = s2;
}

// FDPG-3's primal at a check: z = prox_{g_c}(d + y_0 + y_1) along the
// contiguous axis c = 2 (tv_aniso.cpp:118-123).
template <class T>
__global__ void __launch_bounds__(128) an_fdpg3_primal(AnGeom g, AnCall c, AnBuffers bf, int stage) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || st.stage != stage) return;
    const AnImage &im = bf.img[b];
    if (im.mode != kAnFdpg3) return;
    const Fib fb = fibers(g, 2);
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= fb.nfib) return;
    const int64_t N = g.N, base = fb.base(f), s = fb.s;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N + base;
    const T *Y0 = static_cast<const T *>(bf.y) + (int64_t)b * 3 * N + base;
    const T *Y1 = Y0 + N;
    T *Z = static_cast<T *>(bf.z) + (int64_t)b * N + base;
    auto in = [D, Y0, Y1, s](int64_t i) -> double { return (double)(D[i * s] + Y0[i * s] + Y1[i * s]); };
    auto out = [Z, s](int64_t i, double v) { Z[i * s] = (T)v; };
    fibre_prox<T>(c, bf, 2, base, fb, im.lam[2], in, out);
}

// ---------------------------------------------------------------------------
// The gap of a point: sum_a lam_e |z_j - z_i| - <z, d - z> (tv_aniso.cpp:192-226)
// ---------------------------------------------------------------------------

template <class T>
__device__ __forceinline__ double tv_at(const AnGeom &g, const AnCall &c, const AnBuffers &bf, const AnImage &im,
                                        const T *Z, int p, double z) {
    double s = 0.0;
    int co[3];
    coords(g, p, co);
    for (int a = 0; a < g.k; ++a) {
        const double l = im.lam[a];
        if (l == 0.0) continue;
        if (co[a] + 1 >= g.L[a]) continue;
        double le = l;
        if (c.has_beta) le = l * (double)static_cast<const T *>(bf.beta)[(int64_t)a * g.N + p];
        s += le * fabs((double)Z[p + g.S[a]] - z);
    }
    return s;
}

// The stage after a check (and its polish, if any) that left the image
// unconverged. In the loop: CheckSchedule::done for ADBPG, then iterate (or
// finish at max_iter). A warm start's first check is followed by its pass
// (ADBPG) and second check, which take no part in the schedule
// (tv_aniso.cpp:473-486).
__device__ __forceinline__ void after_check(AnState &s2, const AnImage &im, bool last) {
    if (s2.wphase == 1 && im.mode == kAnAdbpg) {
        s2.wphase = 2;
        s2.stage = kStWarm;
        return;
    }
    if (s2.wphase != 0) {
        s2.wphase = 0;
    } else if (im.mode == kAnAdbpg) {
        check_done(s2, s2.gp, im.target);
    }
    s2.stage = last ? kStFinal : kStIter;
}

// stage kStCheck: the gap of z; kStFinal: the gap of zp (the final rebuild).
template <class T>
__global__ void __launch_bounds__(kThreads) an_gap(AnGeom g, AnCall c, AnBuffers bf, int stage) {
    __shared__ double sh[32];
    __shared__ int flag;
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState st = bf.st[b];
    if (st.status != kLive || st.stage != stage) return;
    if (stage == kStFinal && (st.polished || st.it == 0 || bf.img[b].mode != kAnAdbpg)) return;
    const AnImage im = bf.img[b];
    const int64_t N = g.N;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N;
    const T *Z = static_cast<const T *>(stage == kStCheck ? bf.z : bf.zp) + (int64_t)b * N;
    auto term = [&](int p) {
        const double z = (double)Z[p];
        return tv_at<T>(g, c, bf, im, Z, p, z) - z * ((double)D[p] - z);
    };
    double gz;
    if (!reduce_chunks(bf, b, N, pixel_chunks(N), term, sh, &flag, gz)) return;
    AnState s2 = st;
    if (stage == kStFinal) {
        // d - q1 - q2 in place of the iterate, unless rounding alone takes its
        // gap over the target (tv_aniso.cpp:87-96)
        if (gz <= im.target || !(s2.gp <= im.target)) {
            s2.zsel = 1;
            s2.gp = gz;
        }
        s2.stage = kStDone;
        bf.st[b] = s2;
        return;
    }
    const bool last = s2.it == c.max_iter;
    s2.gz = gz;
    if (gz <= im.target) {
        s2.gp = gz;
        s2.stage = kStFinal;
    } else if (last ? !s2.polished
                    : (im.mode == kAnAdbpg ? ((s2.warm || s2.it >= kCheck) && gz <= s2.pol_next) : gz <= s2.pol_next)) {
        s2.accept = last ? gz : im.target;
        s2.stage = kStPolish;
    } else {
        s2.gp = gz;
        after_check(s2, im, last);
    }
    bf.st[b] = s2;
}

// ---------------------------------------------------------------------------
// The polish (tv_aniso.cpp:630-953)
// ---------------------------------------------------------------------------

// dual(z) (tv_aniso.cpp:443-449, 124-131) into the dual, and the polish's
// scratch reset: zp = d, flags 0, parent = self, sums 0.
// stage kStPolish: for a polish; kStFinal: the final rebuild zp = d - q1 - q2.
template <class T>
__global__ void an_dual(AnGeom g, AnBuffers bf, int stage) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || st.stage != stage) return;
    if (stage == kStFinal && (st.polished || st.it == 0)) return;
    const AnImage &im = bf.img[b];
    const int64_t N = g.N, B = g.B;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N;
    const T *Z = static_cast<const T *>(bf.z) + (int64_t)b * N;
    const T *Y = static_cast<const T *>(bf.y) + (int64_t)b * g.k * N;
    T *Q = static_cast<T *>(bf.dual);
    T *ZP = static_cast<T *>(bf.zp) + (int64_t)b * N;
    uint8_t *F = bf.flag + (int64_t)b * N;
    int *P = bf.parent + (int64_t)b * N;
    unsigned long long *S = bf.sum + (int64_t)b * N;
    int *C = bf.cnt + (int64_t)b * N;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x) {
        T q[3] = {T(0), T(0), T(0)};
        if (im.mode == kAnAdbpg) {
            q[im.a1] = D[p] + Y[p] - Z[p];
            q[im.a2] = -Y[p];
        } else {
            q[0] = -Y[p];
            q[1] = -Y[N + p];
            q[2] = D[p] + Y[p] + Y[N + p] - Z[p];
        }
        for (int a = 0; a < g.k; ++a) Q[((int64_t)a * B + b) * N + p] = q[a];
        if (stage == kStFinal) {
            if (im.mode == kAnAdbpg) {
                T s = T(0);
                for (int a = 0; a < g.k; ++a) s += q[a];
                ZP[p] = D[p] - s;
            }
        } else {
            ZP[p] = D[p];
            F[p] = 0;
            P[p] = (int)p;
            S[p] = 0ull;
            C[p] = 0;
        }
    }
}

// mark_edges (tv_aniso.cpp:256-297) along axis a: the 1D dual of each edge
// from the running sum of q_a along its fibre; an edge strictly inside its
// bound is flat (bit a), the others move lam_e sign(p_e) from j to i in zp.
// The running sums are formed by parts (a thread walking a whole fibre took
// 500 us on 64 x 512^2 and 600 on one 1400^2 image, all of it the wait for one
// load after another).
template <class T>
struct EdgeMark {
    const T *q, *bw;
    double lam;
    // Whether edge i (pe its dual) is flat, else ls = lam_e sign(p_e).
    __device__ __forceinline__ bool flat(int64_t o, double pe, double &ls) const {
        const double lb = bw ? lam * (double)bw[o] : lam;
        ls = copysign(lb, pe);
        return fabs(pe) < lb * (1.0 - polish_eta<T>());
    }
};
// zp of entry i from the edges before and after it, in that order.
template <class T>
__device__ __forceinline__ T moved(T z, bool before, double lsb, bool after, double lsa) {
    if (before) z = (T)((double)z - lsb);
    if (after) z = (T)((double)z + lsa);
    return z;
}

// A strided axis: kMarkCols fibres side by side (adjacent in memory), each cut
// into kMarkParts parts whose sums come first.
constexpr int kMarkCols = 32, kMarkParts = 16;

template <class T>
__global__ void __launch_bounds__(kMarkCols *kMarkParts) an_mark_cols(AnGeom g, AnCall c, AnBuffers bf, int a) {
    __shared__ double part[kMarkParts][kMarkCols];
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || st.stage != kStPolish) return;
    const double lam = bf.img[b].lam[a];
    if (lam == 0.0) return;
    const Fib fb = fibers(g, a);
    const int tx = threadIdx.x % kMarkCols, ty = threadIdx.x / kMarkCols;
    const int64_t N = g.N, s = fb.s;
    const int n = (int)fb.L, len = (n + kMarkParts - 1) / kMarkParts;
    const uint8_t bit = (uint8_t)(1u << a);
    for (int64_t f0 = (int64_t)blockIdx.x * kMarkCols; f0 < fb.nfib; f0 += (int64_t)gridDim.x * kMarkCols) {
        const int64_t f = f0 + tx;
        const bool act = f < fb.nfib;
        const int64_t base = act ? fb.base(f) : 0;
        const T *Q = static_cast<const T *>(bf.dual) + ((int64_t)a * g.B + b) * N + base;
        const EdgeMark<T> em{Q, c.has_beta ? static_cast<const T *>(bf.beta) + (int64_t)a * N + base : nullptr, lam};
        T *ZP = static_cast<T *>(bf.zp) + (int64_t)b * N + base;
        uint8_t *F = bf.flag + (int64_t)b * N + base;
        const int i0 = ty * len < n ? ty * len : n, i1 = i0 + len < n ? i0 + len : n;
        double acc = 0.0;
        if (act) {
#pragma unroll 8
            for (int i = i0; i < i1; ++i) acc += (double)Q[i * s];
        }
        part[ty][tx] = acc;
        __syncthreads();
        const double own = acc;
        acc = 0.0;
        for (int j = 0; j < ty; ++j) acc += part[j][tx];
        // the sum up to this part's last edge as the next part begins with it:
        // both sides must take the edge alike, and entry by entry it may round
        // to another double
        const double end = acc + own;
        __syncthreads();
        if (act && i0 < i1) {
            double lsb = 0.0;
            bool before = i0 > 0 && !em.flat((i0 - 1) * s, -acc, lsb);
#pragma unroll 4
            for (int i = i0; i < i1; ++i) {
                const int64_t o = i * s;
                const bool edge = i + 1 < n;
                acc += (double)Q[o];
                if (i + 1 == i1) acc = end;
                double ls;
                const bool flat = em.flat(o, -acc, ls);
                if (edge && flat) F[o] |= bit;
                const bool after = edge && !flat;
                ZP[o] = moved(ZP[o], before, lsb, after, ls);
                before = after;
                lsb = ls;
            }
        }
    }
}

// The contiguous axis: a warp per fibre, 32 entries at a time by a warp scan.
// It also starts the components (parent): within 32 entries, those joined by
// flat edges point to the first of them.
template <class T>
__global__ void __launch_bounds__(kThreads) an_mark_rows(AnGeom g, AnCall c, AnBuffers bf, int a) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || st.stage != kStPolish) return;
    const double lam = bf.img[b].lam[a];
    if (lam == 0.0) return;
    const int64_t N = g.N, nfib = N / g.L[a];
    const int n = (int)g.L[a], lane = threadIdx.x & 31;
    const uint8_t bit = (uint8_t)(1u << a);
    for (int64_t f = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); f < nfib;
         f += (int64_t)gridDim.x * (kThreads / 32)) {
        const int64_t base = f * n;
        const T *Q = static_cast<const T *>(bf.dual) + ((int64_t)a * g.B + b) * N + base;
        const EdgeMark<T> em{Q, c.has_beta ? static_cast<const T *>(bf.beta) + (int64_t)a * N + base : nullptr, lam};
        T *ZP = static_cast<T *>(bf.zp) + (int64_t)b * N + base;
        uint8_t *F = bf.flag + (int64_t)b * N + base;
        int *P = bf.parent + (int64_t)b * N + base;
        double carry = 0.0, lsc = 0.0;  // the sum and the last edge of the entries before
        bool beforec = false;
        for (int c0 = 0; c0 < n; c0 += 32) {
            const int i = c0 + lane;
            const bool in = i < n, edge = i + 1 < n;
            double x = in ? (double)Q[i] : 0.0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            x += carry;
            carry = __shfl_sync(0xffffffffu, x, 31);
            double ls = 0.0;
            const bool flat = edge && em.flat(i, -x, ls);
            const bool after = edge && !flat;
            double lsb = __shfl_up_sync(0xffffffffu, ls, 1);
            const unsigned am = __ballot_sync(0xffffffffu, after), fm = __ballot_sync(0xffffffffu, flat);
            bool before = lane > 0 && (am >> (lane - 1) & 1u);
            if (lane == 0) {
                before = beforec;
                lsb = lsc;
            }
            if (in) {
                if (flat) F[i] |= bit;
                ZP[i] = moved(ZP[i], before, lsb, after, ls);
                // the last entry at or before this one that no flat edge joins to the one before
                const unsigned heads = ~(fm << 1) & (0xffffffffu >> (31 - lane));
                P[i] = (int)(base + c0 + 31 - __clz(heads));
            }
            beforec = am >> 31 & 1u;
            lsc = __shfl_sync(0xffffffffu, ls, 31);
        }
    }
}

__device__ __forceinline__ int uf_find(int *P, int i) {
    // parents point to smaller indices, so the walk ends; path halving
    for (int n = 0; n < (1 << 30); ++n) {
        const int p = P[i];
        if (p == i) return i;
        const int q = P[p];
        if (q != p) P[i] = q;
        i = p;
    }
    return i;
}

// components (tv_aniso.cpp:324-439) by union-find: the flat edges join
// their ends, the larger root hooked under the smaller by compare-and-swap,
// so each root is the smallest index of its component. Along the contiguous
// axis an_mark_rows has joined every 32 entries already; a flat edge of another
// axis whose neighbour on the left is flat too, and joined to it at both ends,
// adds nothing. (The unions of every edge took 621 us on 64 x 512^2.)
__global__ void an_union(AnGeom g, AnBuffers bf) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || st.stage != kStPolish) return;
    const int64_t N = g.N;
    const uint8_t *F = bf.flag + (int64_t)b * N;
    int *P = bf.parent + (int64_t)b * N;
    const int last = g.k - 1;
    const unsigned row = 1u << last;  // the contiguous axis' bit
    const unsigned L = (unsigned)g.L[last];
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x) {
        const uint8_t fl = F[p];
        if (!fl) continue;
        const unsigned co = (unsigned)p % L;
        for (int a = 0; a < g.k; ++a) {
            if (!(fl & (1u << a))) continue;
            if (a == last) {
                if ((co & 31) != 31) continue;
            } else if (co > 0) {
                const unsigned fq = F[p - 1], fr = F[p - 1 + g.S[a]];
                if ((fq & row) && (fr & row) && (fq & (1u << a))) continue;
            }
            int x = (int)p, y = (int)(p + g.S[a]);
            int tries = 0;
            for (;;) {
                x = uf_find(P, x);
                y = uf_find(P, y);
                if (x == y) break;
                const int hi = x > y ? x : y, lo = x > y ? y : x;
                const int old = atomicCAS(P + hi, hi, lo);
                if (old == hi) break;
                x = old;  // hi was hooked meanwhile: retry from there
                y = lo;
                if (++tries > (1 << 24)) {
                    atomicExch(bf.err, 2);
                    break;
                }
            }
        }
    }
}

// The root of i by a walk that writes nothing (parents point to smaller
// indices, so it ends). After the unions, each thread stores its own
// entry's root only: a halving write here could put a stale, non-root
// ancestor over an entry whose root another thread has already stored.
__device__ __forceinline__ int uf_root(const int *P, int i) {
    for (int n = 0; n < (1 << 30); ++n) {
        const int p = P[i];
        if (p == i) return i;
        i = p;
    }
    return i;
}

// every entry to its root; the region sums of zp (64-bit fixed point) and
// sizes. A warp takes kRunSegs x 32 consecutive entries; while all 32 lie in
// the region of the last ones each lane adds its own, else the entries are
// added run by run (equal roots side by side), one atomic per run and sum: an
// atomic per entry took 2.5 ms on 64 x 512^2 and 1.3 ms on one 1400^2 image,
// nearly all of them on the few largest regions. The sums are integers, so
// their order does not matter.
constexpr int kRunSegs = 16;

template <class T>
__global__ void __launch_bounds__(kThreads) an_region_sum(AnGeom g, AnBuffers bf) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || st.stage != kStPolish) return;
    const int64_t N = g.N;
    const int sh = bf.img[b].fx_shift, lane = threadIdx.x & 31;
    int *P = bf.parent + (int64_t)b * N;
    const T *ZP = static_cast<const T *>(bf.zp) + (int64_t)b * N;
    unsigned long long *S = bf.sum + (int64_t)b * N;
    int *C = bf.cnt + (int64_t)b * N;
    const int64_t warps = (int64_t)gridDim.x * (kThreads / 32), w0 = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    for (int64_t w = w0; w * (kRunSegs * 32) < N; w += warps) {
        unsigned long long acc = 0;
        int root = -1, cnt = 0;  // the region the lanes are adding up (warp-uniform), 32 entries cnt times
        auto flush = [&]() {
            if (cnt == 0) return;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
            if (lane == 0) {
                atomicAdd(S + root, acc);
                atomicAdd(C + root, 32 * cnt);
            }
            acc = 0;
            cnt = 0;
        };
        for (int j = 0; j < kRunSegs; ++j) {
            const int64_t p = (w * kRunSegs + j) * 32 + lane;
            if (p - lane >= N) break;
            const bool in = p < N;
            int r = -1;
            unsigned long long fx = 0;
            if (in) {
                r = uf_root(P, (int)p);
                P[p] = r;
                fx = (unsigned long long)llrint(ldexp((double)ZP[p], sh));
            }
            const int r31 = __shfl_sync(0xffffffffu, r, 31);
            if (__all_sync(0xffffffffu, in && r == r31)) {
                if (r31 != root) flush();
                root = r31;
                acc += fx;
                ++cnt;
                continue;
            }
            // run sums from the inclusive scan, at each run's last lane
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, fx, o);
                if (lane >= o) fx += y;
            }
            const int rl = __shfl_up_sync(0xffffffffu, r, 1), rn = __shfl_down_sync(0xffffffffu, r, 1);
            const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || r != rl);
            const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
            const unsigned long long before = __shfl_sync(0xffffffffu, fx, first > 0 ? first - 1 : 0);
            if (in && (lane == 31 || r != rn)) {
                atomicAdd(S + r, fx - (first > 0 ? before : 0ull));
                atomicAdd(C + r, lane - first + 1);
            }
        }
        flush();
    }
}

// zp = the region means; the polished gap P(zp) - D(q) (tv_aniso.cpp:504-523);
// the last block accepts or schedules the next attempt (:520-523, :382-391).
template <class T>
__global__ void __launch_bounds__(kThreads) an_polish_gap(AnGeom g, AnCall c, AnBuffers bf) {
    __shared__ double sh[32];
    __shared__ int flag;
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState st = bf.st[b];
    if (st.status != kLive || st.stage != kStPolish) return;
    const AnImage im = bf.img[b];
    const int64_t N = g.N, B = g.B;
    const int shf = im.fx_shift;
    const int *P = bf.parent + (int64_t)b * N;
    const unsigned long long *S = bf.sum + (int64_t)b * N;
    const int *C = bf.cnt + (int64_t)b * N;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N;
    const T *Q = static_cast<const T *>(bf.dual);
    auto mean = [&](int r) -> double { return ldexp((double)(long long)S[r], -shf) / (double)C[r]; };
    auto term = [&](int p) {
        const int r = P[p];
        const double zp = mean(r);
        const double d = (double)D[p];
        const double e = zp - d;
        double sj = 0.0;
        for (int a = 0; a < g.k; ++a) sj += (double)Q[((int64_t)a * B + b) * N + p];
        double tv = 0.0;
        int co[3];
        coords(g, p, co);
        for (int a = 0; a < g.k; ++a) {
            const double l = im.lam[a];
            if (l == 0.0) continue;
            if (co[a] + 1 >= g.L[a]) continue;
            const int rn = P[p + g.S[a]];
            if (rn == r) continue;  // the same region: no jump
            double le = l;
            if (c.has_beta) le = l * (double)static_cast<const T *>(bf.beta)[(int64_t)a * N + p];
            tv += le * fabs(mean(rn) - zp);
        }
        return 0.5 * e * e - (d * sj - 0.5 * sj * sj) + tv;
    };
    // the means are written after every block of this image has read the sums
    // (an_polish_write); here only the gap
    double pz;
    if (!reduce_chunks(bf, b, N, pixel_chunks(N), term, sh, &flag, pz)) return;
    AnState s2 = st;
    const double gz = s2.gz;
    const bool last = s2.it == c.max_iter;
    if (pz <= s2.accept && pz <= kPolishRatio * gz) {
        s2.polished = 1;
        s2.zsel = 1;
        s2.gp = pz;
        s2.pol_accept = 1;
    } else {
        // PolishSchedule::done (tv_aniso.cpp:386-390)
        const bool eager = im.mode == kAnFdpg3;
        double next = gz * kPolishDrop;
        if (pz > 0.0 && pz < (eager ? 1.0 : kPolishRatio) * gz) next = fmax(next, im.target * gz / pz);
        s2.pol_next = next;
        s2.gp = gz;
        s2.pol_accept = 0;
    }
    if (s2.gp <= im.target) s2.stage = kStFinal;
    else after_check(s2, im, last);
    bf.st[b] = s2;
}

// the accepted candidate: zp = region means
template <class T>
__global__ void an_polish_write(AnGeom g, AnBuffers bf) {
    const int b = round_image(bf, blockIdx.y);
    if (b < 0) return;
    const AnState &st = bf.st[b];
    if (st.status != kLive || !st.pol_accept) return;
    const int64_t N = g.N;
    const int shf = bf.img[b].fx_shift;
    const int *P = bf.parent + (int64_t)b * N;
    const unsigned long long *S = bf.sum + (int64_t)b * N;
    const int *C = bf.cnt + (int64_t)b * N;
    T *ZP = static_cast<T *>(bf.zp) + (int64_t)b * N;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x) {
        const int r = P[p];
        ZP[p] = (T)(ldexp((double)(long long)S[r], -shf) / (double)C[r]);
    }
}

// images whose stage is done leave the live set (a final rebuild is not needed
// after a polish or at it = 0, nor by FDPG-3)
__global__ void an_retire(AnGeom g, AnBuffers bf) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= g.B) return;
    AnState &st = bf.st[b];
    st.pol_accept = 0;
    if (st.status == kLive &&
        (st.stage == kStDone ||
         (st.stage == kStFinal && (bf.img[b].mode == kAnFdpg3 || st.polished || st.it == 0)))) {
        st.status = st.gp <= bf.img[b].target ? kConverged : kNotConv;
        atomicSub(bf.live, 1);
    }
}

// ---------------------------------------------------------------------------
// Single active axis, identity, NaN; the output at the input's scale
// ---------------------------------------------------------------------------

template <class T>
__global__ void __launch_bounds__(128) an_single(AnGeom g, AnCall c, AnBuffers bf) {
    const int b = blockIdx.y;
    const AnImage &im = bf.img[b];
    if (im.mode != kAnSingle) return;
    int a = 0;
    for (int x = 0; x < g.k; ++x)
        if (im.lam[x] > 0.0) a = x;
    const Fib fb = fibers(g, a);
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= fb.nfib) return;
    const int64_t N = g.N, base = fb.base(f), s = fb.s;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N + base;
    T *Z = static_cast<T *>(bf.z) + (int64_t)b * N + base;
    auto in = [D, s](int64_t i) -> double { return (double)D[i * s]; };
    auto out = [Z, s](int64_t i, double v) { Z[i * s] = (T)v; };
    fibre_prox<T>(c, bf, a, base, fb, im.lam[a], in, out);
}

template <class T>
__global__ void an_output(AnGeom g, AnBuffers bf, T *__restrict__ out) {
    const int b = blockIdx.y;
    const AnImage im = bf.img[b];
    if (im.mode == kAnInf) return;
    const AnState st = bf.st[b];
    const int64_t N = g.N, B = g.B;
    const T *D = static_cast<const T *>(bf.d) + (int64_t)b * N;
    const T *Z = static_cast<const T *>(st.zsel ? bf.zp : bf.z) + (int64_t)b * N;
    T *Q = static_cast<T *>(bf.dual);
    T *O = out + (int64_t)b * N;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x) {
        if (im.mode == kAnNan) {
            O[p] = (T)CUDART_NAN;
            for (int a = 0; a < g.k; ++a) Q[((int64_t)a * B + b) * N + p] = (T)CUDART_NAN;
        } else if (im.mode == kAnIdentity) {
            O[p] = D[p];
            for (int a = 0; a < g.k; ++a) Q[((int64_t)a * B + b) * N + p] = T(0);
        } else if (im.mode == kAnSingle) {
            const T z = Z[p];
            O[p] = im.e ? ldexp_t(z, im.e) : z;
            for (int a = 0; a < g.k; ++a) {
                T q = im.lam[a] > 0.0 ? D[p] - z : T(0);  // q_a = v - z (tv_aniso.cpp:321-323)
                Q[((int64_t)a * B + b) * N + p] = im.e ? ldexp_t(q, im.e) : q;
            }
        } else {
            const T z = Z[p];
            O[p] = im.e ? ldexp_t(z, im.e) : z;
            if (im.e)
                for (int a = 0; a < g.k; ++a) {
                    T &q = Q[((int64_t)a * B + b) * N + p];
                    q = ldexp_t(q, im.e);
                }
        }
    }
}


template <class T>
cudaError_t setup_t(const AnGeom &g, const AnCall &c, const AnBuffers &bf, const void *x, cudaStream_t s) {
    const int nb = (int)std::min<int64_t>(128, std::max<int64_t>(1, (g.N + kThreads * 8 - 1) / (kThreads * 8)));
    const dim3 grid(nb, (unsigned)g.B);
    an_scan1<T><<<grid, kThreads, 0, s>>>(static_cast<const T *>(x), g, c, bf);
    an_scan2<T><<<grid, kThreads, 0, s>>>(g, c, bf);
    // single-axis images are solved here
    int64_t nfmax = 0;
    for (int a = 0; a < g.k; ++a) nfmax = std::max<int64_t>(nfmax, g.N / g.L[a]);
    an_single<T><<<dim3((unsigned)((nfmax + 127) / 128), (unsigned)g.B), 128, 0, s>>>(g, c, bf);
    return cudaGetLastError();
}

// Fibres per tile along each axis. A block scans its tile with one warp, so
// an SM scans as many fibres at once as the tiles of its resident blocks hold
// (shared memory, registers and threads bound how many blocks it holds): fb
// makes that number largest, up to 8 fibres (a warp's step takes longer the
// more lanes it carries, and more warps hide more of its latency: on 64 x
// 512^2 with edge weights 8 per block ran 3% faster than 16 and 8% faster than
// 26), among tiles of at most budget bytes (default
// kTileSmemMax) and while the launch still gives every SM a block; the larger
// fb on ties, so that fewer warps issue the same steps. fb is 1 or even (the
// tile's row length fb + 1 odd). 0 when one fibre does not fit: the untiled
// pass then runs.
constexpr int kTileSmemMax = 200 * 1024;
constexpr size_t kSmemPerSM = 228 * 1024;  // shared memory of an SM (sm_100)
constexpr size_t kSmemReserve = 1024 + 512;  // per block: the system's and the kernels' static arrays
constexpr int kSMs = 148;
constexpr int kFibSmem = 72 * 1024;  // most shared memory of a block while it can hold fewer fibres

// The tiled kernels may take up to kTileSmemMax of dynamic shared memory. Set
// once per kernel, before any launch: the attribute is per function, and
// threads launching with different sizes must not lower it under one another.
template <class T>
void tile_attributes() {
    static std::atomic<unsigned long long> done{0};  // one bit per device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
    const unsigned long long bit = 1ull << dev;
    if (done.load() & bit) return;
    cudaFuncSetAttribute(an_pass1_tile<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_pass2_tile<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_fdpg3_tile<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_fib_pass<T, 1, false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_fib_pass<T, 1, false, kFibVec<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_fib_pass<T, 1, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_fib_pass<T, 1, true, kFibVec<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_fib_pass<T, 2, false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_fib_pass<T, 2, false, kFibVec<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_fib_pass<T, 2, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    cudaFuncSetAttribute(an_fib_pass<T, 2, true, kFibVec<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax);
    done.fetch_or(bit);
}

// Blocks of the tiled kernels an SM holds by registers and threads (their
// largest register count, allocated per warp in units of 256).
template <class T>
int tile_blocks_by_regs() {
    static const int n = [] {
        int regs = 0;
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, an_pass1_tile<T>) == cudaSuccess) regs = std::max(regs, fa.numRegs);
        if (cudaFuncGetAttributes(&fa, an_pass2_tile<T>) == cudaSuccess) regs = std::max(regs, fa.numRegs);
        if (cudaFuncGetAttributes(&fa, an_fdpg3_tile<T>) == cudaSuccess) regs = std::max(regs, fa.numRegs);
        const int per_warp = ((std::max(regs, 1) * 32 + 255) / 256) * 256;
        const int warps = kTileThreads / 32;
        return std::max(1, std::min(2048 / kTileThreads, 65536 / (per_warp * warps)));
    }();
    return n;
}

template <class T>
TileCfg tile_cfg(const AnGeom &g, const AnCall &c, int64_t nimg, size_t &smem) {
    // tuning hints: FASTPROX_B200_TILE_FB caps fb, FASTPROX_B200_TILE_KB the
    // tile; FASTPROX_B200_TILES=0 runs the untiled passes (for comparison)
    static const bool off = [] {
        const char *v = std::getenv("FASTPROX_B200_TILES");
        return v && v[0] == '0' && v[1] == 0;
    }();
    static const int fb_max = [] {
        const char *v = std::getenv("FASTPROX_B200_TILE_FB");
        const int f = v ? std::atoi(v) : 0;
        return (f >= 1 && f <= 32) ? f : 8;
    }();
    static const size_t budget = [] {
        const char *v = std::getenv("FASTPROX_B200_TILE_KB");
        const int k = v ? std::atoi(v) : 0;
        return (size_t)((k >= 8 && k <= 200) ? k : 200) * 1024;
    }();
    const int by_regs = tile_blocks_by_regs<T>();
    TileCfg tc{{0, 0, 0}};
    smem = 0;
    const int nbuf = c.has_beta ? 2 : 1;
    for (int a = 0; a < g.k && !off; ++a) {
        const int L = (int)g.L[a];
        const int64_t fibres = nimg * (g.N / std::max<int64_t>(g.L[a], 1));
        int best = 0;
        double best_waves = 0.0;
        for (int fb = 1; fb <= fb_max; fb += (fb == 1 ? 1 : 2)) {
            const size_t by = tile_bytes(L, fb, nbuf, sizeof(T));
            if (by > budget || by > (size_t)kTileSmemMax) break;
            const int per_sm = std::min<int>(by_regs, (int)(kSmemPerSM / (by + kSmemReserve)));
            if (per_sm < 1) break;
            const int64_t blocks = (fibres + fb - 1) / fb;
            if (fb > 1 && blocks < kSMs) break;
            const double waves = std::max(1.0, (double)blocks / ((double)per_sm * kSMs));
            if (best == 0 || waves <= best_waves) {
                best = fb;
                best_waves = waves;
            }
        }
        tc.fb[a] = best;
        if (best) smem = std::max(smem, tile_bytes(L, best, nbuf, sizeof(T)));
    }
    return tc;
}

// The pieces of a pass along axis a: P lanes per fibre and nf fibres per block.
// Shorter pieces mean shorter chains but more work (each piece scans about a
// segment twice): pieces have at most 64 entries, and fewer (down to 10) while
// the fibres in flight (the launch's, or those an SM's shared memory holds)
// would give an SM fewer than 8 warps. Measured, ms a solve at P = 4, 8, 16, 32:
// 64 x 512^2 (221 fibres per SM) 85, 75, 77, 96; 16 x 256^2 weighted (28) 13.0,
// 11.7, 11.9, 13.5; 4 x 1024^2 weighted (28) 59, 40, 32, 30; 2048^2 (14) 63,
// 45, 38, 38; 200 x 301 (2) 7.9, 6.6, 6.0, 6.2; 90^2 (0.6) 2.6, 2.2, 2.2, 2.3.
// Blocks of 64, 128 and 256 threads run alike; a block keeps to kFibSmem so
// that an SM holds several. 0 fibres when one does not fit.
template <class T>
FibCfg fib_cfg(const AnGeom &g, int a, bool w, int64_t nimg, size_t &smem) {
    const int L = (int)g.L[a];
    const int64_t fibres = nimg * (g.N / g.L[a]);
    FibCfg c{};
    c.P = 1;
    const int64_t one = (int64_t)(w ? 2 : 1) * L * (int64_t)sizeof(T) + L;  // a fibre's shared memory
    const double flight = std::min((double)fibres / kSMs, (double)kSmemPerSM / (double)std::max<int64_t>(one, 1));
    while (c.P < 32 && (L > 64 * c.P || (flight * c.P < 8 * 32 && L / (2 * c.P) >= 10))) c.P *= 2;
    c.len = ((L + c.P - 1) / c.P) | 1;
    c.pitch = L | 1;
    // at least a warp, and 8 fibres (a 32-byte sector of floats) across a strided axis
    const int lo = std::max(32 / c.P, g.S[a] == 1 ? 1 : std::min(8, kFibThreads / c.P));
    c.nf = std::max(128 / c.P, lo);
    while ((smem = fib_smem<T>(c, L, w)) > (size_t)kFibSmem && c.nf > lo) c.nf /= 2;
    while ((smem = fib_smem<T>(c, L, w)) > (size_t)kTileSmemMax && c.nf > 32 / c.P) c.nf /= 2;
    while (smem > (size_t)kTileSmemMax && c.P < 32) {
        c.P *= 2;
        c.nf = 32 / c.P;
        c.len = ((L + c.P - 1) / c.P) | 1;
        smem = fib_smem<T>(c, L, w);
    }
    if (smem > (size_t)kTileSmemMax) c.nf = 0;
    return c;
}

// Blocks of a pass along any axis: most with the most pieces per fibre. Doubling
// the images of a launch halves its pieces at most, so launches of 1, 2, 4 ..
// images meet every number of pieces that any launch has. (With partial sums for
// the other kernels' blocks only, large volumes along two axes fell back to a
// thread per fibre: 20 iterations of 256 x 512^2 in 120 ms against 97, of
// 128 x 512^2 with edge weights in 78 against 71.)
template <class T>
int64_t piece_parts(const AnGeom &g, bool has_beta) {
    int64_t most = 0;
    for (int a = 0; a < g.k; ++a) {
        if (g.L[a] < 2) continue;
        for (int64_t nimg = 1;; nimg = std::min(2 * nimg, g.B)) {
            size_t smem = 0;
            const FibCfg fc = fib_cfg<T>(g, a, has_beta, nimg, smem);
            if (fc.nf > 0) most = std::max(most, (g.N / g.L[a] + fc.nf - 1) / fc.nf);
            if (nimg >= g.B) break;
        }
    }
    return most;
}

template <class T, int PASS>
cudaError_t fib_pass(const AnGeom &g, const AnCall &c, const AnBuffers &bf, const FibCfg &fc, size_t smem, int a,
                     unsigned B, cudaStream_t s) {
    const dim3 grid((unsigned)((g.N / g.L[a] + fc.nf - 1) / fc.nf), B);
    // 16-byte loads across the fibres where every row starts on 16 bytes
    const bool vec = g.S[a] > 1 && g.S[a] % kFibVec<T> == 0 && fc.nf % kFibVec<T> == 0;
    auto run = [&](auto kernel) { kernel<<<grid, fc.nf * fc.P, smem, s>>>(g, c, bf, fc); };
    if (c.has_beta) run(vec ? an_fib_pass<T, PASS, true, kFibVec<T>> : an_fib_pass<T, PASS, true, 1>);
    else run(vec ? an_fib_pass<T, PASS, false, kFibVec<T>> : an_fib_pass<T, PASS, false, 1>);
    return cudaGetLastError();
}

template <class T>
cudaError_t round_t(const AnGeom &g, const AnCall &c, const AnBuffers &bf, int64_t nimg, bool tail, cudaStream_t s,
                   int64_t *launches) {
    if (nimg <= 0) return cudaSuccess;
    const unsigned B = (unsigned)nimg;
    int64_t nl = 0;
    // blocks per image: enough for the SMs, no more than the image has chunks
    const int64_t per = std::max<int64_t>(1, (int64_t)kSMs * 16 / B);
    const dim3 pg((unsigned)std::min<int64_t>(an_pixel_blocks(g), per), B);
    // the iteration: ADBPG's two passes, or FDPG-3's three
    int64_t nf[3] = {1, 1, 1};
    for (int a = 0; a < g.k; ++a) nf[a] = g.N / g.L[a];
    int64_t nfmax = 0;
    for (int a = 0; a < g.k; ++a) nfmax = std::max(nfmax, nf[a]);
    const unsigned fbk = (unsigned)((nfmax + 127) / 128);
    bool pieces = false;
    int a1 = 0, a2 = 0;
    FibCfg fc1{}, fc2{};
    size_t sm1 = 0, sm2 = 0;
    if (c.has_adbpg && aniso_pieces_enabled()) {
        // the active axes of ADBPG (the same for every image of the call), a1 the
        // one of smaller stride
        int act[3], n = 0;
        for (int a = 0; a < g.k; ++a)
            if (c.w[a] > 0.0 && g.L[a] > 1) act[n++] = a;
        a1 = g.S[act[0]] < g.S[act[1]] ? act[0] : act[1];
        a2 = a1 == act[0] ? act[1] : act[0];
        fc1 = fib_cfg<T>(g, a1, c.has_beta, nimg, sm1);
        fc2 = fib_cfg<T>(g, a2, c.has_beta, nimg, sm2);
        // (whether a fibre fits does not depend on nimg: every round of a solve runs the same passes)
        pieces = fc1.nf > 0 && fc2.nf > 0;
        if (pieces && (nf[a2] + fc2.nf - 1) / fc2.nf > bf.max_part) return cudaErrorInvalidValue;
    }
    if (pieces) {
        tile_attributes<T>();
        cudaError_t e = fib_pass<T, 1>(g, c, bf, fc1, sm1, a1, B, s);
        if (e == cudaSuccess) e = fib_pass<T, 2>(g, c, bf, fc2, sm2, a2, B, s);
        if (e != cudaSuccess) return e;
        nl += 2;
    } else if (c.has_adbpg) {
        size_t smem = 0;
        const TileCfg tc = tile_cfg<T>(g, c, nimg, smem);
        bool tiled = true;
        int64_t tblk = 0;
        for (int a = 0; a < g.k; ++a) {
            if (g.L[a] > 1 && tc.fb[a] == 0) tiled = false;
            if (tc.fb[a]) tblk = std::max<int64_t>(tblk, (nf[a] + tc.fb[a] - 1) / tc.fb[a]);
        }
        if (tiled && tblk > 0 && tblk <= bf.max_part) {
            tile_attributes<T>();
            an_pass1_tile<T><<<dim3((unsigned)tblk, B), kTileThreads, smem, s>>>(g, c, bf, tc);
            an_pass2_tile<T><<<dim3((unsigned)tblk, B), kTileThreads, smem, s>>>(g, c, bf, tc);
        } else {
            an_pass1<T><<<dim3(fbk, B), 128, 0, s>>>(g, c, bf);
            an_pass2<T><<<dim3(fbk, B), 128, 0, s>>>(g, c, bf);
        }
        nl += 2;
    }
    if (c.has_fdpg3) {
        an_fdpg3_u<T><<<pg, kThreads, 0, s>>>(g, bf);
        size_t smem = 0;
        const TileCfg tc = tile_cfg<T>(g, c, nimg, smem);
        int64_t tblk = 0;
        bool tiled = g.k == 3;
        for (int a = 0; a < g.k; ++a) {
            if (tc.fb[a] == 0) tiled = false;
            else tblk = std::max<int64_t>(tblk, (nf[a] + tc.fb[a] - 1) / tc.fb[a]);
        }
        if (tiled && tblk > 0 && 3 * tblk <= bf.max_part) {
            tile_attributes<T>();
            an_fdpg3_tile<T><<<dim3((unsigned)tblk, 3, B), kTileThreads, smem, s>>>(g, c, bf, tc);
        } else {
            an_fdpg3_pass<T><<<dim3(fbk, 3, B), 128, 0, s>>>(g, c, bf);
        }
        nl += 2;
    }
    if (!pieces) {  // the piece passes read y in place of the extrapolation after a restart
        an_restart_copy<T><<<pg, kThreads, 0, s>>>(g, bf);
        ++nl;
    }
    if (c.warm && c.has_adbpg) {
        // a warm start's pass (run by the first pass above) and its dual
        an_warm_z<T><<<pg, kThreads, 0, s>>>(g, bf);
        an_warm_next<<<((unsigned)g.B + 127) / 128, 128, 0, s>>>(g, bf);
        nl += 2;
    }
    // gap check (FDPG-3 forms its primal first)
    if (c.has_fdpg3) {
        an_fdpg3_primal<T><<<dim3((unsigned)((nf[2] + 127) / 128), B), 128, 0, s>>>(g, c, bf, kStCheck);
        ++nl;
    }
    an_gap<T><<<pg, kThreads, 0, s>>>(g, c, bf, kStCheck);
    ++nl;
    if (tail) {
        // polish
        an_dual<T><<<pg, kThreads, 0, s>>>(g, bf, kStPolish);
        for (int a = 0; a < g.k; ++a) {
            if (!(c.w[a] > 0.0 && g.L[a] > 1)) continue;
            if (g.S[a] == 1) {
                const int64_t bl = (nf[a] + kThreads / 32 - 1) / (kThreads / 32);
                an_mark_rows<T><<<dim3((unsigned)std::min(bl, per), B), kThreads, 0, s>>>(g, c, bf, a);
            } else {
                const int64_t bl = (nf[a] + kMarkCols - 1) / kMarkCols;
                an_mark_cols<T>
                    <<<dim3((unsigned)std::min(bl, per), B), kMarkCols * kMarkParts, 0, s>>>(g, c, bf, a);
            }
            ++nl;
        }
        an_union<<<pg, kThreads, 0, s>>>(g, bf);
        an_region_sum<T><<<pg, kThreads, 0, s>>>(g, bf);
        an_polish_gap<T><<<pg, kThreads, 0, s>>>(g, c, bf);
        an_polish_write<T><<<pg, kThreads, 0, s>>>(g, bf);
        // final rebuild, then retirement (over every image)
        const unsigned BA = (unsigned)g.B;
        an_dual<T><<<pg, kThreads, 0, s>>>(g, bf, kStFinal);
        an_gap<T><<<pg, kThreads, 0, s>>>(g, c, bf, kStFinal);
        an_retire<<<(BA + 127) / 128, 128, 0, s>>>(g, bf);
        nl += 8;
    }
    if (launches) *launches += nl;
    return cudaGetLastError();
}

template <class T>
cudaError_t warm_t(const AnGeom &g, const AnCall &c, const AnBuffers &bf, cudaStream_t s) {
    for (int a = 0; a < g.k; ++a) {
        const int64_t nf = g.N / g.L[a];
        an_warm_feasible<T><<<dim3((unsigned)((nf + 127) / 128), (unsigned)g.B), 128, 0, s>>>(g, c, bf, a);
    }
    an_warm_init<T><<<dim3(an_pixel_blocks(g), (unsigned)g.B), kThreads, 0, s>>>(g, bf);
    an_warm_state<<<((unsigned)g.B + 127) / 128, 128, 0, s>>>(g, bf);
    return cudaGetLastError();
}

template <class T>
cudaError_t output_t(const AnGeom &g, const AnBuffers &bf, void *out, cudaStream_t s) {
    an_output<T><<<dim3(an_pixel_blocks(g), (unsigned)g.B), kThreads, 0, s>>>(g, bf, static_cast<T *>(out));
    return cudaGetLastError();
}

}  // namespace

bool aniso_pieces_enabled() {
    static const bool on = [] {  // tuning hint FASTPROX_B200_AN_FIB=0: the tiled passes
        const char *v = std::getenv("FASTPROX_B200_AN_FIB");
        return !(v && v[0] == '0' && v[1] == 0);
    }();
    return on;
}

int64_t aniso_piece_parts(int dtype, const AnGeom &g, bool has_beta) {
    return dtype == 1 ? piece_parts<float>(g, has_beta) : piece_parts<double>(g, has_beta);
}

int an_pixel_blocks(const AnGeom &g) { return pixel_chunks(g.N); }

cudaError_t aniso_setup(int dtype, const AnGeom &g, const AnCall &c, const AnBuffers &bf, const void *x,
                        cudaStream_t s) {
    return dtype == 1 ? setup_t<float>(g, c, bf, x, s) : setup_t<double>(g, c, bf, x, s);
}

cudaError_t aniso_warm(int dtype, const AnGeom &g, const AnCall &c, const AnBuffers &bf, cudaStream_t s) {
    return dtype == 1 ? warm_t<float>(g, c, bf, s) : warm_t<double>(g, c, bf, s);
}

void aniso_prepare(int dtype) {
    if (dtype == 1) tile_attributes<float>();
    else tile_attributes<double>();
}

cudaError_t aniso_round(int dtype, const AnGeom &g, const AnCall &c, const AnBuffers &bf, int64_t nimg, bool tail,
                        cudaStream_t s, int64_t *launches) {
    return dtype == 1 ? round_t<float>(g, c, bf, nimg, tail, s, launches)
                      : round_t<double>(g, c, bf, nimg, tail, s, launches);
}

cudaError_t aniso_live_list(const AnState *st, int64_t B, int *lmap, int *lcnt, cudaStream_t s) {
    an_live_list<<<1, 1024, 0, s>>>(st, B, lmap, lcnt);
    return cudaGetLastError();
}

cudaError_t aniso_output(int dtype, const AnGeom &g, const AnBuffers &bf, void *out, cudaStream_t s) {
    return dtype == 1 ? output_t<float>(g, bf, out, s) : output_t<double>(g, bf, out, s);
}

}  // namespace fpb
