// Weighted Approximate-Min* decoder: forward and adjoint kernels (see ldpc_weighted.cuh).
//
// Both kernels are templates over the real type.  float is the training and simulation type; its
// arithmetic is the plain decoder's (the same correctly rounded operations in the same order, the
// same min* step), so alpha = 1, beta = 0 gives the plain fp32 decoder's values bit for bit.  double
// exists to check the adjoint against central finite differences, which need more precision than
// float has.
#include <algorithm>
#include <cstdio>
#include <string>

#include "../../include/ldpcb200.h"
#include "ldpc_weighted.cuh"

namespace ldpcb200 {

template <typename Real>
struct WOps;

template <>
struct WOps<float> {
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float abs(float a) { return fabsf(a); }
    static __device__ __forceinline__ float min(float a, float b) { return fminf(a, b); }
    // the sign bit in place (bit 31 of the high word), and a value with its sign flipped by such a mask
    static __device__ __forceinline__ uint32_t top(float a) { return __float_as_uint(a); }
    static __device__ __forceinline__ float flip(float a, uint32_t sign) { return __uint_as_float(__float_as_uint(a) ^ sign); }
    static __device__ __forceinline__ float step(float m, float a) { return amin_step_fma(m, a); }
};

template <>
struct WOps<double> {
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double abs(double a) { return fabs(a); }
    static __device__ __forceinline__ double min(double a, double b) { return fmin(a, b); }
    static __device__ __forceinline__ uint32_t top(double a) { return (uint32_t)__double2hiint(a); }
    static __device__ __forceinline__ double flip(double a, uint32_t sign) {
        return __hiloint2double(__double2hiint(a) ^ (int)sign, __double2loint(a));
    }
    // max(min(m, a) - g(|m - a|), 0), g = 0.69315 - 0.4 d (d < 0.5), 0.49315 - 0.328 (d - 0.5) (d < 2), 0
    static __device__ __forceinline__ double step(double m, double a) {
        const double diff = fabs(__dsub_rn(m, a));
        const double cur = fmin(m, a);
        const double g = diff < 0.5 ? __dsub_rn(0.69315, __dmul_rn(0.40, diff))
                                    : (diff < 2.0 ? __dsub_rn(0.49315, __dmul_rn(0.328, __dsub_rn(diff, 0.5))) : 0.0);
        const double v = __dsub_rn(cur, g);
        return v > 0.0 ? v : 0.0;
    }
};

// Row structure shared by forward and backward: sign parity (bit 31), the flags lt[i] ("the argmin lies after
// edge i") and the minimum, as the plain decoder's row update (flags from prefix minima up to degree
// 10, from the argmin's index above: see row_update).
template <typename Real, int d>
__device__ __forceinline__ Real wrow_prep(const Real (&q)[d], uint32_t& par, bool (&lt)[d]) {
    using O = WOps<Real>;
    par = 0;
#pragma unroll
    for (int e = 0; e < d; ++e) par ^= O::top(q[e]);
    Real mn;
    if constexpr (d > 10) {
        mn = Real(9999);
        int am = 0;
#pragma unroll
        for (int e = 0; e < d; ++e) {
            am = O::abs(q[e]) < mn ? e : am;
            mn = O::min(mn, O::abs(q[e]));
        }
#pragma unroll
        for (int i = 0; i < d; ++i) lt[i] = (i + 1 < d) ? (i < am) : false;
    } else {
        Real pm[d];
        pm[0] = O::min(O::abs(q[0]), Real(9999));
#pragma unroll
        for (int e = 1; e < d; ++e) pm[e] = O::min(pm[e - 1], O::abs(q[e]));
        mn = pm[d - 1];
#pragma unroll
        for (int i = 0; i < d; ++i) lt[i] = (i + 1 < d) ? (pm[i] > mn) : false;
    }
    return mn;
}

// Pairs of values (a row's edges 2k and 2k+1, or one edge's alpha and beta).
template <typename Real> struct WPair;
template <> struct WPair<float> { using T = float2; };
template <> struct WPair<double> { using T = double2; };
template <typename Real>
__device__ __forceinline__ typename WPair<Real>::T wpair(Real a, Real b) {
    typename WPair<Real>::T v;
    v.x = a;
    v.y = b;
    return v;
}

// First pair of layer l in a frame's message-shaped arrays (messages, stashed q, adjoints): pair k of
// row j at [k * Z + j], a row of odd degree padded to the next pair.
template <int Z, int D>
__device__ __forceinline__ int wlayer_pair(int l) {
    constexpr int HL = (QC_DEG_LOW + 1) / 2, HD = (D + 1) / 2;
    return l < 4 ? l * HL * Z : (4 * HL + (l - 4) * HD) * Z;
}

// Column of edge e of row j of layer l.  edge[l][e] holds the circulant's block offset and shift in one
// word (the offset a multiple of Z, the shift below it), so the index is an add and a bit select.
template <int Z, int d>
__device__ __forceinline__ void wrow_index(const WParams& p, int l, int j, int (&idx)[d]) {
#pragma unroll
    for (int e = 0; e < d; ++e) {
        const int w = p.edge[l][e];
        idx[e] = ((w + j) & (Z - 1)) | (w & ~(Z - 1));
    }
}

// Forward update of row j of layer l (degree d): q from L and the old messages (rr), new messages and L.
// r: where the row's new messages go, or null when they are not needed.  stash: where q goes, or null.
// w: the layer's (alpha, beta) pairs.
template <typename Real, int Z, int d>
__device__ __forceinline__ void wrow_fwd(const WParams& p, Real* L, const typename WPair<Real>::T* rr,
                                         typename WPair<Real>::T* r, typename WPair<Real>::T* stash,
                                         const typename WPair<Real>::T* w, int l, int j) {
    using O = WOps<Real>;
    using W2 = typename WPair<Real>::T;
    constexpr int H = (d + 1) / 2;
    int idx[d];
    wrow_index<Z, d>(p, l, j, idx);
    Real q[d];
#pragma unroll
    for (int e = 0; e < d; ++e) q[e] = O::sub(L[idx[e]], (e & 1) ? rr[e / 2].y : rr[e / 2].x);
    if (stash) {
#pragma unroll
        for (int k = 0; k < H; ++k) stash[k * Z] = wpair<Real>(q[2 * k], 2 * k + 1 < d ? q[2 * k + 1 < d ? 2 * k + 1 : 0] : Real(0));
    }
    uint32_t par;
    bool lt[d];
    const Real mn = wrow_prep<Real, d>(q, par, lt);
    Real m = O::abs(lt[0] ? q[0] : q[1]);
#pragma unroll
    for (int i = 1; i + 1 < d; ++i) m = O::step(m, O::abs(lt[i] ? q[i] : q[i + 1]));
    const Real mall = O::step(m, mn);
    Real rn[2 * H];
    rn[2 * H - 1] = Real(0);
#pragma unroll
    for (int e = 0; e < d; ++e) {
        const bool is_am = (e == 0 ? true : lt[e - 1]) && !lt[e];
        const W2 ab = w[e];
        Real z = O::sub(O::mul(ab.x, is_am ? m : mall), ab.y);
        z = z > Real(0) ? z : Real(0);
        rn[e] = O::flip(z, (par ^ O::top(q[e])) & 0x80000000u);
        L[idx[e]] = O::add(q[e], rn[e]);
    }
    if (r) {
#pragma unroll
        for (int k = 0; k < H; ++k) r[k * Z] = wpair<Real>(rn[2 * k], rn[2 * k + 1]);
    }
}

// A row's message pairs, loaded one layer ahead: the loads need no barrier (a thread's rows are its own),
// so they are in flight while the row before is updated.
template <typename Real, int Z, int D>
__device__ __forceinline__ void wload(const typename WPair<Real>::T* r, int l, int j,
                                      typename WPair<Real>::T (&rr)[(D + 1) / 2]) {
    constexpr int HL = (QC_DEG_LOW + 1) / 2, HD = (D + 1) / 2;
    const typename WPair<Real>::T* row = r + wlayer_pair<Z, D>(l) + j;
#pragma unroll
    for (int k = 0; k < HD; ++k)
        if (k < HL || l >= 4) rr[k] = row[k * Z];
}

// The 12 layers of one forward iteration (the caller has filled the weights and synchronised L).  r_in: the
// old messages, or null in the first iteration, where they are zero; r: the new ones, or null when they
// are not needed.  rr holds layer 0's old messages on entry, and those of the next iteration (from r) on
// return.  stash may be r_in in an iteration that does not write r.  U: layers unrolled.  Unrolling saves the
// moves between the two sets of message registers (r1/2 K=1024, 4096 frames, 20 iterations: 0.957 ms rolled,
// 0.915 by two, 0.888 by four), until the bodies outgrow the instruction cache (r4/5 K=1024: 0.80 by two,
// 0.88 by four; in the backward kernel only degree 6 gains, by two).
template <typename Real, int Z, int D, int U>
__device__ __forceinline__ void wfwd_iteration(const WParams& p, Real* L, const typename WPair<Real>::T* r_in,
                                               typename WPair<Real>::T* r, typename WPair<Real>::T* stash,
                                               const typename WPair<Real>::T* sw, int j,
                                               typename WPair<Real>::T (&rr)[(D + 1) / 2]) {
    using W2 = typename WPair<Real>::T;
    constexpr int HD = (D + 1) / 2;
#pragma unroll U
    for (int l = 0; l < 4; ++l) {
        const int o = wlayer_pair<Z, D>(l) + j;
        W2 cur[HD];
#pragma unroll
        for (int k = 0; k < HD; ++k) cur[k] = rr[k];
        if (r_in) wload<Real, Z, D>(r_in, l + 1, j, rr);
        wrow_fwd<Real, Z, QC_DEG_LOW>(p, L, cur, r ? r + o : nullptr, stash ? stash + o : nullptr,
                                      sw + qc_edge_slot(l, 0, D), l, j);
        __syncthreads();
    }
#pragma unroll U
    for (int l = 4; l < QC_LAYERS; ++l) {
        const int o = wlayer_pair<Z, D>(l) + j;
        W2 cur[HD];
#pragma unroll
        for (int k = 0; k < HD; ++k) cur[k] = rr[k];
        if (l + 1 < QC_LAYERS) {
            if (r_in) wload<Real, Z, D>(r_in, l + 1, j, rr);
        } else if (r) {
            wload<Real, Z, D>(r, 0, j, rr);
        }
        wrow_fwd<Real, Z, D>(p, L, cur, r ? r + o : nullptr, stash ? stash + o : nullptr, sw + qc_edge_slot(l, 0, D), l,
                             j);
        __syncthreads();
    }
}

// (alpha, beta) of iteration t for every edge slot.
template <typename Real, int Z, int D>
__device__ __forceinline__ void wfill(const WParams& p, typename WPair<Real>::T* sw, const uint8_t* cls, int t, int tid) {
    const Real* a = static_cast<const Real*>(p.alpha) + t * p.n_classes;
    const Real* b = static_cast<const Real*>(p.beta) + t * p.n_classes;
    for (int s = tid; s < wslots(D); s += Z) sw[s] = wpair<Real>(a[cls[s]], b[cls[s]]);
}

template <int Z, int D>
__device__ __forceinline__ void wclasses(const WParams& p, uint8_t* cls, int tid) {
    for (int s = tid; s < wslots(D); s += Z) {
        const int l = s < 4 * QC_DEG_LOW ? s / QC_DEG_LOW : 4 + (s - 4 * QC_DEG_LOW) / D;
        cls[s] = (uint8_t)p.edge_class[l][s - qc_edge_slot(l, 0, D)];
    }
}

// Sums N values over a warp by halving: at each of the five exchanges a lane keeps one half of its
// values and sends the other, so N values take about N exchanges in place of 5 N.  Afterwards v[k],
// k < count, of a lane holds the warp's sum of value first + k (WSum: which values a lane ends with; count
// is 0 in lanes that hold the same sums as a lower lane, or padding).
struct WSum {
    int first, count;
};
template <int N> __device__ __forceinline__ WSum wsum_lane(int lane) {
    int first = 0, count = N, n = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            n = (n + 1) / 2;
            if (lane & o) {
                first += n;
                count -= n;
            } else {
                count = min(count, n);
            }
        } else if (lane & o) {
            count = 0;
        }
    }
    return WSum{first, max(count, 0)};
}
__host__ __device__ constexpr int wsum_left(int n) {
    for (int s = 0; s < 5; ++s) n = n > 1 ? (n + 1) / 2 : 1;
    return n;
}
template <typename Real, int N>
__device__ __forceinline__ void wsum(Real (&v)[N], int lane) {
    int n = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            const int h = (n + 1) / 2;
            const bool up = lane & o;
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (k < h) {
                    const Real lo = v[k], hi = k + h < n ? v[k + h < N ? k + h : 0] : Real(0);
                    const Real got = __shfl_xor_sync(0xFFFFFFFFu, up ? lo : hi, o);
                    v[k] = (up ? hi : lo) + got;
                }
            n = h;
        } else {
            v[0] += __shfl_xor_sync(0xFFFFFFFFu, v[0], o);
        }
    }
}

// Backward of one min* step v = step(m, a): gm (adjoint of v) becomes the adjoint of m, returns that of
// a.  With h = -g'(|m - a|) the smaller operand gets 1 - h and the larger h.  Where the result is
// clamped to 0 both are 0; at m == a the whole adjoint goes to a (a subgradient).
template <typename Real>
__device__ __forceinline__ Real wstep_back(Real m, Real a, Real v, Real& gm) {
    const Real diff = WOps<Real>::abs(WOps<Real>::sub(m, a));
    Real h = diff < Real(0.5) ? Real(0.40) : Real(0.328);
    h = (diff < Real(2.0) && diff > Real(0)) ? h : Real(0);
    const Real g = v > Real(0) ? gm : Real(0);
    const Real big = g * h, small = g - big;
    const bool s = m < a;
    gm = s ? small : big;
    return s ? big : small;
}

// Copies a thread's own pairs from global to its own place in shared memory without waiting
// (cp.async): the row after the current one of the backward pass is fetched while the current one is
// computed, at no cost in registers.
template <typename Real>
__device__ __forceinline__ void wcopy(typename WPair<Real>::T* dst, const typename WPair<Real>::T* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(Real) == 4) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void wcopy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Fetches layer l's q (from stash) and message adjoints (from gr, unless first) into the thread's stage:
// pairs [0, HD) and [HD, 2 HD), stride Z.
template <typename Real, int Z, int D>
__device__ __forceinline__ void wfetch(typename WPair<Real>::T* stage, const typename WPair<Real>::T* stash,
                                       const typename WPair<Real>::T* gr, int l, int j, bool first) {
    constexpr int HL = (QC_DEG_LOW + 1) / 2, HD = (D + 1) / 2;
    const int o = wlayer_pair<Z, D>(l) + j;
#pragma unroll
    for (int k = 0; k < HD; ++k)
        if (k < HL || l >= 4) wcopy<Real>(stage + k * Z, stash + o + k * Z);
    if (first) return;
#pragma unroll
    for (int k = 0; k < HD; ++k)
        if (k < HL || l >= 4) wcopy<Real>(stage + (HD + k) * Z, gr + o + k * Z);
}

// Backward of row j of layer l: adjoint of L (shared) and of the messages in place.  stage: the row's
// q and minus the adjoint of its messages, which are read before `next` starts
// the copy of the row after it into the same place; gr: where the latter goes.  acc: the warp's parameter-gradient
// sums, [alpha, beta][edge slot] from the layer's first slot on.  With row_uniform every edge of a layer
// has one class, so the row's gradients are added up first and go to the layer's first slot.
template <typename Real, int Z, int D, int d, class Next>
__device__ __forceinline__ void wrow_bwd(const WParams& p, Real* gL, typename WPair<Real>::T* gr,
                                         const typename WPair<Real>::T* stage, const typename WPair<Real>::T* w, Real* acc,
                                         int l, int j, int lane, Next next) {
    using O = WOps<Real>;
    using W2 = typename WPair<Real>::T;
    constexpr int H = (d + 1) / 2, HD = (D + 1) / 2;
    Real q[2 * H], A[2 * H];
    wcopy_wait();
#pragma unroll
    for (int k = 0; k < H; ++k) {
        const W2 v = stage[k * Z];
        q[2 * k] = v.x;
        q[2 * k + 1] = v.y;
    }
#pragma unroll
    for (int k = 0; k < H; ++k) {
        const W2 v = stage[(HD + k) * Z];
        A[2 * k] = v.x;
        A[2 * k + 1] = v.y;
    }
    next();
    int idx[d];
    wrow_index<Z, d>(p, l, j, idx);
    uint32_t par;
    bool lt[d];
    Real qd[d];
#pragma unroll
    for (int e = 0; e < d; ++e) qd[e] = q[e];
    const Real mn = wrow_prep<Real, d>(qd, par, lt);
    // the chain m[0] = |o_0|, m[i] = step(m[i - 1], |o_i|), o_i the i-th non-argmin edge
    Real m[d - 1];
    Real o[d - 1];
#pragma unroll
    for (int i = 0; i + 1 < d; ++i) o[i] = O::abs(lt[i] ? q[i] : q[i + 1]);
    m[0] = o[0];
#pragma unroll
    for (int i = 1; i + 1 < d; ++i) m[i] = O::step(m[i - 1], o[i]);
    const Real mall = O::step(m[d - 2], mn);
    Real g_min = Real(0), g_all = Real(0);
    Real gl[d], pg[2 * d];
#pragma unroll
    for (int e = 0; e < d; ++e) {
        const bool is_am = (e == 0 ? true : lt[e - 1]) && !lt[e];
        const W2 ab = w[e];
        gl[e] = gL[idx[e]];
        const Real a = gl[e] - A[e];
        const Real mag = is_am ? m[d - 2] : mall;
        const Real z = O::sub(O::mul(ab.x, mag), ab.y);
        const Real wt = z > Real(0) ? O::flip(a, (par ^ O::top(q[e])) & 0x80000000u) : Real(0);
        pg[e] = wt * mag;
        pg[d + e] = -wt;
        const Real gmag = wt * ab.x;
        g_min = is_am ? gmag : g_min;
        g_all += is_am ? Real(0) : gmag;
    }
    if (p.row_uniform) {
        Real s[2] = {pg[0], pg[d]};
#pragma unroll
        for (int e = 1; e < d; ++e) {
            s[0] += pg[e];
            s[1] += pg[d + e];
        }
        wsum<Real, 2>(s, lane);
        const WSum ws = wsum_lane<2>(lane);
        if (ws.count) acc[ws.first ? wslots(D) : 0] += s[0];
    } else {  // the first exchange pairs an edge's alpha sum with its beta sum
        wsum<Real, 2 * d>(pg, lane);
        const WSum ws = wsum_lane<2 * d>(lane);
        Real* dst = acc + (ws.first >= d ? wslots(D) + ws.first - d : ws.first);
#pragma unroll
        for (int k = 0; k < wsum_left(2 * d); ++k)
            if (k < ws.count) dst[k] += pg[k];
    }
    Real gm = g_all;
    const Real gmn = wstep_back<Real>(m[d - 2], mn, mall, gm);
    gm += g_min;
    Real go[d - 1];
#pragma unroll
    for (int i = d - 2; i >= 1; --i) go[i] = wstep_back<Real>(m[i - 1], o[i], m[i], gm);
    go[0] = gm;
    Real gq[2 * H];
    gq[2 * H - 1] = Real(0);
#pragma unroll
    for (int e = 0; e < d; ++e) {
        const bool is_am = (e == 0 ? true : lt[e - 1]) && !lt[e];
        const Real gabs = is_am ? gmn : (lt[e] ? go[e < d - 1 ? e : 0] : go[e > 0 ? e - 1 : 0]);
        gq[e] = gl[e] + O::flip(gabs, O::top(q[e]) & 0x80000000u);
        gL[idx[e]] = gq[e];
    }
#pragma unroll
    for (int k = 0; k < H; ++k) gr[k * Z] = wpair<Real>(gq[2 * k], gq[2 * k + 1]);
}

// Shared-memory arrays are padded to 16 bytes.
template <typename Real>
__host__ __device__ constexpr int wpad(int n) {
    return (n + (int)(16 / sizeof(Real)) - 1) & ~((int)(16 / sizeof(Real)) - 1);
}

// State i of frame b, at the start of a segment (iteration i * keep): L [N], then for i > 0 the messages (none
// before the first iteration).
template <typename Real, int Z, int D>
__device__ __forceinline__ Real* wckpt(const WParams& p, int i, int b) {
    const size_t n = p.n_frames, N = p.n_vars, S = N + 2 * (size_t)wedge_pairs(Z, D);
    return static_cast<Real*>(p.ckpt) + (i == 0 ? b * N : n * N + ((size_t)(i - 1) * n + b) * S);
}

// One CTA of Z threads per frame slot (persistent over the frames); thread j updates row j of every
// layer and is the only thread that touches those rows' pairs in the message-shaped arrays, so they
// need no synchronisation.  L lives in shared memory, a barrier after every layer.
//
// The state kept for the backward pass: the q of every row of the last `keep` iterations (stash), and
// when those are not all, the decoder's state at the iterations 0, keep, 2 keep, .. before them (ckpt).
// The messages of the frame being decoded sit in the stash's last iteration, which is written only when
// they are no longer needed.  (A state at the first kept iteration as well, for repeated backward passes
// only, took the room of a kept iteration's rows and cost 3 % here, 5 % of the backward kernel.)
//
// Bound by instruction issue (76 % of the slots, 42 lane instructions per edge and iteration at degree 6;
// 2.9 TB/s of posteriors and stash written).  The layers of one degree share one body in a loop, so a kernel
// is a few thousand instructions and its warps do not miss the instruction cache; a row's messages are
// read and written as pairs and loaded a layer ahead.  r1/2 K=1024, 4096 frames, 20 iterations (B200,
// 1965 MHz): 0.89 ms, 1.18 ms with the twelve layers unrolled and one word per message.
template <typename Real, int Z, int D>
__global__ void __launch_bounds__(Z) wfwd_kernel(const __grid_constant__ WParams p) {
    using W2 = typename WPair<Real>::T;
    constexpr int EP = wedge_pairs(Z, D);
    extern __shared__ __align__(16) unsigned char smw_raw[];
    const int N = p.n_vars, T = p.n_iter, K = p.keep, R = T - K;
    Real* L = reinterpret_cast<Real*>(smw_raw);
    W2* sw = reinterpret_cast<W2*>(L + wpad<Real>(N));
    uint8_t* cls = reinterpret_cast<uint8_t*>(sw + wslots(D));
    const int tid = threadIdx.x;
    Real* post = static_cast<Real*>(p.post);
    wclasses<Z, D>(p, cls, tid);
    for (int b = blockIdx.x; b < p.n_frames; b += gridDim.x) {
        const Real* llr = static_cast<const Real*>(p.llr) + (size_t)b * p.n_tx;
        W2* stash = static_cast<W2*>(p.stash) + (size_t)b * K * EP;
        W2* r = stash + (size_t)(K - 1) * EP;
        if (tid == 0) p.used[b] = 0;
        __syncthreads();  // the previous frame's last posteriors have been read; the classes are written
        for (int i = tid; i < N; i += Z) L[i] = i < p.n_tx ? llr[i] : Real(0);
        W2 rr[(D + 1) / 2] = {};
        for (int t = 0; t < T; ++t) {
            wfill<Real, Z, D>(p, sw, cls, t, tid);
            if (t < R && t % K == 0) {  // each thread stores its own variables and messages
                Real* ck = wckpt<Real, Z, D>(p, t / K, b);
                for (int i = tid; i < N; i += Z) ck[i] = L[i];
                if (t)
                    for (int i = tid; i < EP; i += Z) reinterpret_cast<W2*>(ck + N)[i] = r[i];
            }
            __syncthreads();
            wfwd_iteration<Real, Z, D, D <= 10 ? 4 : 2>(p, L, t ? r : nullptr, t < T - 1 ? r : nullptr,
                                       t >= R ? stash + (size_t)(t - R) * EP : nullptr, sw, tid, rr);
            if (p.post_all || t == T - 1) {
                Real* dst = post + ((size_t)(p.post_all ? t : 0) * p.n_frames + b) * N;
                for (int i = tid; i < N; i += Z) dst[i] = L[i];
            }
        }
    }
}

// Adjoint of one iteration: X (adjoint of the posteriors) in shared memory, gr (minus the adjoint of the
// messages), stash (its q), after (the q of the iteration walked next, or null).  primed: the stage holds,
// or is being sent, the last layer's row.
template <typename Real, int Z, int D>
__device__ __forceinline__ void wbwd_iteration(const WParams& p, Real* X, typename WPair<Real>::T* gr,
                                               const typename WPair<Real>::T* stash, typename WPair<Real>::T* sw,
                                               const uint8_t* cls, Real* acc, Real* gacc,
                                               typename WPair<Real>::T* stage, const typename WPair<Real>::T* after,
                                               bool primed, int b, int t, int tid) {
    const int N = p.n_vars, lane = tid & 31;
    const bool first = t == p.n_iter - 1;
    Real* wacc = acc + (tid >> 5) * 2 * wslots(D);
    if (!primed) wfetch<Real, Z, D>(stage, stash, gr, QC_LAYERS - 1, tid, first);
    wfill<Real, Z, D>(p, sw, cls, t, tid);
    if (p.gpost && (p.post_all || first)) {
        const Real* gp = static_cast<const Real*>(p.gpost) + ((size_t)(p.post_all ? t : 0) * p.n_frames + b) * N;
        for (int i = tid; i < N; i += Z) X[i] += gp[i];
    }
    __syncthreads();
#pragma unroll 1
    for (int l = QC_LAYERS - 1; l >= 4; --l) {
        const int o = wlayer_pair<Z, D>(l) + tid, s = qc_edge_slot(l, 0, D);
        wrow_bwd<Real, Z, D, D>(p, X, gr + o, stage, sw + s, wacc + s, l, tid, lane,
                                [&] { wfetch<Real, Z, D>(stage, stash, gr, l - 1, tid, first); });
        __syncthreads();
    }
#pragma unroll 1
    for (int l = 3; l >= 0; --l) {
        const int o = wlayer_pair<Z, D>(l) + tid, s = qc_edge_slot(l, 0, D);
        wrow_bwd<Real, Z, D, QC_DEG_LOW>(p, X, gr + o, stage, sw + s, wacc + s, l, tid, lane, [&] {
            if (l) wfetch<Real, Z, D>(stage, stash, gr, l - 1, tid, first);
            else if (after) wfetch<Real, Z, D>(stage, after, gr, QC_LAYERS - 1, tid, false);
        });
        __syncthreads();
    }
    // the iteration's parameter gradients: edge slots of all warps into their classes
    for (int i = tid; i < 2 * wslots(D); i += Z) {
        Real v = Real(0);
#pragma unroll
        for (int w = 0; w < Z / 32; ++w) {
            v += acc[w * 2 * wslots(D) + i];
            acc[w * 2 * wslots(D) + i] = Real(0);
        }
        if (v != Real(0)) {
            const int beta = i >= wslots(D);
            atomicAdd(&gacc[2 * (t * p.n_classes + cls[beta ? i - wslots(D) : i]) + beta], v);
        }
    }
}

// Adjoint: the iterations whose q the forward pass kept first, then the segments before them, each run
// forward again from its state (stashing every layer's q in the frame's stash, whose kept iterations
// are done with) and walked back.  The adjoint of the posteriors waits in global memory meanwhile.  A
// second backward pass of the same forward pass finds the frame's stash used and runs its kept
// iterations again as well, from the last state before them.
//
// Bound by instruction issue (64 % of the slots at 17 resident warps; about 75 lane instructions per edge
// and iteration walked back, half of them on the half-rate ALU pipe, plus the forward's for those run
// again).  What keeps it there: one body per degree instead of twelve unrolled layers (no instruction-cache
// misses), the next row's q and message adjoints on their way to shared memory while a row is computed,
// parameter gradients halved across the warp (wsum: 13 exchanges per degree-6 row instead of 60) and
// kept per edge slot until the iteration ends, CTAs that stay for many frames (one global atomic per
// CTA and parameter), and no second run of the kept iterations.  ms of the kernel, 20 iterations, every 5:
// r1/2 K=1024, 4096 frames 7.47 -> 2.47; r4/5 K=4096, 512 frames, one class per row 5.37 -> 1.02.
template <typename Real, int Z, int D, int B>
__global__ void __launch_bounds__(Z, B) wbwd_kernel(const __grid_constant__ WParams p) {
    using W2 = typename WPair<Real>::T;
    constexpr int EP = wedge_pairs(Z, D), WS = wslots(D);
    extern __shared__ __align__(16) unsigned char smw_raw[];
    const int N = p.n_vars, T = p.n_iter, K = p.keep, R = T - K, n_seg = (R + K - 1) / K, TC = T * p.n_classes;
    Real* X = reinterpret_cast<Real*>(smw_raw);
    W2* sw = reinterpret_cast<W2*>(X + wpad<Real>(N));
    Real* acc = reinterpret_cast<Real*>(sw + WS);
    Real* gacc = acc + 2 * WS * (Z / 32);
    const int tid = threadIdx.x;
    W2* stage = reinterpret_cast<W2*>(gacc + wpad<Real>(2 * TC)) + tid;
    uint8_t* cls = reinterpret_cast<uint8_t*>(stage - tid + 2 * ((D + 1) / 2) * Z);
    wclasses<Z, D>(p, cls, tid);
    for (int i = tid; i < 2 * WS * (Z / 32) + 2 * TC; i += Z) acc[i] = Real(0);
    W2* gr = static_cast<W2*>(p.gr) + (size_t)blockIdx.x * EP;
    Real* save = static_cast<Real*>(p.save) + (size_t)blockIdx.x * N;
    for (int b = blockIdx.x; b < p.n_frames; b += gridDim.x) {
        W2* stash = static_cast<W2*>(p.stash) + (size_t)b * K * EP;
        W2* r = stash + (size_t)(K - 1) * EP;
        __syncthreads();  // the previous frame's adjoints have been read; the classes are written
        for (int i = tid; i < N; i += Z) X[i] = Real(0);
#pragma unroll
        for (int k = 0; k < (D + 1) / 2; ++k)  // the last iteration's messages have no adjoint yet
            stage[((D + 1) / 2 + k) * Z] = wpair<Real>(Real(0), Real(0));
        const bool used = p.used[b];  // a backward pass has already run segments over the kept q
        for (int seg = n_seg; seg >= 0; --seg) {
            const int t0 = seg < n_seg ? seg * K : R, t1 = seg < n_seg ? min(R, t0 + K) : T;
            if (seg < n_seg || used) {
                // from the segment's own state, the kept part's again from the last one before it
                const int ts = seg < n_seg ? t0 : (n_seg - 1) * K;
                const Real* ck = wckpt<Real, Z, D>(p, ts / K, b);
                for (int i = tid; i < N; i += Z) {  // each thread's own variables
                    save[i] = X[i];
                    X[i] = ck[i];
                }
                if (tid == 0) p.used[b] = 1;
                const W2* r_in = ts ? reinterpret_cast<const W2*>(ck + N) : nullptr;
                W2 rr[(D + 1) / 2] = {};
                if (r_in) wload<Real, Z, D>(r_in, 0, tid, rr);
                for (int t = ts; t < t1; ++t) {
                    wfill<Real, Z, D>(p, sw, cls, t, tid);
                    __syncthreads();
                    wfwd_iteration<Real, Z, D, D <= 6 ? 2 : 1>(p, X, r_in, t < t1 - 1 ? r : nullptr,
                                                               t >= t0 ? stash + (size_t)(t - t0) * EP : nullptr, sw,
                                                               tid, rr);
                    r_in = r;
                }
                for (int i = tid; i < N; i += Z) X[i] = save[i];
            }
            for (int t = t1 - 1; t >= t0; --t)
                wbwd_iteration<Real, Z, D>(p, X, gr, stash + (size_t)(t - t0) * EP, sw, cls, acc, gacc, stage,
                                           t > t0 ? stash + (size_t)(t - 1 - t0) * EP : nullptr, t < t1 - 1, b, t, tid);
        }
        if (p.gllr) {
            Real* g = static_cast<Real*>(p.gllr) + (size_t)b * p.n_tx;
            for (int i = tid; i < p.n_tx; i += Z) g[i] = X[i];
        }
    }
    __syncthreads();
    Real* galpha = static_cast<Real*>(p.galpha);
    Real* gbeta = static_cast<Real*>(p.gbeta);
    for (int i = tid; i < TC; i += Z) {
        if (gacc[2 * i] != Real(0)) atomicAdd(&galpha[i], gacc[2 * i]);
        if (gacc[2 * i + 1] != Real(0)) atomicAdd(&gbeta[i], gacc[2 * i + 1]);
    }
}

// ----------------------------------------------------------------------------- host side

static size_t wsmem_bytes(const WParams& p, int Z, int D, bool fwd, size_t rb) {
    const size_t slots = wslots(D);
    size_t elems = (rb == 8 ? wpad<double>(p.n_vars) : wpad<float>(p.n_vars)) + 2 * slots;
    if (!fwd) {
        const int tc2 = 2 * p.n_iter * p.n_classes;
        elems += 2 * slots * (Z / 32) + (rb == 8 ? wpad<double>(tc2) : wpad<float>(tc2));
        elems += 2 * 2 * (size_t)((D + 1) / 2) * Z;  // one row's q and message adjoints per thread
    }
    return elems * rb + slots;
}

// Resident CTAs per SM the backward kernel is compiled for, the most it is launched with (its CTAs own
// one message-adjoint slot each).
static int wslots_per_sm(int Z, int D, size_t rb);

// Chooses how many iterations' q the forward pass keeps: as many as fit the memory that checkpoints
// of the whole state every ckpt_every iterations, one segment's q and two message arrays would take
// (what ckpt_every asks for), so every kept iteration is one the backward pass need not run again.
size_t weighted_plan(WParams* p, int Z, int D, int ckpt_every, int n_sm, size_t rb) {
    const size_t n = p->n_frames, N = p->n_vars, E = (size_t)Z * wslots(D), EP2 = 2 * (size_t)wedge_pairs(Z, D);
    const int T = p->n_iter;
    const size_t n_ckpt = (T + ckpt_every - 1) / ckpt_every;
    const size_t budget = n * (n_ckpt * (N + E) + (size_t)(ckpt_every + 2) * E) * rb;
    p->n_slots = (int)std::min<size_t>(n, (size_t)n_sm * wslots_per_sm(Z, D, rb));
    if (!n) return 0;
    auto lay = [&](int K) {
        const size_t R = T - K, seg = (R + K - 1) / K;
        p->keep = K;
        p->off_ckpt = n * (size_t)K * EP2;
        p->off_gr = p->off_ckpt + (R ? n * (N + (seg - 1) * (N + EP2)) : 0);
        p->off_save = p->off_gr + p->n_slots * EP2;
        p->off_used = p->off_save + p->n_slots * N;
        return (p->off_used + n) * rb + W_ALIGN;
    };
    int K = T;
    while (K > 1 && lay(K) > budget) --K;
    if (lay(K) > budget) K = ckpt_every;
    return lay(K);
}

template <typename Real, int Z, int D, int B>
static int wlaunch(const WParams& p, bool fwd, int n_sm, cudaStream_t s, std::string& err) {
    const void* fn = fwd ? reinterpret_cast<const void*>(&wfwd_kernel<Real, Z, D>)
                         : reinterpret_cast<const void*>(&wbwd_kernel<Real, Z, D, B>);
    const size_t smem = wsmem_bytes(p, Z, D, fwd, sizeof(Real));
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        err = "weighted decoder: frame too large for shared memory";
        return LDPC_ENOTSUP;
    }
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, Z, smem);
    if (e != cudaSuccess || per_sm <= 0) {
        cudaGetLastError();
        err = "weighted decoder: the kernel does not fit on an SM";
        return LDPC_ENOTSUP;
    }
    const int64_t most = fwd ? (int64_t)p.n_frames : (int64_t)p.n_slots;
    const unsigned grid = (unsigned)std::min<int64_t>(most, (int64_t)per_sm * n_sm);
    void* args[] = {const_cast<WParams*>(&p)};
    e = cudaLaunchKernel(fn, dim3(grid), dim3(Z), args, smem, s);
    if (e != cudaSuccess) {
        err = std::string("weighted decoder launch: ") + cudaGetErrorString(e);
        return LDPC_EIO;
    }
    return 0;
}

// Code shapes (Z, D, resident CTAs per SM the backward kernel's registers must allow) of the float
// kernels: rate 1/2 and 4/5 at K = 1024 and 4096, rate 2/3 at K = 1024.  The caps are the fastest measured
// (ms of the backward kernel, 20 iterations): r1/2 K=1024, 4096 frames: 5 CTAs (88 registers) 2.56, 6 2.62,
// 7 2.75; r1/2 K=4096, 900 frames: 2 (64) 2.72, 1 (96) 3.04; r2/3 K=1024, 4000 frames: 8 (126) 2.21, 10 2.46,
// 12 2.35; r4/5 K=1024, 4000 frames: 16 (128) 3.02, 20 3.89; r4/5 K=4096, 512 frames: 4 (128) 1.17, 5 1.54, 3
// 1.36.  The double kernels (adjoint checks) cover rate 1/2 and 4/5 at K = 1024.
#define W_SHAPES_F32(X) X(128, 6, 5) X(512, 6, 2) X(64, 10, 8) X(32, 18, 16) X(128, 18, 4)
#define W_SHAPES_F64(X) X(128, 6, 2) X(32, 18, 8)

bool weighted_supported(int Z, int D, int real_bytes) {
#define W_SUP(z, d, b) if (Z == z && D == d) return true;
    if (real_bytes == 4) { W_SHAPES_F32(W_SUP) }
    if (real_bytes == 8) { W_SHAPES_F64(W_SUP) }
#undef W_SUP
    return false;
}

static int wslots_per_sm(int Z, int D, size_t rb) {
#define W_PER_SM(z, d, b) if (Z == z && D == d) return b;
    if (rb == 4) { W_SHAPES_F32(W_PER_SM) }
    if (rb == 8) { W_SHAPES_F64(W_PER_SM) }
#undef W_PER_SM
    return 1;
}

int weighted_launch(const WParams& p, int Z, int D, int real_bytes, bool fwd, int n_sm, cudaStream_t s,
                    std::string& err) {
    if (!p.n_frames) return 0;
#define W_CALL_F32(z, d, b) if (Z == z && D == d) return wlaunch<float, z, d, b>(p, fwd, n_sm, s, err);
#define W_CALL_F64(z, d, b) if (Z == z && D == d) return wlaunch<double, z, d, b>(p, fwd, n_sm, s, err);
    if (real_bytes == 4) { W_SHAPES_F32(W_CALL_F32) }
    if (real_bytes == 8) { W_SHAPES_F64(W_CALL_F64) }
#undef W_CALL_F32
#undef W_CALL_F64
    err = "weighted decoder is not built for this code shape";
    return LDPC_ENOTSUP;
}

}  // namespace ldpcb200
