// Translations without atomics: the FP64 matvec, its float-float form (FMM_FLOAT2) and the
// deterministic mixed matvec.
//
// Every translation is rotation - coaxial - rotation (transMatsVecsMul_SR_rcr, reference
// translation.cu:1864-1961).  A pass's translations are grouped by operator class: the M2L
// directions of equal (dz, dx^2 + dy^2) have one polar angle and one length, so they share the
// rotation block and the coaxial block and differ only by azimuthal phases (61 classes of the
// 316 directions; two polar angles for the octants of M2M and L2L).  A CTA takes TC
// translations of one class as columns and applies the three stages in shared memory; a lane
// owns one column (and one of 32/TC row groups), so that every rotation or coaxial entry is one
// load for all columns and no lane idles on a short row.  The result of a translation goes to
// its own slot of a scratch buffer (slots in destination order), and own_reduce_kernel adds
// each destination's slots in list order: no atomics, results repeat bit for bit.  Passes whose
// results exceed the scratch run in chunks of consecutive destination boxes.
//
// FP64 and float-float keep the expansions between P2M and L2P in the basis x+_m = x_m + x_-m,
// x-_m = x_m - x_-m (m > 0; x+_0 = x_0).  The rotation block is centrally symmetric,
// H_{-m',-m} = H_{m',m}, so it splits into one block for x+ and one for x-: half the multiply-adds
// of the rotations; the coaxial block is the same for +m and -m and does not see the basis; and
// the phases cost 4 instead of 6 operations per entry and side.  The FP32 instantiation keeps the
// plain basis and the order of operations of the mixed tiles' predecessor, so that deterministic
// results stay what they were bit for bit.
//
// What bounds it: the FP64 pipe (2 multiply-adds per clock and SM; the tiles keep it 95-97 %
// busy), in float-float the FP32 pipes (15 instructions per multiply-add): 16 p^3 / 3
// multiply-adds per translation against 8 p^3 with the whole rotation block.  Measured against one
// CTA per destination box, which took its translations one after another with a lane per
// output: FP64 matvec on the 81,920-triangle sphere (p = 40 .. 10) 69.7 -> 27.3 ms (level-6 M2L
// 23.5 -> 8.4), float-float on the 200,000-triangle head (p = 40 .. 8) 30.1 -> 15.1 ms,
// deterministic mixed on the 20,480-triangle sphere 2.36 -> 1.14 ms.
#include "plan.h"
#include "ff.cuh"
#include "f32x2.cuh"
#include <algorithm>
#include <condition_variable>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

namespace fmm {

namespace {

// folded rotation table: degree n holds (n+1) x (2n+1) entries [m][j], m = 0..n, row j <= n the
// x+ row m' = j, row j > n the x- row m' = j - n (its m = 0 entry is zero)
__host__ __device__ __forceinline__ int fold_off(int n) { return n * (4 * n * n + 3 * n - 1) / 6; }
__host__ __device__ __forceinline__ int fold_size(int p) { return fold_off(p); }
// ---- arithmetic of one type: V a complex number (one 8- or 16-byte value in memory), X the same
// prepared for multiply-adds, S a real table entry, K a complex one, E a phase; V accumulates
// real and CA complex products, value() is the finished sum.
template <typename T> struct Ops;

template <> struct Ops<double> {
    typedef double2 V;
    typedef double S;
    typedef double2 K;
    typedef double2 E, X, CA;
    static constexpr bool FOLD = true;
    static constexpr int NORM = 4;
    static constexpr int R = 1;  // rows per lane
    static __device__ __forceinline__ V load(const V *p) { return *p; }
    static __device__ __forceinline__ void store(V *p, V v) { *p = v; }
    static __device__ __forceinline__ V zero() { return make_double2(0.0, 0.0); }
    static __device__ __forceinline__ CA czero() { return zero(); }
    static __device__ __forceinline__ S table(const S *p) { return __ldg(p); }
    static __device__ __forceinline__ K table(const K *p) { return __ldg(p); }
    static __device__ __forceinline__ X prep(V v) { return v; }
    static __device__ __forceinline__ V add(V a, V b) { return make_double2(a.x + b.x, a.y + b.y); }
    static __device__ __forceinline__ void mac(V &a, S h, X x)
    {
        a.x = fma(h, x.x, a.x);
        a.y = fma(h, x.y, a.y);
    }
    static __device__ __forceinline__ void cmac(CA &a, K c, X x)
    {
        a.x = fma(c.x, x.x, a.x);
        a.x = fma(-c.y, x.y, a.x);
        a.y = fma(c.x, x.y, a.y);
        a.y = fma(c.y, x.x, a.y);
    }
    static __device__ __forceinline__ V value(V a) { return a; }
    static __device__ __forceinline__ V norm(V a) { return a; }
    // cos x + i sin y, the phases in the folded basis; e = (cos, sin)
    static __device__ __forceinline__ V phase(E e, V x, V y)
    {
        return make_double2(fma(-e.y, y.y, e.x * x.x), fma(e.y, y.x, e.x * x.y));
    }
    static __device__ __forceinline__ E conj(E e) { return make_double2(e.x, -e.y); }
};

// Float-float: the pairs (re, im) of the high and of the low parts side by side, so that the packed
// FP32 instructions (two FP32 operations each, at the FP32 pipes' rate but half the issue slots)
// work on re and im together.  Each half rounds as the scalar operation would.
struct __align__(16) ffv {
    f2 hi, lo;
};
// a table entry with both halves equal, so that a 16-byte load gives the operands of the packed
// instructions
struct __align__(16) ffs {
    f2 hi, lo;
};
struct __align__(16) ffk {
    ffs x, y;
};

template <> struct Ops<ff> {
    typedef ffv V;
    typedef ffs S;
    typedef ffk K;
    typedef float4 E;  // (cos hi, cos lo, sin hi, sin lo)
    struct X {
        f2 hi, nhi, lo;  // nhi = -hi
    };
    struct CA {
        V x, y;  // sums of re(c) v and of im(c) v
    };
    static constexpr bool FOLD = true;
    static constexpr int R = 2;
    static constexpr int NORM = 1;  // products between two norm()
    static __device__ __forceinline__ V load(const V *p)
    {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
        return V{v.x, v.y};
    }
    static __device__ __forceinline__ void store(V *p, V v) { *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v.hi, v.lo); }
    static __device__ __forceinline__ S table(const S *p)
    {
        const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(p));
        return S{v.x, v.y};
    }
    static __device__ __forceinline__ K table(const K *p) { return K{table(&p->x), table(&p->y)}; }
    static __device__ __forceinline__ V zero() { return V{0ull, 0ull}; }
    static __device__ __forceinline__ CA czero() { return CA{zero(), zero()}; }
    static __device__ __forceinline__ X prep(V v) { return X{v.hi, v.hi ^ 0x8000000080000000ull, v.lo}; }
    static __device__ __forceinline__ V add(V a, V b)
    {
        const float2 ah = f2_parts(a.hi), al = f2_parts(a.lo), bh = f2_parts(b.hi), bl = f2_parts(b.lo);
        const ff x = ff(ah.x, al.x) + ff(bh.x, bl.x), y = ff(ah.y, al.y) + ff(bh.y, bl.y);
        return V{f2_pack(x.hi, y.hi), f2_pack(x.lo, y.lo)};
    }
    static __device__ __forceinline__ V norm(V a)
    {
        const f2 h = f2_add(a.hi, a.lo);
        return V{h, f2_sub(a.lo, f2_sub(h, a.hi))};
    }
    static __device__ __forceinline__ CA norm(CA a) { return CA{norm(a.x), norm(a.y)}; }
    // a += h x: the product of the high parts as p + e exactly (TwoProd), a.hi + p as s + t exactly
    // (TwoSum); e, t and the cross products go to the low part, which norm() brings back under the
    // high one (FastTwoSum) after every product: a sum of n products is accurate to about n 2^-47 of
    // the sum of their magnitudes, the same form of bound as FP64 summation (n 2^-53).  A norm()
    // after every second product only measured 4 % faster and 10 % further from FP64; none until
    // the end, twice as far.
    static __device__ __forceinline__ void mac(V &a, S h, X x)
    {
        const f2 np = f2_mul(h.hi, x.nhi);  // -p
        const f2 e = f2_fma(h.hi, x.hi, np);
        const f2 s = f2_sub(a.hi, np), bb = f2_sub(s, a.hi), d = f2_sub(a.hi, f2_sub(s, bb));
        const f2 t = f2_sub(d, f2_add(np, bb));
        a.lo = f2_fma(h.hi, x.lo, a.lo);
        a.lo = f2_fma(h.lo, x.hi, a.lo);
        a.lo = f2_add(a.lo, f2_add(e, t));
        a.hi = s;
    }
    static __device__ __forceinline__ void cmac(CA &a, K c, X x)
    {
        mac(a.x, c.x, x);
        mac(a.y, c.y, x);
    }
    static __device__ __forceinline__ V times_i(V v)
    {
        const float2 h = f2_parts(v.hi), l = f2_parts(v.lo);
        return V{f2_pack(-h.y, h.x), f2_pack(-l.y, l.x)};
    }
    static __device__ __forceinline__ V value(V a) { return norm(a); }
    static __device__ __forceinline__ V value(CA a) { return add(norm(a.x), times_i(norm(a.y))); }
    static __device__ __forceinline__ V phase(E e, V x, V y)
    {
        V r = zero();
        mac(r, S{f2_pack(e.x, e.x), f2_pack(e.y, e.y)}, prep(x));
        mac(r, S{f2_pack(e.z, e.z), f2_pack(e.w, e.w)}, prep(times_i(y)));
        return norm(r);
    }
    static __device__ __forceinline__ E conj(E e) { return make_float4(e.x, e.y, -e.z, -e.w); }
};

// FP32 (deterministic mixed plans): the plain basis; every product and sum rounds in one fixed
// way, spelled out so that no compilation of it can contract them differently.
template <> struct Ops<float> {
    typedef float2 V;
    typedef float S;
    typedef float2 K;
    typedef float2 E, X, CA;
    static constexpr bool FOLD = false;
    static constexpr int NORM = 4;
    static constexpr int R = 4;
    static __device__ __forceinline__ V load(const V *p) { return *p; }
    static __device__ __forceinline__ void store(V *p, V v) { *p = v; }
    static __device__ __forceinline__ V zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ CA czero() { return zero(); }
    static __device__ __forceinline__ S table(const S *p) { return __ldg(p); }
    static __device__ __forceinline__ K table(const K *p) { return __ldg(p); }
    static __device__ __forceinline__ X prep(V v) { return v; }
    static __device__ __forceinline__ V add(V a, V b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
    static __device__ __forceinline__ void mac(V &a, S h, X x)
    {
        a.x = __fmaf_rn(h, x.x, a.x);
        a.y = __fmaf_rn(h, x.y, a.y);
    }
    // c x
    static __device__ __forceinline__ V mul(V c, V x)
    {
        return make_float2(__fmaf_rn(c.x, x.x, -__fmul_rn(c.y, x.y)), __fmaf_rn(c.y, x.x, __fmul_rn(c.x, x.y)));
    }
    // conj(e) x
    static __device__ __forceinline__ V cjmul(V e, V x)
    {
        return make_float2(__fmaf_rn(e.x, x.x, __fmul_rn(e.y, x.y)), __fmaf_rn(e.x, x.y, -__fmul_rn(e.y, x.x)));
    }
    static __device__ __forceinline__ void cmac(CA &a, K c, X x) { a = add(a, mul(c, x)); }
    static __device__ __forceinline__ V value(V a) { return a; }
    static __device__ __forceinline__ V norm(V a) { return a; }
};

// pair index q -> (n, m), 0 <= m <= n, q = n (n + 1) / 2 + m
__device__ __forceinline__ void pair_nm(int q, int &n, int &m)
{
    int k = (int)((sqrtf(8.f * q + 1.f) - 1.f) * 0.5f);
    while (k * (k + 1) / 2 > q) k--;
    while ((k + 1) * (k + 2) / 2 <= q) k++;
    n = k;
    m = q - k * (k + 1) / 2;
}

template <typename T> struct OwnArgs {
    typedef typename Ops<T>::V V;
    typedef typename Ops<T>::S S;
    typedef typename Ops<T>::K K;
    int p, nin, nq, pin, pout, pmax;  // RCR order; degrees used of the source and of the result
    int rows;                         // rows of each of the two shared-memory tiles
    const int4 *items;                // (rotation table row, first translation, count, coaxial block)
    const int *slot;                  // translations in class order -> slot
    const int *src;                   // per slot: source box and phase row
    const short *key;
    const S *rot;
    size_t rot_stride;
    const typename Ops<T>::E *ph;     // [row][m + pmax - 1]
    const K *Cc;
    const V *in;
    V *out;
    int slot0;                        // slot of out[0]
    const int *u1, *u2, *u3;          // work units of the three stages
    int n1, n2, n3;
};

// One rotation stage.  The rows of degree n are taken in groups of R rows of one sign (x+ or x-;
// FP32: any rows); unit = n | first group << 8, a lane takes one group of its column.
template <typename T, int TC>
__device__ __forceinline__ void rot_stage(const typename Ops<T>::S *__restrict__ rot, const typename Ops<T>::V *X,
                                          typename Ops<T>::V *Y, const int *__restrict__ units, int nu)
{
    typedef Ops<T> O;
    constexpr int R = O::R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int c = lane % TC, rl = lane / TC;
    for (int u = warp; u < nu; u += nw) {
        const int info = __ldg(units + u), n = info & 255, w = 2 * n + 1, r0 = n * n + n;
        const int np = O::FOLD ? (n + R) / R : (w + R - 1) / R, nm = O::FOLD ? (n + R - 1) / R : 0;
        const int g = min((info >> 8) + rl, np + nm - 1), minus = O::FOLD && g >= np;
        const int first = minus ? 1 + (g - np) * R : g * R;         // m' (FP32: row) of the first row
        const int last = O::FOLD ? n : w - 1;
        const int steps = O::FOLD ? n + 1 : w;
        const typename O::S *h = rot + (O::FOLD ? fold_off(n) : whole_off(n)) + (minus ? n : 0) + first;
        const int ld = O::FOLD ? w : pad4(w);
        auto rows = [](typename O::S(&v)[R], const typename O::S *p) {
            if constexpr (O::FOLD) {
#pragma unroll
                for (int k = 0; k < R; k++) v[k] = O::table(p + k);  // rows past the last read the next entry; their sums are dropped
            } else {
                static_assert(R == 4, "four rows a load");
                const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
                v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
            }
        };
        const typename O::V *x = X + (O::FOLD ? r0 : n * n) * TC + c;
        const int dx = minus ? -TC : TC;
        typename O::V acc[R];
        typename O::S hn[R];
#pragma unroll
        for (int k = 0; k < R; k++) acc[k] = O::zero();
        rows(hn, h);
#pragma unroll 4
        for (int m = 0; m < steps; m++) {
            typename O::S hc[R];
            if (m + 1 < steps) h += ld;  // the last step loads its own entries again
#pragma unroll
            for (int k = 0; k < R; k++) hc[k] = hn[k];
            rows(hn, h);
            const typename O::X xv = O::prep(O::load(x));
            x += dx;
#pragma unroll
            for (int k = 0; k < R; k++) {
                O::mac(acc[k], hc[k], xv);
                if ((m & (O::NORM - 1)) == O::NORM - 1) acc[k] = O::norm(acc[k]);
            }
        }
        if ((info >> 8) + rl < np + nm) {
#pragma unroll
            for (int k = 0; k < R; k++)
                if (first + k <= last) {
                    const int q = O::FOLD ? (minus ? r0 - first - k : r0 + first + k) : n * n + first + k;
                    O::store(Y + q * TC + c, O::value(acc[k]));
                }
        }
    }
}

// The coaxial stage: rows n' of +m then of -m in groups of R; unit = |m| | first group << 8.
template <typename T, int TC>
__device__ __forceinline__ void coax_stage(int p, int nin, int nq, const typename Ops<T>::K *__restrict__ Cc,
                                           const typename Ops<T>::V *X, typename Ops<T>::V *Y,
                                           const int *__restrict__ units, int nu)
{
    typedef Ops<T> O;
    constexpr int R = O::R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int c = lane % TC, rl = lane / TC;
    for (int u = warp; u < nu; u += nw) {
        const int info = __ldg(units + u), am = info & 255, sz = p - am, nrow = nq - am;
        const int np = (nrow + R - 1) / R, nm = am > 0 ? np : 0;
        const int g = min((info >> 8) + rl, np + nm - 1), minus = g >= np;
        const int first = (minus ? g - np : g) * R, sm = minus ? -am : am;
        const typename O::K *cb = Cc + coax_off(p, am) + first;
        const typename O::V *x = X + (am * am + am + sm) * TC + c;
        int dx = (2 * am + 2) * TC;
        typename O::CA acc[R];
        typename O::K cn[R];
#pragma unroll
        for (int k = 0; k < R; k++) {
            acc[k] = O::czero();
            cn[k] = O::table(cb + k);
        }
#pragma unroll 4
        for (int n = 0; n < nin - am; n++) {
            typename O::K cc[R];
            if (n + 1 < nin - am) cb += sz;
#pragma unroll
            for (int k = 0; k < R; k++) {
                cc[k] = cn[k];
                cn[k] = O::table(cb + k);
            }
            const typename O::X xv = O::prep(O::load(x));
            x += dx;
            dx += 2 * TC;
#pragma unroll
            for (int k = 0; k < R; k++) {
                O::cmac(acc[k], cc[k], xv);
                if ((n & (O::NORM - 1)) == O::NORM - 1) acc[k] = O::norm(acc[k]);
            }
        }
        if ((info >> 8) + rl < np + nm) {
#pragma unroll
            for (int k = 0; k < R; k++)
                if (first + k < nrow) {
                    const int nn = am + first + k;
                    O::store(Y + (nn * nn + nn + sm) * TC + c, O::value(acc[k]));
                }
        }
    }
}

template <typename T, int TC>
__global__ void __launch_bounds__(512, 1) own_tile_kernel(OwnArgs<T> a)
{
    typedef Ops<T> O;
    typedef typename O::V V;
    typedef typename O::E E;
    constexpr int GI = 32 / TC;  // gather / scatter: TC columns x GI pairs (n, m >= 0) per warp
    extern __shared__ double2 own_smem[];
    __shared__ int s_src[TC], s_key[TC], s_out[TC];
    V *X = reinterpret_cast<V *>(own_smem), *W = X + (size_t)a.rows * TC;
    const int4 it = a.items[blockIdx.x];
    const int cnt = it.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (threadIdx.x < TC) {
        const int s = a.slot[it.y + min((int)threadIdx.x, cnt - 1)];
        s_src[threadIdx.x] = a.src[s];
        s_key[threadIdx.x] = a.key[s];
        s_out[threadIdx.x] = s - a.slot0;
    }
    __syncthreads();
    const int c = lane % TC, gi = lane / TC, w = 2 * a.pmax - 1, off = a.pmax - 1;
    const E *ph = a.ph + (size_t)s_key[c] * w + off;
    // gather with the phases e^{i m phi}
    {
        const int np = a.nin * (a.nin + 1) / 2;
        const V *src = a.in + (size_t)s_src[c] * a.pin * a.pin;
        for (int q = warp * GI + gi; q < np; q += nw * GI) {
            int n, m;
            pair_nm(q, n, m);
            const int r0 = n * n + n;
            V xp = O::zero(), xm = xp;
            if (c < cnt) {
                const V *in = src + r0;
                xp = O::load(in + m);
                if constexpr (O::FOLD) {
                    if (m > 0) {
                        const V vp = xp, vm = O::load(in - m);
                        const E e = __ldg(ph + m);
                        xp = O::phase(e, vp, vm);
                        xm = O::phase(e, vm, vp);
                    }
                } else {
                    xp = O::mul(xp, __ldg(ph + m));
                    if (m > 0) xm = O::mul(O::load(in - m), __ldg(ph - m));
                }
            }
            O::store(X + (r0 + m) * TC + c, xp);
            if (m > 0) O::store(X + (r0 - m) * TC + c, xm);
        }
    }
    __syncthreads();
    const typename O::S *rot = a.rot + (size_t)it.x * a.rot_stride;
    rot_stage<T, TC>(rot, X, W, a.u1, a.n1);
    __syncthreads();
    coax_stage<T, TC>(a.p, a.nin, a.nq, a.Cc + (size_t)it.w * coax_size(a.p), W, X, a.u2, a.n2);
    __syncthreads();
    rot_stage<T, TC>(rot, X, W, a.u3, a.n3);
    __syncthreads();
    // results with the phases e^{-i m phi}
    if (c < cnt) {
        const int np = a.nq * (a.nq + 1) / 2;
        V *dst = a.out + (size_t)s_out[c] * a.pout * a.pout;
        for (int q = warp * GI + gi; q < np; q += nw * GI) {
            int n, m;
            pair_nm(q, n, m);
            const int r0 = n * n + n;
            V *out = dst + r0;
            const V yp = O::load(W + (r0 + m) * TC + c);
            if constexpr (O::FOLD) {
                if (m > 0) {
                    const V ym = O::load(W + (r0 - m) * TC + c);
                    const E e = O::conj(__ldg(ph + m));
                    O::store(out + m, O::phase(e, yp, ym));
                    O::store(out - m, O::phase(e, ym, yp));
                } else {
                    O::store(out, yp);
                }
            } else {
                O::store(out + m, O::cjmul(__ldg(ph + m), yp));
                if (m > 0) O::store(out - m, O::cjmul(__ldg(ph - m), O::load(W + (r0 - m) * TC + c)));
            }
        }
    }
}

// Dst[b] = (add ? Dst[b] : 0) + the slots beg[b] .. beg[b+1]-1 of part (slot s at s - slot0), n2
// entries each, in order; with S > 1 in S runs whose sums are added in order
template <typename T>
__global__ void own_reduce_kernel(int b0, int b1, int n2, int S, int add, int slot0, const int *__restrict__ beg,
                                  const typename Ops<T>::V *__restrict__ part, typename Ops<T>::V *__restrict__ Dst)
{
    typedef Ops<T> O;
    const size_t n = (size_t)(b1 - b0) * n2;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
        const int b = b0 + (int)(t / n2), i = (int)(t % n2), s0 = beg[b], ns = beg[b + 1] - s0;
        const typename O::V *q = part + (size_t)(s0 - slot0) * n2 + i;
        typename O::V *d = Dst + (size_t)b * n2 + i, tot = O::zero();
        for (int c = 0; c < S; c++) {
            const int sa = (int)((long long)ns * c / S), sb = (int)((long long)ns * (c + 1) / S);
            typename O::V acc = c == 0 && add ? O::load(d) : O::zero();
#pragma unroll 4
            for (int s = sa; s < sb; s++) acc = O::add(acc, O::load(q + (size_t)s * n2));
            tot = c == 0 ? acc : O::add(tot, acc);
        }
        O::store(d, tot);
    }
}

// in place: plain -> x+/x- (fwd), or back
__global__ void own_fold_kernel(double2 *x, size_t nb, int p, int fwd)
{
    const int np = p * (p + 1) / 2;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nb * np; t += (size_t)gridDim.x * blockDim.x) {
        int n, m;
        pair_nm((int)(t % np), n, m);
        if (m == 0) continue;
        double2 *q = x + (t / np) * (size_t)p * p + n * n + n;
        const double2 a = q[m], b = q[-m];
        const double f = fwd ? 1.0 : 0.5;
        q[m] = make_double2(f * (a.x + b.x), f * (a.y + b.y));
        q[-m] = make_double2(f * (a.x - b.x), f * (a.y - b.y));
    }
}

// FP64 plain -> float-float x+/x- (times ds[n] where given), and back
__global__ void own_fold_ff_kernel(const double2 *__restrict__ in, ffv *__restrict__ out, size_t nb, int p,
                                   const double *__restrict__ ds)
{
    const int np = p * (p + 1) / 2;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nb * np; t += (size_t)gridDim.x * blockDim.x) {
        int n, m;
        pair_nm((int)(t % np), n, m);
        const size_t base = (t / np) * (size_t)p * p + n * n + n;
        const double f = ds ? ds[n] : 1.0;
        auto put = [&](size_t i, double re, double im) {
            const ff a = ff_from(re * f), b = ff_from(im * f);
            Ops<ff>::store(out + i, ffv{f2_pack(a.hi, b.hi), f2_pack(a.lo, b.lo)});
        };
        const double2 a = in[base + m];
        if (m == 0) {
            put(base, a.x, a.y);
        } else {
            const double2 b = in[base - m];
            put(base + m, a.x + b.x, a.y + b.y);
            put(base - m, a.x - b.x, a.y - b.y);
        }
    }
}
__global__ void own_unfold_ff_kernel(const ffv *__restrict__ in, double2 *__restrict__ out, size_t nb, int p,
                                     const double *__restrict__ ds)
{
    const int np = p * (p + 1) / 2;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nb * np; t += (size_t)gridDim.x * blockDim.x) {
        int n, m;
        pair_nm((int)(t % np), n, m);
        const size_t base = (t / np) * (size_t)p * p + n * n + n;
        const double f = (ds ? ds[n] : 1.0) * (m ? 0.5 : 1.0);
        auto get = [&](size_t i) {
            const ffv v = Ops<ff>::load(in + i);
            const float2 h = f2_parts(v.hi), l = f2_parts(v.lo);
            return make_double2((double)h.x + (double)l.x, (double)h.y + (double)l.y);
        };
        const double2 a = get(base + m);
        if (m == 0) {
            out[base] = make_double2(f * a.x, f * a.y);
        } else {
            const double2 b = get(base - m);
            out[base + m] = make_double2(f * (a.x + b.x), f * (a.y + b.y));
            out[base - m] = make_double2(f * (a.x - b.x), f * (a.y - b.y));
        }
    }
}

// folded rotation tables of the classes' representative rows rep[k] of H (see fold_off)
__global__ void own_fold_table_kernel(int pmax, const int *__restrict__ rep, const double *__restrict__ H,
                                      double *__restrict__ o64, ffs *__restrict__ off2)
{
    const int n = blockIdx.x, k = blockIdx.y, w = 2 * n + 1;
    const double *Hn = H + (size_t)rep[k] * rot_size(pmax) + rot_off(n);
    const size_t base = (size_t)k * fold_size(pmax) + fold_off(n);
    for (int t = threadIdx.x; t < (n + 1) * w; t += blockDim.x) {
        const int m = t / w, j = t % w, mp = j <= n ? j : j - n;
        const double a = Hn[(n + m) * w + n + mp], b = Hn[(n - m) * w + n + mp];
        double v;
        if (j > n)
            v = m ? a - b : 0.0;
        else if (m)
            v = mp ? a + b : 0.5 * (a + b);
        else
            v = mp ? a + Hn[n * w + n - mp] : a;
        if (o64) o64[base + t] = v;
        if (off2) {
            const ff f = ff_from(v);
            off2[base + t] = ffs{f2_pack(f.hi, f.hi), f2_pack(f.lo, f.lo)};
        }
    }
}

// ---- lists
// per slot of M2M (children in the parents' order) and L2L (boxes): source box and phase row
__global__ void own_m2m_slots_kernel(int nb, const int *child_list, const unsigned char *octant, int *src, short *key)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nb; s += gridDim.x * blockDim.x) {
        src[s] = child_list[s];
        key[s] = (short)(NDIR + octant[child_list[s]]);
    }
}
__global__ void own_l2l_slots_kernel(int nb, const unsigned char *octant, short *key)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nb; s += gridDim.x * blockDim.x)
        key[s] = (short)(NDIR + 8 + octant[s]);
}
// class order: bin (chunk of the slot) * ncls + class; counts (list null), then positions
__global__ void own_bin_kernel(int n, const short *__restrict__ key, const int *__restrict__ cls_of_key,
                               const int *__restrict__ chunk_slot, int nchunk, int ncls, int *bins, int *list)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        int c = 0;
        while (c + 1 < nchunk && s >= chunk_slot[c + 1]) c++;
        const int pos = atomicAdd(bins + c * ncls + cls_of_key[key[s]], 1);
        if (list) list[pos] = s;
    }
}

unsigned ew_grid(size_t n) { return (unsigned)std::max<size_t>(1, std::min<size_t>((n + 255) / 256, 152 * 16)); }

// Columns of a tile: two tiles of `rows` rows in shared memory, at most TWO_CTA bytes where two
// CTAs (of 256 threads) are to share an SM, so that one computes while the other gathers or waits
// at a barrier; else one CTA of 512 threads.  Most columns first: a table entry then serves more
// multiply-adds (M2L of the head in float-float, 8 / 16 / 32 columns: p = 8 8.2 / 6.8 / 5.9 ms,
// p = 10 4.0 / 3.3 / 3.1); where only 8 columns leave room for two CTAs (p = 20) 16 columns in one
// CTA measured the same (FP64 5.08 against 5.02 ms), and 4 columns in one of two CTAs as 8 in one
// (p = 30: 3.86 against 3.91).  FP32 tiles stop at 76 KB: their tables, four rows a load, then keep room in
// L1 (a deterministic matvec on 20,480 triangles 1.20 -> 1.15 ms; 40 KB: 1.25; float-float 15.05 with
// TWO_CTA, 15.38 with 76 KB).
constexpr size_t TWO_CTA = 112 * 1024 + 512, ONE_CTA = 226 * 1024, F32_TILE = 76 * 1024;

int pick_cols(int rows, size_t elem, size_t most)
{
    for (int tc : {32, 16, 8})
        if (2 * elem * rows * tc <= most) return tc;
    for (int tc : {8, 4, 2})
        if (2 * elem * rows * tc <= ONE_CTA) return tc;
    return 0;
}

// bytes of the scratch that holds one chunk of translated expansions
constexpr size_t PART_CAP = 128u << 20;

// ---- scratch, shared by the plans of a device.  A plan takes a buffer while it enqueues its translations and gives it
// back with an event behind them: the next plan to take it waits for that event on its own stream (or finds it
// passed).  A plan prefers the buffer that it used last, if no other has since: its own stream orders that (24 spheres
// solved in FP64 on 4 threads: 53.4 ms; 65.4 with a buffer by its number, the same one for many plans).  Buffers are
// added while they stay under POOL_CAP in all, so that plans on several streams run side by side; the last plan of the
// device to go frees them.  (128 MB in each plan for its life: 256 bodies of a scene would have held 32 GB.)
constexpr size_t POOL_CAP = 512u << 20, SMALL_PART = 16u << 20;
struct Scratch {
    void *ptr = nullptr;
    size_t bytes = 0;
    cudaEvent_t done = nullptr;
    const Plan *owner = nullptr;  // who used it last (null: gone)
    bool busy = false;
};
struct Pool {
    std::vector<Scratch> buf;
    int users = 0;
};
std::mutex pool_mutex;
std::condition_variable pool_free;
std::map<int, Pool> pools;  // per device

int pool_take(Plan *P, size_t bytes, void **ptr)
{
    std::unique_lock<std::mutex> lock(pool_mutex);
    Pool &pool = pools[P->opt.device];
    if (P->own_scratch == Plan::NO_POOL) {
        pool.users++;
        P->own_scratch = Plan::NO_SCRATCH;
    }
    for (;;) {
        int mine = -1, idle = -1, behind = -1, small = -1, room = -1;
        size_t all = 0;
        bool busy = false;
        for (int i = 0; i < (int)pool.buf.size(); i++) {
            Scratch &s = pool.buf[i];
            all += s.bytes;
            if (!s.ptr) {
                if (!s.busy) room = i;
                continue;
            }
            busy = busy || s.busy;
            if (s.busy) continue;
            if (s.bytes < bytes) {
                small = i;
            } else if (s.owner == P) {
                mine = i;
            } else if (cudaEventQuery(s.done) == cudaSuccess) {
                idle = i;
            } else {
                cudaGetLastError();
                behind = i;
            }
        }
        int take = mine >= 0 ? mine : idle;
        if (take < 0 && all > 0 && all + bytes > POOL_CAP) {
            take = behind;
            if (take < 0 && small >= 0) {  // none is large enough: a free one gives way
                Scratch &s = pool.buf[small];
                FMM_CUDA_TRY(cudaEventSynchronize(s.done));
                cudaFree(s.ptr);
                s = Scratch{nullptr, 0, s.done};
                continue;
            }
            if (take < 0 && busy) {  // all are being handed to kernels by other threads
                pool_free.wait(lock);
                continue;
            }
        }
        if (take < 0) {
            if (room < 0) {
                pool.buf.emplace_back();
                room = (int)pool.buf.size() - 1;
            }
            Scratch &s = pool.buf[room];
            if (!s.done) FMM_CUDA_TRY(cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming));
            const cudaError_t ce = cudaMalloc(&s.ptr, bytes);
            if (ce != cudaSuccess && behind < 0) {
                s.ptr = nullptr;
                FMM_CUDA_TRY(ce);
            }
            if (ce == cudaSuccess) {
                s.bytes = bytes;
                take = room;
            } else {  // no memory for another one
                cudaGetLastError();
                s.ptr = nullptr;
                take = behind;
            }
        }
        Scratch &s = pool.buf[take];
        if (s.owner != P) FMM_CUDA_TRY(cudaStreamWaitEvent(P->stream, s.done, 0));
        s.busy = true;
        s.owner = P;
        P->own_scratch = take;
        *ptr = s.ptr;
        return FMM_OK;
    }
}

int pool_give(Plan *P)
{
    std::lock_guard<std::mutex> lock(pool_mutex);
    Scratch &s = pools[P->opt.device].buf[P->own_scratch];
    s.busy = false;
    pool_free.notify_all();
    FMM_CUDA_TRY(cudaEventRecord(s.done, P->stream));
    return FMM_OK;
}

void pool_leave(Plan *P)
{
    if (P->own_scratch == Plan::NO_POOL) return;
    std::lock_guard<std::mutex> lock(pool_mutex);
    Pool &pool = pools[P->opt.device];
    P->own_scratch = Plan::NO_POOL;
    pool.users--;
    for (Scratch &s : pool.buf)
        if (s.owner == P) s.owner = nullptr;
    if (pool.users > 0) return;
    for (Scratch &s : pool.buf) {
        cudaFree(s.ptr);
        if (s.done) cudaEventDestroy(s.done);
    }
    pool.buf.clear();
}

template <typename T, int TC>
int launch_tc(const OwnArgs<T> &a, int n_items, cudaStream_t st)
{
    static size_t attr = 0;
    const size_t sm = 2 * sizeof(typename Ops<T>::V) * (size_t)a.rows * TC;
    int e = raise_smem_limit((const void *)own_tile_kernel<T, TC>, sm, &attr);
    if (e) return e;
    own_tile_kernel<T, TC><<<n_items, sm > TWO_CTA ? 512 : 256, sm, st>>>(a);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

// device memory that is freed unless keep() takes it
struct DevMem {
    void *ptr = nullptr;
    ~DevMem() { cudaFree(ptr); }
    template <class Q> Q *keep()
    {
        Q *q = (Q *)ptr;
        ptr = nullptr;
        return q;
    }
};

const int WHICH[3] = {PASS_M2M, PASS_M2L, PASS_L2L};
int key_base(int which) { return which == PASS_M2L ? 0 : which == PASS_M2M ? NDIR : NDIR + 8; }
int slot_bytes(int wide) { return wide ? 16 : 8; }

// The lists of every pass for coefficients of 16 bytes (wide) or 8, on the plan's stream: one allocation, one
// count of all passes' (chunk, class) bins with one read-back (pass by pass, with four synchronizations each, the
// first FP64 matvec on 320 triangles took 0.57 ms where later ones take 0.17).
int build_lists(Plan *P, int wide)
{
    OwnLists &lists = P->own_lists[wide ? 0 : 1];
    if (lists.ready) return FMM_OK;
    cudaStream_t st = P->stream;
    OwnLists L;
    std::vector<OwnPass *> passes;
    std::vector<int> where;  // level * 3 + which
    for (int l = P->lmin; l <= P->lmax; l++)
        for (int which : WHICH) {
            if (which != PASS_M2L && l == P->lmin) continue;
            const LevelDev &D = P->lev[l];
            OwnPass &O = L.pass[l][which];
            O.p = which == PASS_M2L ? D.p : P->lev[l - 1].p;
            O.pin = which == PASS_M2M ? D.p : O.p;
            O.pout = which == PASS_L2L ? D.p : O.p;
            O.rows = std::max(std::min(O.pin, O.p), std::min(O.pout, O.p));
            O.rows *= O.rows;
            O.n = which == PASS_M2L ? (int)D.num_sr : D.nb;
            O.ndst = which == PASS_M2M ? P->lev[l - 1].nb : D.nb;
            O.beg = which == PASS_M2L ? D.sr_beg : which == PASS_M2M ? P->lev[l - 1].child_beg : nullptr;
            passes.push_back(&O);
            where.push_back(3 * l + which);
        }
    // chunks of destinations whose results fit the scratch
    const int np = (int)passes.size();
    std::vector<std::vector<int>> beg(np);
    bool wait = false;
    for (int k = 0; k < np; k++) {
        OwnPass &O = *passes[k];
        const size_t cap = std::max<size_t>(1, PART_CAP / ((size_t)slot_bytes(wide) * O.pout * O.pout));
        if (!O.beg || (size_t)O.n <= cap) continue;
        beg[k].resize(O.ndst + 1);
        FMM_CUDA_TRY(cudaMemcpyAsync(beg[k].data(), O.beg, sizeof(int) * (O.ndst + 1), cudaMemcpyDeviceToHost, st));
        wait = true;
    }
    if (wait) FMM_CUDA_TRY(cudaStreamSynchronize(st));
    size_t ints = 0;
    std::vector<int> host(NDIR + 16, 0);  // class of each key, then the passes' chunk beginnings, then their bins
    std::vector<size_t> at_slot(np), at_src(np), at_key(np), at_chunk(np), at_bin(np);
    auto take = [&](size_t n) {
        const size_t at = ints;
        ints += (n + 3) & ~(size_t)3;
        return at;
    };
    size_t nbin = 0;
    for (int k = 0; k < np; k++) {
        OwnPass &O = *passes[k];
        const int which = where[k] % 3, cap = (int)std::max<size_t>(1, std::min<size_t>(1u << 30, PART_CAP / ((size_t)slot_bytes(wide) * O.pout * O.pout)));
        O.chunk_box.assign(1, 0);
        O.chunk_slot.assign(1, 0);
        if (beg[k].empty()) {
            O.chunk_box.push_back(O.ndst);
            O.chunk_slot.push_back(O.n);
        } else {
            for (int b = 0; b < O.ndst;) {
                int e = b + 1;
                while (e < O.ndst && beg[k][e + 1] - beg[k][b] <= cap) e++;
                O.chunk_box.push_back(e);
                O.chunk_slot.push_back(beg[k][e]);
                b = e;
            }
        }
        std::vector<int> cls;
        direction_classes(P, which, which == PASS_M2L ? NDIR : 8, cls, O.rep);
        for (size_t d = 0; d < cls.size(); d++) host[key_base(which) + d] = cls[d];
        O.bins.assign((O.chunk_slot.size() - 1) * O.rep.size(), 0);
        nbin += O.bins.size();
        at_slot[k] = take(O.n);
        if (which == PASS_M2M) at_src[k] = take(O.n);
        if (which != PASS_M2L) at_key[k] = take((O.n + 1) / 2);
    }
    for (int k = 0; k < np; k++) {
        at_chunk[k] = host.size();
        host.insert(host.end(), passes[k]->chunk_slot.begin(), passes[k]->chunk_slot.end());
    }
    const size_t bins0 = host.size();
    host.resize(bins0 + nbin, 0);
    DevMem mem, tmp;
    FMM_CUDA_TRY(cudaMalloc(&mem.ptr, sizeof(int) * std::max<size_t>(1, ints)));
    FMM_CUDA_TRY(cudaMalloc(&tmp.ptr, sizeof(int) * host.size()));
    int *m = (int *)mem.ptr, *t = (int *)tmp.ptr;
    FMM_CUDA_TRY(cudaMemcpyAsync(t, host.data(), sizeof(int) * host.size(), cudaMemcpyHostToDevice, st));
    size_t bin = bins0;
    for (int k = 0; k < np; k++) {
        OwnPass &O = *passes[k];
        const int which = where[k] % 3, l = where[k] / 3;
        const LevelDev &D = P->lev[l];
        O.slot = m + at_slot[k];
        if (which == PASS_M2L) {
            O.src = D.sr_src;
            O.key = D.sr_dir;
        } else {
            O.key = O.key_own = (short *)(m + at_key[k]);
            if (which == PASS_M2M) {
                O.src = O.src_own = m + at_src[k];
                own_m2m_slots_kernel<<<ew_grid(D.nb), 256, 0, st>>>(D.nb, P->lev[l - 1].child_list, D.octant, O.src_own, O.key_own);
            } else {
                O.src = D.parent;
                own_l2l_slots_kernel<<<ew_grid(D.nb), 256, 0, st>>>(D.nb, D.octant, O.key_own);
            }
        }
        at_bin[k] = bin;
        bin += O.bins.size();
        own_bin_kernel<<<ew_grid(O.n), 256, 0, st>>>(O.n, O.key, t, t + at_chunk[k], (int)O.chunk_slot.size() - 1, (int)O.rep.size(),
                                                     t + at_bin[k], nullptr);
    }
    FMM_CUDA_TRY(cudaGetLastError());
    FMM_CUDA_TRY(cudaMemcpyAsync(host.data() + bins0, t + bins0, sizeof(int) * nbin, cudaMemcpyDeviceToHost, st));
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
    for (int k = 0; k < np; k++) {
        OwnPass &O = *passes[k];
        int pos = 0;
        for (size_t q = 0; q < O.bins.size(); q++) {
            O.bins[q] = host[at_bin[k] + q];
            host[at_bin[k] + q] = pos;
            pos += O.bins[q];
        }
    }
    FMM_CUDA_TRY(cudaMemcpyAsync(t + bins0, host.data() + bins0, sizeof(int) * nbin, cudaMemcpyHostToDevice, st));
    for (int k = 0; k < np; k++) {
        OwnPass &O = *passes[k];
        own_bin_kernel<<<ew_grid(O.n), 256, 0, st>>>(O.n, O.key, t, t + at_chunk[k], (int)O.chunk_slot.size() - 1, (int)O.rep.size(),
                                                     t + at_bin[k], O.slot);
    }
    FMM_CUDA_TRY(cudaGetLastError());
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
    L.mem = mem.keep<int>();
    L.ready = 1;
    P->device_bytes += sizeof(int) * ints;
    lists = L;
    return FMM_OK;
}

// Tile shapes, items and work units of every pass of one type, in one allocation.
template <typename T>
int build_form(Plan *P, OwnForm &form)
{
    if (form.ready) return FMM_OK;
    typedef typename Ops<T>::V C;
    const bool wide = sizeof(C) == 16;
    const OwnLists &lists = P->own_lists[wide ? 0 : 1];
    OwnForm F;
    std::vector<int4> items;
    std::vector<int> un;
    std::vector<std::pair<size_t, size_t>> at;  // the passes' first item and unit
    const int rows_m2l = (int)lists.pass[P->lmin][PASS_M2L].rep.size();
    for (int l = P->lmin; l <= P->lmax; l++)
        for (int which : WHICH) {
            if (which != PASS_M2L && l == P->lmin) continue;
            const OwnPass &O = lists.pass[l][which];
            OwnTiles &W = F.pass[l][which];
            W.tc = pick_cols(O.rows, sizeof(C), std::is_same<T, float>::value ? F32_TILE : TWO_CTA);
            if (!W.tc) {
                fmm_set_error("translation order %d above 60", O.p);
                return FMM_ERR_CUDA;
            }
            at.push_back({items.size(), un.size()});
            const size_t item0 = items.size(), ncls = O.rep.size();
            const int row0 = which == PASS_M2L ? 0 : rows_m2l + (which == PASS_M2M ? 0 : 2);
            W.chunk_item.assign(1, 0);
            int pos = 0;
            for (size_t q = 0; q < O.bins.size(); q++) {
                const int k = (int)(q % ncls), cnt = O.bins[q];
                for (int a = 0; a < cnt; a += W.tc)
                    items.push_back(make_int4(row0 + k, pos + a, std::min(W.tc, cnt - a), which == PASS_M2L ? P->dir_dist[O.rep[k]] : 0));
                pos += cnt;
                if (k + 1 == (int)ncls) W.chunk_item.push_back((int)(items.size() - item0));
            }
            if (which != PASS_L2L)
                for (size_t c = 0; c + 1 < O.chunk_slot.size(); c++)
                    F.part_bytes = std::max(F.part_bytes, sizeof(C) * (size_t)(O.chunk_slot[c + 1] - O.chunk_slot[c]) * O.pout * O.pout);
            // work units, longest first: groups of R rows of one sign, 32 / tc groups each
            const int nin = std::min(O.pin, O.p), nq = std::min(O.pout, O.p), rl = 32 / W.tc, R = Ops<T>::R;
            auto rot_units = [&](int deg) {
                int k = 0;
                for (int d = deg - 1; d >= 0; d--) {
                    const int ng = Ops<T>::FOLD ? (d + R) / R + (d + R - 1) / R : (2 * d + R) / R;
                    for (int g = 0; g < ng; g += rl, k++) un.push_back(d | g << 8);
                }
                return k;
            };
            W.n1 = rot_units(nin);
            // orders m that the source does not reach (nq > nin) give rows of zeros
            for (int am = 0; am < nq; am++) {
                const int ng = (am ? 2 : 1) * ((nq - am + R - 1) / R);
                for (int g = 0; g < ng; g += rl, W.n2++) un.push_back(am | g << 8);
            }
            W.n3 = rot_units(nq);
        }
    DevMem mem;
    const size_t bytes = sizeof(int4) * items.size() + sizeof(int) * un.size();
    FMM_CUDA_TRY(cudaMalloc(&mem.ptr, std::max<size_t>(1, bytes)));
    int4 *it = (int4 *)mem.ptr;
    int *u = (int *)(it + items.size());
    FMM_CUDA_TRY(cudaMemcpyAsync(it, items.data(), sizeof(int4) * items.size(), cudaMemcpyHostToDevice, P->stream));
    FMM_CUDA_TRY(cudaMemcpyAsync(u, un.data(), sizeof(int) * un.size(), cudaMemcpyHostToDevice, P->stream));
    FMM_CUDA_TRY(cudaStreamSynchronize(P->stream));
    size_t k = 0;
    for (int l = P->lmin; l <= P->lmax; l++)
        for (int which : WHICH) {
            if (which != PASS_M2L && l == P->lmin) continue;
            F.pass[l][which].items = it + at[k].first;
            F.pass[l][which].units = u + at[k++].second;
        }
    F.mem = mem.keep<int4>();
    F.ready = 1;
    P->device_bytes += bytes;
    form = F;
    return FMM_OK;
}

// folded rotation tables of the classes (M2L, then M2M and L2L)
int build_folded(Plan *P, bool ff)
{
    if (ff ? (void *)P->own_rot_ff : (void *)P->own_rot64) return FMM_OK;
    std::vector<int> reps, cls, rep;
    for (int which : {PASS_M2L, PASS_M2M, PASS_L2L}) {
        direction_classes(P, which, which == PASS_M2L ? NDIR : 8, cls, rep);
        for (int r : rep) reps.push_back(key_base(which) + r);
    }
    const size_t bytes = (ff ? sizeof(ffs) : sizeof(double)) * (reps.size() * (size_t)fold_size(P->pmax) + TABLE_PAD);
    DevMem tab, d_rep;
    FMM_CUDA_TRY(cudaMalloc(&tab.ptr, bytes));
    FMM_CUDA_TRY(cudaMalloc(&d_rep.ptr, sizeof(int) * reps.size()));
    FMM_CUDA_TRY(cudaMemcpyAsync(d_rep.ptr, reps.data(), sizeof(int) * reps.size(), cudaMemcpyHostToDevice, P->stream));
    own_fold_table_kernel<<<dim3(P->pmax, (unsigned)reps.size()), 128, 0, P->stream>>>(
        P->pmax, (const int *)d_rep.ptr, P->Hsr64, ff ? nullptr : (double *)tab.ptr, ff ? (ffs *)tab.ptr : nullptr);
    FMM_CUDA_TRY(cudaGetLastError());
    FMM_CUDA_TRY(cudaStreamSynchronize(P->stream));
    if (ff)
        P->own_rot_ff = tab.keep<float4>();
    else
        P->own_rot64 = tab.keep<double>();
    P->device_bytes += bytes;
    return FMM_OK;
}

template <typename T> int tables_of(Plan *P, OwnArgs<T> &a);
template <> int tables_of<double>(Plan *P, OwnArgs<double> &a)
{
    a.rot = P->own_rot64;
    a.rot_stride = fold_size(P->pmax);
    a.ph = P->PHsr64;
    return FMM_OK;
}
template <> int tables_of<ff>(Plan *P, OwnArgs<ff> &a)
{
    a.rot = reinterpret_cast<const ffs *>(P->own_rot_ff);
    a.rot_stride = fold_size(P->pmax);
    a.ph = P->PHall_ff;
    return FMM_OK;
}
template <> int tables_of<float>(Plan *P, OwnArgs<float> &a)
{
    a.rot = P->rot32_whole;
    a.rot_stride = whole_off(P->pmax);
    a.ph = P->PHsr32;
    return FMM_OK;
}

template <typename T> struct LevelArrays {
    typename Ops<T>::V *Cm, *Dl;
    const typename Ops<T>::K *Csr, *Cup, *Cdown;
};
template <typename T> LevelArrays<T> arrays_of(LevelDev &L);
template <> LevelArrays<double> arrays_of<double>(LevelDev &L) { return {L.Cm64, L.Dl64, L.Csr64, L.Crr64, L.Crr64}; }
template <> LevelArrays<float> arrays_of<float>(LevelDev &L)
{
    return {L.Cm32, L.Dl32, L.Csr32, L.Crr32, L.Crr32L ? L.Crr32L : L.Crr32};
}
template <> LevelArrays<ff> arrays_of<ff>(LevelDev &L)
{
    return {reinterpret_cast<ffv *>(L.Cm_ff), reinterpret_cast<ffv *>(L.Dl_ff), reinterpret_cast<const ffk *>(L.Csr_ff),
            reinterpret_cast<const ffk *>(L.Crr_ff), reinterpret_cast<const ffk *>(L.CrrL_ff ? L.CrrL_ff : L.Crr_ff)};
}

template <typename T>
int run_pass(Plan *P, int l, int which, const OwnPass &O, const OwnTiles &W, void *part)
{
    typedef typename Ops<T>::V C;
    cudaStream_t st = P->stream;
    LevelDev &L = P->lev[l];
    LevelArrays<T> A = arrays_of<T>(L), U = l > P->lmin ? arrays_of<T>(P->lev[l - 1]) : A;
    OwnArgs<T> a;
    int e = tables_of<T>(P, a);
    if (e) return e;
    a.p = O.p;
    a.pin = O.pin;
    a.pout = O.pout;
    a.nin = std::min(O.pin, O.p);
    a.nq = std::min(O.pout, O.p);
    a.pmax = P->pmax;
    a.rows = O.rows;
    a.slot = O.slot;
    a.src = O.src;
    a.key = O.key;
    a.Cc = which == PASS_M2L ? A.Csr : which == PASS_M2M ? A.Cup : A.Cdown;
    a.in = which == PASS_L2L ? U.Dl : A.Cm;
    a.u1 = W.units;
    a.u2 = W.units + W.n1;
    a.u3 = W.units + W.n1 + W.n2;
    a.n1 = W.n1;
    a.n2 = W.n2;
    a.n3 = W.n3;
    C *dst = which == PASS_M2M ? U.Cm : A.Dl;
    const int n2 = O.pout * O.pout;
    // a parent of lower order than the child reaches the child's first degrees only
    if (which == PASS_L2L && a.nq < O.pout)
        FMM_CUDA_TRY(cudaMemsetAsync(dst, 0, sizeof(C) * (size_t)L.nb * n2, st));
    for (size_t c = 0; c + 1 < O.chunk_box.size(); c++) {
        const int n = W.chunk_item[c + 1] - W.chunk_item[c];
        a.items = W.items + W.chunk_item[c];
        a.slot0 = O.chunk_slot[c];
        a.out = which == PASS_L2L ? dst : (C *)part;
        if (n > 0) {
            switch (W.tc) {
            case 32: e = launch_tc<T, 32>(a, n, st); break;
            case 16: e = launch_tc<T, 16>(a, n, st); break;
            case 8: e = launch_tc<T, 8>(a, n, st); break;
            case 4: e = launch_tc<T, 4>(a, n, st); break;
            default: e = launch_tc<T, 2>(a, n, st); break;
            }
            if (e) return e;
        }
        if (which != PASS_L2L) {
            const int b0 = O.chunk_box[c], b1 = O.chunk_box[c + 1];
            const int S = which == PASS_M2L ? std::max(1, L.m2l_split) : 1;
            own_reduce_kernel<T><<<ew_grid((size_t)(b1 - b0) * n2), 256, 0, st>>>(
                b0, b1, n2, S, which == PASS_M2L && l > P->lmin, a.slot0, O.beg, (const C *)part, dst);
            FMM_CUDA_TRY(cudaGetLastError());
        }
    }
    return FMM_OK;
}

template <typename T> int type_of() { return std::is_same<T, double>::value ? OWN_FP64 : std::is_same<T, ff>::value ? OWN_FF : OWN_FP32; }

// lists, tiles and tables of a type
template <typename T>
int ensure_own(Plan *P)
{
    OwnForm &form = P->own_form[type_of<T>()];
    int e = build_lists(P, sizeof(typename Ops<T>::V) == 16);
    if (!e) e = std::is_same<T, float>::value ? ensure_whole_tables(P) : build_folded(P, std::is_same<T, ff>::value);
    if (!e) e = build_form<T>(P, form);
    return e;
}

template <typename T>
int translate(Plan *P, void (*beg)(Plan *, int, int), void (*end)(Plan *))
{
    int e = ensure_own<T>(P);
    if (e) return e;
    const OwnLists &lists = P->own_lists[sizeof(typename Ops<T>::V) == 16 ? 0 : 1];
    const OwnForm &form = P->own_form[type_of<T>()];
    LevelDev &LL = P->lev[P->lmax];
    cudaStream_t st = P->stream;
    void *part = nullptr;
    if (form.part_bytes && (e = pool_take(P, form.part_bytes, &part))) return e;
    auto pass = [&](int l, int which) { return run_pass<T>(P, l, which, lists.pass[l][which], form.pass[l][which], part); };
    const size_t np = (size_t)LL.nb * LL.p * (LL.p + 1) / 2;
    if (std::is_same<T, double>::value)
        own_fold_kernel<<<ew_grid(np), 256, 0, st>>>(LL.Cm64, LL.nb, LL.p, 1);
    else if (std::is_same<T, ff>::value)
        own_fold_ff_kernel<<<ew_grid(np), 256, 0, st>>>(LL.Cm64, reinterpret_cast<ffv *>(LL.Cm_ff), LL.nb, LL.p, P->dsc_leaf_dev);
    for (int l = P->lmax; l > P->lmin && !e; l--) {
        beg(P, PASS_M2M, l);
        e = pass(l, PASS_M2M);
        end(P);
    }
    for (int l = P->lmin; l <= P->lmax && !e; l++) {
        beg(P, PASS_M2L, l);
        if (l > P->lmin) e = pass(l, PASS_L2L);
        if (!e) e = pass(l, PASS_M2L);
        end(P);
    }
    if (form.part_bytes) {
        const int g = pool_give(P);
        if (!e) e = g;
    }
    if (e) return e;
    if (std::is_same<T, double>::value)
        own_fold_kernel<<<ew_grid(np), 256, 0, st>>>(LL.Dl64, LL.nb, LL.p, 0);
    else if (std::is_same<T, ff>::value)
        own_unfold_ff_kernel<<<ew_grid(np), 256, 0, st>>>(reinterpret_cast<const ffv *>(LL.Dl_ff), LL.Dl64, LL.nb, LL.p, P->dsc_leaf_dev);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

} // namespace

int translate_owner(Plan *P, int type, void (*beg)(Plan *, int, int), void (*end)(Plan *))
{
    return type == OWN_FP64 ? translate<double>(P, beg, end)
                            : type == OWN_FF ? translate<ff>(P, beg, end) : translate<float>(P, beg, end);
}

int prepare_owner(Plan *P, int type)
{
    int e = type == OWN_FP64 ? ensure_own<double>(P) : type == OWN_FF ? ensure_own<ff>(P) : ensure_own<float>(P);
    // a small scratch too (0.1 ms of a first matvec)
    void *part = nullptr;
    const size_t bytes = P->own_form[type].part_bytes;
    if (!e && bytes && bytes <= SMALL_PART && !(e = pool_take(P, bytes, &part))) e = pool_give(P);
    return e;
}

void free_owner(Plan *P)
{
    for (OwnLists &l : P->own_lists) cudaFree(l.mem);
    for (OwnForm &f : P->own_form) cudaFree(f.mem);
    cudaFree(P->own_rot64);
    cudaFree(P->own_rot_ff);
    pool_leave(P);
}

} // namespace fmm
