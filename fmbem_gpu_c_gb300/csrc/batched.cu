// Batched translations for the mixed-precision matvec: M2M, M2L and L2L as tiles of
// register-blocked small matrix products.
//
// Every translation is rotation - coaxial - rotation (RCR) as in transMatsVecsMul_SR_rcr
// (reference translation.cu:1864-1961).  Translations of one operator class -- the M2L directions
// of equal (dz, dx^2 + dy^2), which have one polar angle and one length (61 classes of the 316
// directions); the octants of M2M / L2L of equal z bit -- share the rotation and coaxial blocks
// and differ by their azimuthal phases.  A CTA takes TC of them (times the right-hand sides) as the
// columns of a matrix in shared memory:
//   gather   x_m e^{i m phi}, as the sums x+_m = x_m + x_-m and differences x-_m = x_m - x_-m;
//   rotate   W+_n = P_n X+_n, W-_n = Q_n X-_n for every degree n: the rotation block is centrally
//            symmetric (H_{-m',-m} = H_{m',m}), so it splits into two blocks of half its size;
//   coaxial  X+-_m = C_m W+-_m for every order m (complex, the same block for both signs);
//   rotate   back, and write x_+-m = (W+ +- W-)/2 times e^{-+i m phi} into the destinations.
// A lane owns 4 columns x R rows of one block (a unit): an operand row of 4 columns is two 16-byte
// shared-memory loads and R table entries one load (the tables are padded for it), for 8 R
// (rotation) or 32 (coaxial, two rows) multiply-adds, issued as packed pairs (re, im).  The stages work
// in place: a round of units holds whole blocks, which depend on their own rows only, and writes
// after a barrier.  That halves the shared memory, so that three CTAs share an SM and its L1 keeps
// the class's tables.  Every output is summed in the same order whatever the tile.  Destinations
// are added with FP32 vector atomics where several items reach the same box (M2M, M2L), and with a
// plain read-add-write where every box is reached once (L2L).
// Small bodies with many columns take another form of the tiles (FORM_WHOLE, tile_form()): one direction each, the
// rotations whole, every product and sum rounded as by one thread per row of the plain basis.
//
// What bounds it: the shared-memory / L1 path (16 bytes of table and 32 of operands per lane for 32
// multiply-adds: 65-80 % busy at p = 10-20) and, at p = 30-40, the latency of table rows from L2.
// M2L of 16 columns on the 81,920-triangle sphere, against one tile per direction with the whole
// rotation blocks in two buffers: p = 40 2.50 -> 1.31 ms, p = 30 4.55 -> 2.60, p = 20 6.65 -> 4.03;
// the sphere's matvec 2.15 -> 1.59 ms, 64 columns on the head 145 -> 117 ms, 24 bodies as a scene
// 2.74 -> 1.93 ms.  Tried: two CTAs of 128 registers (28 -> 32 ms for 16 columns), 8 columns per
// lane (28 -> 31), table rows loaded 2 to 6 steps ahead (slower than one ahead).
#include "plan.h"
#include "f32x2.cuh"
#include <algorithm>
#include <cstdlib>
#include <vector>

namespace fmm {

// ---- table layouts
__host__ __device__ __forceinline__ int up_to(int n, int q) { return (n + q - 1) / q * q; }
// folded rotation tables: degree n holds P_n as [m = 0..n][rows 0..n, padded to 4], then Q_n as
// [m = 1..n][rows 1..n, padded to 4]
static int rot32_size(int p)
{
    int s = 0;
    for (int n = 0; n < p; n++) s += (n + 1) * up_to(n + 1, 4) + n * up_to(n, 4);
    return s;
}
// coaxial tables of order p: order m holds [n = m..p-1][rows m..p-1, padded to 2]
__host__ __device__ __forceinline__ int coax2_sum(int n) { return n * (n + 1) * (2 * n + 1) / 6 + ((n + 1) / 2) * ((n + 1) / 2); }
__host__ __device__ __forceinline__ int coax2_off(int p, int m) { return coax2_sum(p) - coax2_sum(p - m); }
static int coax2_size(int p) { return coax2_sum(p); }

// P and Q of the classes' representative rows rep[k] of H, degree blockIdx.x (see rot32_size)
__global__ void rot32_table_kernel(int pmax, const int *__restrict__ rep, const int *__restrict__ off, int stride,
                                   const double *__restrict__ H, float *__restrict__ out)
{
    const int n = blockIdx.x, k = blockIdx.y, w = 2 * n + 1, rp = up_to(n + 1, 4), rm = up_to(n, 4);
    const double *Hn = H + (size_t)rep[k] * rot_size(pmax) + rot_off(n);
    float *o = out + (size_t)k * stride + off[n];
    for (int t = threadIdx.x; t < (n + 1) * rp + n * rm; t += blockDim.x) {
        double v = 0.0;
        if (t < (n + 1) * rp) {
            const int m = t / rp, r = t % rp;
            if (r <= n) {
                const double a = Hn[(n + m) * w + n + r], b = Hn[(n - m) * w + n + r];
                v = m ? (r ? a + b : 0.5 * (a + b)) : (r ? a + Hn[n * w + n - r] : a);
            }
        } else {
            const int u = t - (n + 1) * rp, m = u / rm + 1, r = u % rm + 1;
            if (r <= n) v = Hn[(n + m) * w + n + r] - Hn[(n - m) * w + n + r];
        }
        o[t] = (float)v;
    }
}

// the coaxial tables of order p (layout of coax_off, blockIdx.y = table) in the padded layout
__global__ void coax2_table_kernel(int p, const float2 *__restrict__ in, float2 *__restrict__ out)
{
    const int m = blockIdx.x, sz = p - m, ld = up_to(sz, 2);
    const float2 *a = in + (size_t)blockIdx.y * coax_size(p) + coax_off(p, m);
    float2 *o = out + (size_t)blockIdx.y * coax2_sum(p) + coax2_off(p, m);
    for (int t = threadIdx.x; t < sz * ld; t += blockDim.x) {
        const int n = t / ld, r = t % ld;
        o[t] = r < sz ? a[n * sz + r] : make_float2(0.f, 0.f);
    }
}

// element (row, column) of a tile: the 16-byte chunks (2 columns) of a row are XOR-swizzled by the
// row, so that lanes on different rows spread over the banks
template <int TC>
__device__ __forceinline__ int swz(int row)
{
    constexpr int M = (TC / 2 < 8 ? TC / 2 : 8) - 1;
    return row & M;
}

template <int R> struct Rows;
template <> struct Rows<4> { typedef float4 t; };
template <> struct Rows<2> { typedef float2 t; };
constexpr int THREADS = 256, CG = 4;  // threads of a CTA, columns of a lane

// A table entry, from global memory or (S) from the tile's copy in shared memory
template <bool S, class T> __device__ __forceinline__ T entry(const T *p)
{
    if constexpr (S) return *p;
    else return __ldg(p);
}

// One rotation stage, in place.  Round k gives thread t unit k UC + t / CL and the
// column pairs cl, cl + CL (cl = t % CL): (n | sign << 8 | first row << 16, table offset), R rows of P_n or Q_n
// (whole rotations: of H_n, no sign).  All units of a block (n, sign) are in one round, which writes after everyone
// has read.
template <int TC, int R, bool S, bool FOLD>
__device__ __forceinline__ void rot_stage(const float *__restrict__ rot, ulonglong2 *X, const int2 *__restrict__ units, int rounds)
{
    constexpr int CL = TC / CG, UC = THREADS / CL, NC = CG / 2;
    const int cl = threadIdx.x % CL, ul = threadIdx.x / CL;
    for (int k = 0; k < rounds; k++) {
        const int2 info = __ldg(units + k * UC + ul);
        const bool on = info.x >= 0;
        const int n = on ? info.x & 255 : 0, minus = on ? (info.x >> 8) & 1 : 0, row0 = on ? info.x >> 16 : 0;
        const int len = FOLD ? (minus ? n : n + 1) : 2 * n + 1, steps = on ? len : 0, ld = up_to(len, 4), c0 = FOLD ? n * n + n : n * n;
        const float *h = rot + info.y;
        f2 acc[R][CG];
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int c = 0; c < CG; c++) acc[r][c] = 0ull;
        int row = minus ? c0 - 1 : c0;
        const int dr = minus ? -1 : 1;
        typename Rows<R>::t hn = entry<S>(reinterpret_cast<const typename Rows<R>::t *>(h));
#pragma unroll 2
        for (int m = 0; m < steps; m++) {
            const typename Rows<R>::t hv = hn;
            if (m + 1 < steps) h += ld;  // the last step loads its own entries again
            hn = entry<S>(reinterpret_cast<const typename Rows<R>::t *>(h));
            ulonglong2 x[NC];
            const ulonglong2 *xr = X + row * (TC / 2);
            const int s = swz<TC>(row);
#pragma unroll
            for (int i = 0; i < NC; i++) x[i] = xr[(cl + i * CL) ^ s];
            row += dr;
            const float *hc = reinterpret_cast<const float *>(&hv);
#pragma unroll
            for (int r = 0; r < R; r++) {
                const f2 hh = f2_pack(hc[r], hc[r]);
#pragma unroll
                for (int i = 0; i < NC; i++) {
                    acc[r][2 * i] = f2_fma(hh, x[i].x, acc[r][2 * i]);
                    acc[r][2 * i + 1] = f2_fma(hh, x[i].y, acc[r][2 * i + 1]);
                }
            }
        }
        __syncthreads();
        const int nrow = steps - row0;  // rows of the block from row0 on
#pragma unroll
        for (int r = 0; r < R; r++)
            if (r < nrow) {
                const int q = minus ? c0 - 1 - row0 - r : c0 + row0 + r;
#pragma unroll
                for (int i = 0; i < NC; i++)
                    X[q * (TC / 2) + ((cl + i * CL) ^ swz<TC>(q))] = make_ulonglong2(acc[r][2 * i], acc[r][2 * i + 1]);
            }
    }
}

// The coaxial stage, in place, in rounds as above.  Unit: |m| | sign << 8 | first row << 16, two of
// the rows of order +-m.  Folded: the products with re(c) and im(c) in sums of their own; else one sum.
template <int TC, bool S, bool FOLD>
__device__ __forceinline__ void coax_stage(int p, int nin, int nq, const float2 *__restrict__ Cc, ulonglong2 *X,
                                           const int *__restrict__ units, int rounds)
{
    constexpr int CL = TC / CG, UC = THREADS / CL, NC = CG / 2;
    const int cl = threadIdx.x % CL, ul = threadIdx.x / CL;
    for (int k = 0; k < rounds; k++) {
        const int info = __ldg(units + k * UC + ul);
        const bool on = info >= 0;
        const int am = on ? info & 255 : 0, minus = on ? (info >> 8) & 1 : 0, row0 = on ? info >> 16 : 0;
        const int steps = on ? nin - am : 0, ld = up_to(p - am, 2);
        const float4 *c = reinterpret_cast<const float4 *>(Cc + coax2_off(p, am) + row0);
        f2 a0[2][CG], a1[2][CG];
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int j = 0; j < CG; j++) a0[r][j] = a1[r][j] = 0ull;
        const int sm = minus ? -am : am;
        int row = am * am + am + sm, dr = 2 * am + 2;
        float4 cn = entry<S>(c);
#pragma unroll 2
        for (int n = 0; n < steps; n++) {
            const float4 cc = cn;
            if (n + 1 < steps) c += ld / 2;
            cn = entry<S>(c);
            ulonglong2 x[NC];
            const ulonglong2 *xr = X + row * (TC / 2);
            const int s = swz<TC>(row);
#pragma unroll
            for (int i = 0; i < NC; i++) x[i] = xr[(cl + i * CL) ^ s];
            row += dr;
            dr += 2;
            const f2 re[2] = {f2_pack(cc.x, cc.x), f2_pack(cc.z, cc.z)}, im[2] = {f2_pack(FOLD ? cc.y : -cc.y, cc.y), f2_pack(FOLD ? cc.w : -cc.w, cc.w)};
#pragma unroll
            for (int r = 0; r < 2; r++) {
#pragma unroll
                for (int i = 0; i < NC; i++) {
                    a0[r][2 * i] = f2_fma(re[r], x[i].x, a0[r][2 * i]);
                    a0[r][2 * i + 1] = f2_fma(re[r], x[i].y, a0[r][2 * i + 1]);
                    if constexpr (FOLD) {
                        a1[r][2 * i] = f2_fma(im[r], x[i].x, a1[r][2 * i]);
                        a1[r][2 * i + 1] = f2_fma(im[r], x[i].y, a1[r][2 * i + 1]);
                    } else {
                        a0[r][2 * i] = f2_fma(im[r], f2_swap(x[i].x), a0[r][2 * i]);
                        a0[r][2 * i + 1] = f2_fma(im[r], f2_swap(x[i].y), a0[r][2 * i + 1]);
                    }
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 2; r++)
            if (on && row0 + r < nq - am) {
                const int nn = am + row0 + r, q = nn * nn + nn + sm;
                f2 y[CG];
#pragma unroll
                for (int j = 0; j < CG; j++) {
                    y[j] = a0[r][j];
                    if constexpr (FOLD) {
                        const float2 v = f2_parts(a0[r][j]), w = f2_parts(a1[r][j]);
                        y[j] = f2_pack(v.x - w.y, v.y + w.x);
                    }
                }
#pragma unroll
                for (int i = 0; i < NC; i++)
                    X[q * (TC / 2) + ((cl + i * CL) ^ swz<TC>(q))] = make_ulonglong2(y[2 * i], y[2 * i + 1]);
            }
    }
}

// v e and conj(e) v, each product and sum rounded in one fixed way
__device__ __forceinline__ float2 phase_mul(float2 v, float2 e)
{
    return make_float2(__fmaf_rn(v.x, e.x, -__fmul_rn(v.y, e.y)), __fmaf_rn(v.y, e.x, __fmul_rn(v.x, e.y)));
}
__device__ __forceinline__ float2 conj_phase_mul(float2 e, float2 v)
{
    return make_float2(__fmaf_rn(e.x, v.x, __fmul_rn(e.y, v.y)), __fmaf_rn(e.x, v.y, -__fmul_rn(e.y, v.x)));
}

// One tile: item it = (class, first column, count, coaxial table) of pass ps, with the
// CTA's dynamic shared memory and its column indices.  S: the class's rotation table and the
// coaxial table are copied to shared memory behind the tile (ps.tile_words 16-byte words) while the
// columns are gathered.  Each step of a stage waits for its table entries; in a pass of so few tiles that each SM
// has one or two, nothing hides their way from the L2.
// FOLD = false: the rotations whole, in the plain basis, and each product and sum rounded in one fixed way.
template <int TC, int R, bool S, bool FOLD>
__device__ __forceinline__ void rcr_tile(const RcrPass &ps, const int4 it, float4 *smem4, int *s_src, int *s_dst, int *s_dir)
{
    const int p = ps.p, nin = min(ps.pin, p), nq = min(ps.pout, p), cnt = it.z;
    ulonglong2 *X = reinterpret_cast<ulonglong2 *>(smem4);
    float2 *Xf = reinterpret_cast<float2 *>(X);
    const float *rot = ps.rot + (size_t)(FOLD ? it.x : it.x & 255) * ps.rot_stride;
    const float2 *coax = ps.coax + (size_t)it.w * coax2_sum(p);
    if constexpr (S) {
        const float4 *r4 = reinterpret_cast<const float4 *>(rot), *c4 = reinterpret_cast<const float4 *>(coax);
        float4 *to = smem4 + ps.tile_words;
        const int nr = ps.rot_words, nc = coax2_sum(p) / 2;
        for (int i = threadIdx.x; i < nr + nc; i += THREADS)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to + i)),
                         "l"(i < nr ? r4 + i : c4 + (i - nr)) : "memory");
        rot = reinterpret_cast<const float *>(to);
        coax = reinterpret_cast<const float2 *>(to + nr);
    }
    if (threadIdx.x < TC) {
        // column e = translation t x nrhs + right-hand side r; the expansions hold the columns
        // of a box next to each other ([box][rhs][p^2])
        const int e = it.y + min((int)threadIdx.x, cnt - 1), t = e / ps.nrhs, r = e - t * ps.nrhs;
        s_src[threadIdx.x] = ps.g_src[t] * ps.nrhs + r;
        s_dst[threadIdx.x] = ps.g_dst[t] * ps.nrhs + r;
        s_dir[threadIdx.x] = FOLD ? ps.g_dir[t] : ps.key0 + (it.x >> 8);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int gi = lane & 7, gc = lane >> 3;  // gather / scatter: 8 pairs (n, m >= 0) x 4 columns per warp
    {
        const int np = nin * (nin + 1) / 2, nb = (np + 7) / 8 * (TC / 4), sstride = ps.pin * ps.pin;
        constexpr int GU = 4;  // blocks in flight per warp
        for (int b0 = warp; b0 < nb; b0 += GU * nw) {
            int nm[GU];
            float2 vp[GU], vm[GU], e[GU];
#pragma unroll
            for (int j = 0; j < GU; j++) {
                const int b = b0 + j * nw, q = b / (TC / 4) * 8 + gi;
                nm[j] = b < nb && q < np ? __ldg(ps.pairs + q) : -1;
            }
#pragma unroll
            for (int j = 0; j < GU; j++) {
                const int c = (b0 + j * nw) % (TC / 4) * 4 + gc, m = nm[j] >> 16, r0 = nm[j] & 0xffff;
                vp[j] = vm[j] = make_float2(0.f, 0.f);
                e[j] = make_float2(1.f, 0.f);
                if (nm[j] >= 0 && c < cnt) {
                    const float2 *in = ps.src + (size_t)s_src[c] * sstride + r0;
                    vp[j] = __ldg(in + m);
                    if (m > 0) {
                        vm[j] = __ldg(in - m);
                        e[j] = __ldg(ps.PHall + (size_t)s_dir[c] * ps.phstride + ps.phoff + m);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < GU; j++) {
                if (nm[j] < 0) continue;
                const int c = (b0 + j * nw) % (TC / 4) * 4 + gc, m = nm[j] >> 16, r0 = nm[j] & 0xffff, rp = r0 + m, rm = r0 - m;
                // m = 0: x itself (vm = 0, e = 1)
                if constexpr (!FOLD) {
                    Xf[rp * TC + (((c >> 1) ^ swz<TC>(rp)) << 1) + (c & 1)] = phase_mul(vp[j], e[j]);
                    if (m > 0) Xf[rm * TC + (((c >> 1) ^ swz<TC>(rm)) << 1) + (c & 1)] = phase_mul(vm[j], make_float2(e[j].x, -e[j].y));
                    continue;
                }
                const float2 a = make_float2(vp[j].x + vm[j].x, vp[j].y + vm[j].y);
                const float2 d = make_float2(vp[j].x - vm[j].x, vp[j].y - vm[j].y);
                Xf[rp * TC + (((c >> 1) ^ swz<TC>(rp)) << 1) + (c & 1)] =
                    make_float2(e[j].x * a.x - e[j].y * d.y, e[j].x * a.y + e[j].y * d.x);
                if (m > 0)
                    Xf[rm * TC + (((c >> 1) ^ swz<TC>(rm)) << 1) + (c & 1)] =
                        make_float2(e[j].x * d.x - e[j].y * a.y, e[j].x * d.y + e[j].y * a.x);
            }
        }
    }
    if constexpr (S) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    rot_stage<TC, R, S, FOLD>(rot, X, ps.u1, ps.n1);
    __syncthreads();
    coax_stage<TC, S, FOLD>(p, nin, nq, coax, X, ps.u2, ps.n2);
    __syncthreads();
    rot_stage<TC, R, S, FOLD>(rot, X, ps.u3, ps.n3);
    __syncthreads();
    {
        const int np = nq * (nq + 1) / 2, nb = (np + 7) / 8 * (TC / 4), dstride = ps.pout * ps.pout;
        for (int b = warp; b < nb; b += nw) {
            const int q = b / (TC / 4) * 8 + gi, c = b % (TC / 4) * 4 + gc;
            if (q >= np || c >= cnt) continue;
            const int nm = __ldg(ps.pairs + q), m = nm >> 16, r0 = nm & 0xffff, rp = r0 + m, rm = r0 - m;
            float2 *out = ps.dst + (size_t)s_dst[c] * dstride + r0;
            float2 yp = Xf[rp * TC + (((c >> 1) ^ swz<TC>(rp)) << 1) + (c & 1)], ym = yp;
            if (m > 0) {
                const float2 v = Xf[rm * TC + (((c >> 1) ^ swz<TC>(rm)) << 1) + (c & 1)];
                const float2 e = __ldg(ps.PHall + (size_t)s_dir[c] * ps.phstride + ps.phoff + m);
                if constexpr (FOLD) {
                    const float2 a = make_float2(0.5f * (yp.x + v.x), 0.5f * (yp.y + v.y));
                    const float2 d = make_float2(0.5f * (yp.x - v.x), 0.5f * (yp.y - v.y));
                    yp = make_float2(e.x * a.x + e.y * a.y, e.x * a.y - e.y * a.x);
                    ym = make_float2(e.x * d.x - e.y * d.y, e.x * d.y + e.y * d.x);
                } else {
                    yp = conj_phase_mul(e, yp);
                    ym = conj_phase_mul(make_float2(e.x, -e.y), v);
                }
            }
            if (ps.atomic) {
                atomicAdd(out + m, yp);
                if (m > 0) atomicAdd(out - m, ym);
            } else {
                const float2 o = out[m];
                out[m] = make_float2(o.x + yp.x, o.y + yp.y);
                if (m > 0) {
                    const float2 v = out[-m];
                    out[-m] = make_float2(v.x + ym.x, v.y + ym.y);
                }
            }
        }
    }
}

template <int TC, int R, bool S, bool FOLD>
__global__ void __launch_bounds__(THREADS, 3) rcr_tile_kernel(RcrPass ps)
{
    extern __shared__ float4 smem4[];
    __shared__ int s_src[TC], s_dst[TC], s_dir[TC];
    rcr_tile<TC, R, S, FOLD>(ps, ps.items[blockIdx.x], smem4, s_src, s_dst, s_dir);
}

// Persistent form for many passes at once (the translation passes of many plans, one phase
// of a lockstep matvec): a grid of resident CTAs takes work items (pass, tile) from a device
// queue, in the order given (longest first), until it is empty.  The queue head is an
// atomic counter, zeroed before the launch; no CTA waits on another.
template <int TC, int R>
__global__ void __launch_bounds__(THREADS, 3) rcr_queue_kernel(const RcrPass *__restrict__ passes, const int *__restrict__ work_pass,
                                                           const int4 *__restrict__ work_item, const int *__restrict__ nwork,
                                                           int *head)
{
    extern __shared__ float4 smem4[];
    __shared__ int s_src[TC], s_dst[TC], s_dir[TC];
    __shared__ int s_w;
    const int n = *nwork;
    for (;;) {
        if (threadIdx.x == 0) s_w = atomicAdd(head, 1);
        __syncthreads();
        const int w = s_w;
        if (w >= n) break;
        rcr_tile<TC, R, false, true>(passes[work_pass[w]], work_item[w], smem4, s_src, s_dst, s_dir);
        __syncthreads();
    }
}

// a tile of p^2 rows (p the larger of the orders a pass uses) of tc complex columns
size_t rcr_tile_smem(int p, int tc) { return (size_t)p * p * tc * sizeof(float2); }

template <int TC_, int R_> struct Tile {
    static constexpr int TC = TC_, R = R_;
};

// Calls f(Tile<...>{}) for tc columns and units of four rows (bal = 0) or two (1)
template <class F>
static int with_tile(int tc, int bal, F &&f)
{
    switch (tc) {
    case 64: return bal ? f(Tile<64, 2>{}) : f(Tile<64, 4>{});
    case 32: return bal ? f(Tile<32, 2>{}) : f(Tile<32, 4>{});
    case 16: return bal ? f(Tile<16, 2>{}) : f(Tile<16, 4>{});
    case 8: return bal ? f(Tile<8, 2>{}) : f(Tile<8, 4>{});
    default: return bal ? f(Tile<4, 2>{}) : f(Tile<4, 4>{});
    }
}

// Raise the queue kernel's shared-memory limit and size its grid: every CTA resident at once
// (SMs x CTAs per SM at this shared memory), no more than the items.
int rcr_queue_prepare(int tc, int bal, size_t sm, int nwork, int *grid)
{
    return with_tile(tc, bal, [&](auto t) -> int {
        using T = decltype(t);
        static size_t attr = 0;
        const void *fn = (const void *)rcr_queue_kernel<T::TC, T::R>;
        int e = raise_smem_limit(fn, sm, &attr);
        if (e) return e;
        int dev = 0, nsm = 0, per_sm = 0;
        FMM_CUDA_TRY(cudaGetDevice(&dev));
        FMM_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        FMM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 256, sm));
        *grid = std::max(1, std::min(nwork, nsm * std::max(per_sm, 1)));
        return FMM_OK;
    });
}

int launch_rcr_queue(int tc, int bal, const RcrPass *passes, const int *work_pass, const int4 *work_item,
                     const int *nwork, int *head, size_t sm, int grid, cudaStream_t st)
{
    return with_tile(tc, bal, [&](auto t) -> int {
        using T = decltype(t);
        rcr_queue_kernel<T::TC, T::R><<<grid, 256, sm, st>>>(passes, work_pass, work_item, nwork, head);
        FMM_CUDA_TRY(cudaGetLastError());
        return FMM_OK;
    });
}

// Work items over the columns e = t nrhs + r of a list: tiles of at most `width` columns of
// one key, item .w = the key's coaxial block when coax_w.  Where the
// expansions a pass touches for nrhs columns (ws_bytes) are more than L2 keeps, the
// destination boxes are cut into Morton ranges and the items ordered range by range, so that
// the tiles in flight share their sources and destinations in L2.  Each key's
// translations are sorted by the Morton rank of their destination, so a range is one
// contiguous run of every key.
static const size_t L2_BUDGET = 48u << 20;

void build_items(const KeyedList &Lst, int nrhs, int width, size_t ws_bytes, bool coax_w, std::vector<int4> &items)
{
    items.clear();
    const int nkeys = (int)Lst.key_beg.size() - 1, nd = std::max(Lst.ndst_rank, 1);
    const long long nblk = std::min<long long>(nd, std::max<long long>(1, (long long)((ws_bytes + L2_BUDGET - 1) / L2_BUDGET)));
    const int *rk = Lst.dst_rank.data();
    for (long long k = 0; k < nblk; k++) {
        const int lo = (int)(k * nd / nblk), hi = (int)((k + 1) * nd / nblk);
        for (int d = 0; d < nkeys; d++) {
            int a0 = Lst.key_beg[d], a1 = Lst.key_beg[d + 1];
            if (nblk > 1) {
                a0 = (int)(std::lower_bound(rk + Lst.key_beg[d], rk + Lst.key_beg[d + 1], lo) - rk);
                a1 = (int)(std::lower_bound(rk + Lst.key_beg[d], rk + Lst.key_beg[d + 1], hi) - rk);
            }
            const long long e0 = (long long)a0 * nrhs, e1 = (long long)a1 * nrhs;
            for (long long a = e0; a < e1; a += width)
                items.push_back(make_int4(d, (int)a, (int)std::min<long long>(width, e1 - a), coax_w ? Lst.key_w[d] : 0));
        }
    }
}

// translations in class order: source, destination, phase row of direction key0 + d
__global__ void class_order_kernel(int n, const int *__restrict__ perm, const int *__restrict__ src, const int *__restrict__ dst,
                                   const int *__restrict__ key_beg, int nkeys, int key0, int *__restrict__ csrc,
                                   int *__restrict__ cdst, short *__restrict__ cdir)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int t = perm[i];
        int lo = 0, hi = nkeys;  // the last direction whose run begins at or before t
        while (hi - lo > 1) {
            const int m = (lo + hi) >> 1;
            if (key_beg[m] <= t) lo = m; else hi = m;
        }
        csrc[i] = src[t];
        cdst[i] = dst[t];
        cdir[i] = (short)(key0 + lo);
    }
}

// The list by operator class, on first use of the SIMT tiles.
static int ensure_classes(RcrList &Lst)
{
    if (Lst.csrc || Lst.key_beg.empty() || Lst.key_beg.back() == 0) return FMM_OK;
    const int n = Lst.key_beg.back(), nkeys = (int)Lst.key_beg.size() - 1;
    KeyedList &C = Lst.cls;
    const int ncls = *std::max_element(Lst.cls_of_key.begin(), Lst.cls_of_key.end()) + 1, nd = Lst.ndst_rank;
    // two stable counting sorts: by destination rank, then by class
    std::vector<int> cls(n), byrank(n), perm(n), cnt(nd + 1, 0);
    for (int d = 0; d < nkeys; d++)
        for (int t = Lst.key_beg[d]; t < Lst.key_beg[d + 1]; t++) cls[t] = Lst.cls_of_key[d];
    for (int t = 0; t < n; t++) cnt[Lst.dst_rank[t] + 1]++;
    for (int r = 0; r < nd; r++) cnt[r + 1] += cnt[r];
    for (int t = 0; t < n; t++) byrank[cnt[Lst.dst_rank[t]]++] = t;
    C.key_beg.assign(ncls + 1, 0);
    C.key_w.assign(ncls, 0);
    C.ndst_rank = nd;
    for (int d = 0; d < nkeys; d++) C.key_w[Lst.cls_of_key[d]] = Lst.key_w[d];
    for (int t = 0; t < n; t++) C.key_beg[cls[t] + 1]++;
    for (int c = 0; c < ncls; c++) C.key_beg[c + 1] += C.key_beg[c];
    std::vector<int> fill(C.key_beg.begin(), C.key_beg.end());
    C.dst_rank.resize(n);
    for (int t : byrank) {
        const int i = fill[cls[t]]++;
        perm[i] = t;
        C.dst_rank[i] = Lst.dst_rank[t];
    }
    int *tmp = nullptr, *cs = nullptr;
    FMM_CUDA_TRY(cudaMalloc(&tmp, sizeof(int) * (n + nkeys + 1)));
    cudaError_t ce = cudaMalloc(&cs, sizeof(int) * n);
    if (ce == cudaSuccess) ce = cudaMalloc(&Lst.cdst, sizeof(int) * n);
    if (ce == cudaSuccess) ce = cudaMalloc(&Lst.cdir, sizeof(short) * n);
    if (ce == cudaSuccess) ce = upload(tmp, perm.data(), sizeof(int) * n);
    if (ce == cudaSuccess) ce = upload(tmp + n, Lst.key_beg.data(), sizeof(int) * (nkeys + 1));
    if (ce == cudaSuccess) {
        class_order_kernel<<<std::min((n + 255) / 256, 152 * 16), 256>>>(n, tmp, Lst.src, Lst.dst, tmp + n, nkeys, Lst.key0, cs,
                                                                        Lst.cdst, Lst.cdir);
        ce = cudaGetLastError();
    }
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(0);
    cudaFree(tmp);
    if (ce != cudaSuccess) {
        cudaFree(cs);
        cudaFree(Lst.cdst);
        cudaFree(Lst.cdir);
        Lst.cdst = nullptr;
        Lst.cdir = nullptr;
    }
    FMM_CUDA_TRY(ce);
    Lst.csrc = cs;
    return FMM_OK;
}

// Device items of a form of a SIMT pass for nrhs right-hand sides, rebuilt when nrhs changes.
static int ensure_items(RcrList &Lst, int form, int nrhs, size_t ws_bytes)
{
    TileForm &f = Lst.form[form];
    if (f.items_nrhs == nrhs) return FMM_OK;
    std::vector<int4> items;
    if (form == FORM_FOLDED) {
        if (int e = ensure_classes(Lst)) return e;
        build_items(Lst.cls, nrhs, f.tc, ws_bytes, true, items);
    } else {
        build_items(Lst, nrhs, f.tc, ws_bytes, true, items);
        for (int4 &it : items) it.x = Lst.cls_of_key[it.x] | it.x << 8;
    }
    if (items.size() > f.items_cap) {
        if (f.items) cudaFree(f.items);
        f.items = nullptr;
        f.items_cap = 0;
        FMM_CUDA_TRY(cudaMalloc(&f.items, sizeof(int4) * items.size()));
        f.items_cap = items.size();
    }
    if (!items.empty()) FMM_CUDA_TRY(upload(f.items, items.data(), sizeof(int4) * items.size()));
    f.n_items = (int)items.size();
    f.items_nrhs = nrhs;
    return FMM_OK;
}

int rcr_list_items(RcrList &Lst, std::vector<int4> &items)
{
    int e = ensure_classes(Lst);
    if (e) return e;
    build_items(Lst.cls, 1, Lst.form[FORM_FOLDED].tc, 0, true, items);
    return FMM_OK;
}

static size_t tile_bytes(const RcrPass &ps, int tc)
{
    return rcr_tile_smem(std::max(std::min(ps.pin, ps.p), std::min(ps.pout, ps.p)), tc);
}

// The form of the SIMT tiles for nrhs columns.  Folded rotations by class are the faster ones (27 columns on an
// 8,820-triangle sphere 4.7 ms against 5.2, 49 on a 4,500-triangle ellipsoid 4.7 against 6.2; one tile per
// direction with two buffers and units over the whole block took 6.4 and 7.3), but add a box's translations in
// an order of their own: two runs of many columns on a small body differ by 2e-8 where directions one after
// another, with several tiles each, differ by 5e-9, and the results move by four to ten times that.  So from
// 16 columns on, bodies of fewer than 100,000 translations keep whole rotations
// and the order of directions; with fewer columns, and on larger bodies, whose orders are no more
// reproducible one way than the other, the results differ by what two runs differ by.
static int tile_form(const Plan *P, int nrhs)
{
    long long T = 0;
    for (int l = P->lmin; l <= P->lmax; l++) T += P->lev[l].num_sr;
    return nrhs >= 16 && T < 100000 ? FORM_WHOLE : FORM_FOLDED;
}

int launch_rcr_pass(Plan *P, RcrList &Lst, RcrPass ps, cudaStream_t st)
{
    if (Lst.key_beg.empty() || Lst.key_beg.back() == 0) return FMM_OK;
    const int form = tile_form(P, ps.nrhs);
    if (form == FORM_WHOLE)
        if (int e = ensure_whole_tables(P)) return e;
    TileForm &f = Lst.form[form];
    if (int e = set_tile_tables(P, Lst, form, ps)) return e;
    {
        size_t ws = ((size_t)ps.nsrc * ps.pin * ps.pin + (size_t)ps.ndst * ps.pout * ps.pout) * sizeof(float2) * ps.nrhs;
        int e = ensure_items(Lst, form, ps.nrhs, ws);
        if (e) return e;
    }
    ps.items = f.items;
    const size_t sm = tile_bytes(ps, f.tc);
    ps.tile_words = (int)(sm / 16);
    ps.rot_words = rot32_size(ps.p) / 4;
    const size_t sm_tab = sm + (size_t)ps.rot_words * 16 + (size_t)coax2_size(ps.p) * sizeof(float2);
    static int nsm = 0;
    if (!nsm) {
        int dev = 0;
        FMM_CUDA_TRY(cudaGetDevice(&dev));
        FMM_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    }
    // tables in shared memory where every tile is resident at once all the same, three CTAs of up to 74 KB on an
    // SM (a matvec on 5,120 triangles, orders 16, 14, 12: 198 us without, 179 with; larger tables, 81,920
    // triangles with orders up to 40: no gain)
    const bool staged = form == FORM_FOLDED && sm_tab <= 74 * 1024 && f.n_items <= 3 * nsm;
    return with_tile(f.tc, f.bal, [&](auto t) -> int {
        using T = decltype(t);
        static size_t attr[3] = {0, 0, 0};
        const auto kernel = form == FORM_WHOLE ? rcr_tile_kernel<T::TC, T::R, false, false>
                            : staged ? rcr_tile_kernel<T::TC, T::R, true, true> : rcr_tile_kernel<T::TC, T::R, false, true>;
        int e = raise_smem_limit((const void *)kernel, staged ? sm_tab : sm, &attr[form == FORM_WHOLE ? 2 : staged]);
        if (e) return e;
        kernel<<<f.n_items, 256, staged ? sm_tab : sm, st>>>(ps);
        FMM_CUDA_TRY(cudaGetLastError());
        return FMM_OK;
    });
}

// Shared memory that keeps two CTAs on an SM: 228 KB per SM, 1 KB reserved and the static
// arrays per CTA.
static const size_t TWO_CTA_SMEM = (228 * 1024) / 2 - 1024 - 1024;

// Columns per CTA: the most that keep two CTAs on an SM, so that one computes while the other
// gathers or waits at a barrier; at least 4 (p <= 60).
static int pick_tile(int p)
{
    for (int tc = 64; tc > 4; tc /= 2)
        if (rcr_tile_smem(p, tc) <= TWO_CTA_SMEM) return tc;
    return 4;
}

// Classes of a pass's keys with one rotation and length: M2L directions of equal (dz, dx^2 + dy^2),
// M2M / L2L octants of equal z bit.  cls[key] = class, rep[class] = its first key.
void direction_classes(const Plan *P, int which, int nkeys, std::vector<int> &cls, std::vector<int> &rep)
{
    cls.assign(nkeys, -1);
    rep.clear();
    std::vector<int> off(nkeys, 0), seen;
    if (which == PASS_M2L)
        for (int q = 0; q < 343; q++)
            if (P->dir_slot[q] >= 0 && P->dir_slot[q] < nkeys) off[P->dir_slot[q]] = q;
    for (int d = 0; d < nkeys; d++) {
        const int dx = off[d] / 49 - 3, dy = (off[d] / 7) % 7 - 3, dz = off[d] % 7 - 3;
        const int key = which == PASS_M2L ? (dz + 8) * 1000 + dx * dx + dy * dy : d & 1;
        const size_t c = std::find(seen.begin(), seen.end(), key) - seen.begin();
        if (c == seen.size()) {
            seen.push_back(key);
            rep.push_back(d);
        }
        cls[d] = (int)c;
    }
}

// Folded rotation tables of the classes (M2L, then M2M and L2L), padded coaxial tables, and the
// coefficient pairs (n, m >= 0).
static int build_tile_tables(Plan *P)
{
    const int pmax = P->pmax;
    std::vector<int> cls, rep, rows, off(pmax + 1, 0);
    for (int which : {PASS_M2L, PASS_M2M, PASS_L2L}) {
        direction_classes(P, which, which == PASS_M2L ? NDIR : 8, cls, rep);
        if (which == PASS_M2L) P->rot32_m2l = (int)rep.size();
        for (int r : rep) rows.push_back((which == PASS_M2L ? 0 : which == PASS_M2M ? NDIR : NDIR + 8) + r);
    }
    for (int n = 0; n < pmax; n++) off[n + 1] = off[n] + (n + 1) * up_to(n + 1, 4) + n * up_to(n, 4);
    P->rot32_stride = rot32_size(pmax);
    FMM_CUDA_TRY(dev_alloc(P, (void **)&P->rot32, sizeof(float) * rows.size() * (size_t)P->rot32_stride));
    int *tmp = nullptr;
    FMM_CUDA_TRY(cudaMalloc(&tmp, sizeof(int) * (rows.size() + off.size())));
    cudaError_t ce = cudaMemcpy(tmp, rows.data(), sizeof(int) * rows.size(), cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaMemcpy(tmp + rows.size(), off.data(), sizeof(int) * off.size(), cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) {
        rot32_table_kernel<<<dim3(pmax, (unsigned)rows.size()), 128, 0, P->stream>>>(pmax, tmp, tmp + rows.size(), P->rot32_stride,
                                                                                    P->Hsr64, P->rot32);
        ce = cudaStreamSynchronize(P->stream);
    }
    cudaFree(tmp);
    FMM_CUDA_TRY(ce);
    for (int l = P->lmin; l <= P->lmax; l++) {
        LevelDev &L = P->lev[l];
        FMM_CUDA_TRY(dev_alloc(P, (void **)&L.Csr32p, sizeof(float2) * NDIST * (size_t)coax2_size(L.p)));
        coax2_table_kernel<<<dim3(L.p, NDIST), 128, 0, P->stream>>>(L.p, L.Csr32, L.Csr32p);
        if (l > P->lmin) {
            const int pp = P->lev[l - 1].p;
            FMM_CUDA_TRY(dev_alloc(P, (void **)&L.Crr32p, sizeof(float2) * coax2_size(pp)));
            coax2_table_kernel<<<dim3(pp, 1), 128, 0, P->stream>>>(pp, L.Crr32, L.Crr32p);
            if (L.Crr32L) {
                FMM_CUDA_TRY(dev_alloc(P, (void **)&L.Crr32Lp, sizeof(float2) * coax2_size(pp)));
                coax2_table_kernel<<<dim3(pp, 1), 128, 0, P->stream>>>(pp, L.Crr32L, L.Crr32Lp);
            }
        }
    }
    FMM_CUDA_TRY(cudaGetLastError());
    std::vector<int> pairs;
    P->rot32_off = off;
    for (int n = 0; n < pmax; n++)
        for (int m = 0; m <= n; m++) pairs.push_back((n * n + n) | m << 16);
    FMM_CUDA_TRY(dev_alloc(P, (void **)&P->pairs, sizeof(int) * pairs.size()));
    FMM_CUDA_TRY(upload(P->pairs, pairs.data(), sizeof(int) * pairs.size()));
    return FMM_OK;
}

// whole rotation tables of the classes' representative rows rep[k] of H (see whole_off)
__global__ void whole_table_kernel(int pmax, const int *__restrict__ rep, const float *__restrict__ H, float *__restrict__ out)
{
    const int n = blockIdx.x, k = blockIdx.y, w = 2 * n + 1, ld = pad4(w);
    const float *Hn = H + (size_t)rep[k] * rot_size(pmax) + rot_off(n);
    float *o = out + (size_t)k * whole_off(pmax) + whole_off(n);
    for (int t = threadIdx.x; t < w * ld; t += blockDim.x) o[t] = t % ld < w ? Hn[t / ld * w + t % ld] : 0.f;
}

int ensure_whole_tables(Plan *P)
{
    if (P->rot32_whole) return FMM_OK;
    std::vector<int> rows, cls, rep;
    for (int which : {PASS_M2L, PASS_M2M, PASS_L2L}) {
        direction_classes(P, which, which == PASS_M2L ? NDIR : 8, cls, rep);
        for (int r : rep) rows.push_back((which == PASS_M2L ? 0 : which == PASS_M2M ? NDIR : NDIR + 8) + r);
    }
    int *tmp = nullptr;
    float *tab = nullptr;
    FMM_CUDA_TRY(cudaMalloc(&tmp, sizeof(int) * rows.size()));
    cudaError_t ce = dev_alloc(P, (void **)&tab, sizeof(float) * (rows.size() * (size_t)whole_off(P->pmax) + TABLE_PAD));
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(tmp, rows.data(), sizeof(int) * rows.size(), cudaMemcpyHostToDevice, P->stream);
    if (ce == cudaSuccess) {
        whole_table_kernel<<<dim3(P->pmax, (unsigned)rows.size()), 128, 0, P->stream>>>(P->pmax, tmp, P->Hsr32, tab);
        ce = cudaStreamSynchronize(P->stream);
    }
    cudaFree(tmp);
    FMM_CUDA_TRY(ce);
    P->rot32_whole = tab;
    return FMM_OK;
}

// Rounds of a stage's work units: blocks (all units of one degree or order and sign) in the given
// order, longest first, as many as fit the UC units of a round; idle places elsewhere.
template <class U>
static int pack_rounds(const std::vector<std::vector<U>> &blocks, int UC, U idle, std::vector<U> &out)
{
    int rounds = 0, left = 0;
    for (const std::vector<U> &b : blocks) {
        if (b.empty()) continue;
        if ((int)b.size() > left) {
            out.resize(out.size() + left, idle);
            left = UC;
            rounds++;
        }
        out.insert(out.end(), b.begin(), b.end());
        left -= (int)b.size();
    }
    out.resize(out.size() + left, idle);
    return rounds;
}

// The work units of a form's tile shape, on the device (kept until the shape changes).
static int ensure_units(const std::vector<int> &rot_off, TileForm &f, bool fold, const RcrPass &ps)
{
    if (f.units_tc == f.tc && f.units_bal == f.bal) return FMM_OK;
    const int UC = THREADS / (f.tc / CG), R = f.bal ? 2 : 4, nin = std::min(ps.pin, ps.p), nq = std::min(ps.pout, ps.p);
    std::vector<int2> ur;
    std::vector<int> uc;
    auto rot = [&](int deg) {
        std::vector<std::vector<int2>> blocks;
        for (int n = deg - 1; n >= 0; n--)
            for (int sg = 0; sg < (fold ? 2 : 1); sg++) {
                const int nr = !fold ? 2 * n + 1 : sg ? n : n + 1;
                const int base = fold ? rot_off[n] + (sg ? (n + 1) * up_to(n + 1, 4) : 0) : whole_off(n);
                std::vector<int2> b;
                for (int r = 0; r < nr; r += R) b.push_back(make_int2(n | sg << 8 | r << 16, base + r));
                blocks.push_back(b);
            }
        return pack_rounds(blocks, UC, make_int2(-1, 0), ur);
    };
    f.n1 = rot(nin);
    f.at3 = ur.size();
    f.n3 = rot(nq);
    std::vector<std::vector<int>> blocks;
    for (int am = 0; am < nq; am++)
        for (int sg = 0; sg < (am ? 2 : 1); sg++) {
            std::vector<int> b;
            for (int r = 0; r < nq - am; r += 2) b.push_back(am | sg << 8 | r << 16);
            blocks.push_back(b);
        }
    f.n2 = pack_rounds(blocks, UC, -1, uc);
    cudaFree(f.urot);
    cudaFree(f.ucoax);
    f.urot = nullptr;
    f.ucoax = nullptr;
    f.units_tc = 0;
    FMM_CUDA_TRY(cudaMalloc(&f.urot, sizeof(int2) * ur.size()));
    FMM_CUDA_TRY(cudaMalloc(&f.ucoax, sizeof(int) * uc.size()));
    FMM_CUDA_TRY(upload(f.urot, ur.data(), sizeof(int2) * ur.size()));
    FMM_CUDA_TRY(upload(f.ucoax, uc.data(), sizeof(int) * uc.size()));
    f.units_tc = f.tc;
    f.units_bal = f.bal;
    return FMM_OK;
}

// The tile kernels' tables, order of the translations and units of a pass
int set_tile_tables(const Plan *P, RcrList &Lst, int form, RcrPass &ps)
{
    TileForm &f = Lst.form[form];
    const bool fold = form == FORM_FOLDED;
    int e = fold ? ensure_classes(Lst) : FMM_OK;
    if (!e) e = ensure_units(P->rot32_off, f, fold, ps);
    if (e) return e;
    ps.rot_stride = fold ? P->rot32_stride : whole_off(P->pmax);
    ps.rot = (fold ? P->rot32 : P->rot32_whole) + (size_t)Lst.rot0 * ps.rot_stride;
    ps.PHall = P->PHsr32;
    ps.u1 = f.urot;
    ps.n1 = f.n1;
    ps.u3 = f.urot + f.at3;
    ps.n3 = f.n3;
    ps.u2 = f.ucoax;
    ps.n2 = f.n2;
    ps.pairs = P->pairs;
    ps.g_src = fold ? Lst.csrc : Lst.src;
    ps.g_dst = fold ? Lst.cdst : Lst.dst;
    ps.g_dir = fold ? Lst.cdir : nullptr;
    ps.key0 = Lst.key0;
    return FMM_OK;
}

// drank: Morton rank of each destination box among the ndst boxes of its level.  The list is
// sorted by key, and within a key by the destination's Morton rank (two stable counting sorts).
static int upload_list(Plan *P, RcrList &Lst, int which, const std::vector<int> &key, const std::vector<int> &src,
                       const std::vector<int> &dst, int nkeys, const std::vector<int> &key_w, int p,
                       const std::vector<int> &drank, int ndst)
{
    size_t T = key.size();
    std::vector<int> byrank(std::max<size_t>(T, 1));
    {
        std::vector<int> rc(ndst + 1, 0);
        for (size_t i = 0; i < T; i++) rc[drank[dst[i]] + 1]++;
        for (int r = 0; r < ndst; r++) rc[r + 1] += rc[r];
        for (size_t i = 0; i < T; i++) byrank[rc[drank[dst[i]]]++] = (int)i;
    }
    std::vector<int> cnt(nkeys + 1, 0);
    for (size_t i = 0; i < T; i++) cnt[key[i] + 1]++;
    for (int d = 0; d < nkeys; d++) cnt[d + 1] += cnt[d];
    std::vector<int> gs(std::max<size_t>(T, 1)), gd(std::max<size_t>(T, 1)), fill(nkeys, 0);
    Lst.dst_rank.assign(T, 0);
    for (size_t q = 0; q < T; q++) {
        const int i = byrank[q];
        int pos = cnt[key[i]] + fill[key[i]]++;
        gs[pos] = src[i];
        gd[pos] = dst[i];
        Lst.dst_rank[pos] = drank[dst[i]];
    }
    Lst.ndst_rank = ndst;
    Lst.key_beg.assign(cnt.begin(), cnt.end());
    Lst.key_w = key_w;
    Lst.form[FORM_FOLDED].tc = pick_tile(p);
    // half as many: fewer directions in flight at a time, and four CTAs on an SM; all at orders up to 6, whose tiles
    // are small and the work of a column little (33 columns on 5,120 triangles, orders 5, 4, 3: 417 us against 619,
    // 567 in the former tiles; orders 8, 7, 6: 440 against 424)
    Lst.form[FORM_WHOLE].tc = p <= 6 ? pick_tile(p) : std::max(4, pick_tile(p) / 2);
    Lst.rot0 = which == PASS_M2L ? 0 : which == PASS_M2M ? P->rot32_m2l : P->rot32_m2l + 2;
    Lst.key0 = which == PASS_M2L ? 0 : which == PASS_M2M ? NDIR : NDIR + 8;
    {
        std::vector<int> rep;
        direction_classes(P, which, nkeys, Lst.cls_of_key, rep);
    }
    if (T == 0) return FMM_OK;
    FMM_CUDA_TRY(dev_alloc(P, (void **)&Lst.src, sizeof(int) * T));
    FMM_CUDA_TRY(dev_alloc(P, (void **)&Lst.dst, sizeof(int) * T));
    FMM_CUDA_TRY(upload(Lst.src, gs.data(), sizeof(int) * T));
    FMM_CUDA_TRY(upload(Lst.dst, gd.data(), sizeof(int) * T));
    return FMM_OK;
}

// Work lists of the batched passes: per level, the M2L translations grouped by direction,
// the M2M pairs (box -> parent) and the L2L pairs (parent -> box) grouped by octant.
int build_rcr_lists(Plan *P)
{
    int e = build_tile_tables(P);
    if (e) return e;
    // Morton rank of every box of every level (the level sets hold the boxes' Morton numbers
    // in first-occurrence order)
    std::vector<std::vector<int>> rank(P->lmax + 1);
    for (int l = P->lmin; l <= P->lmax; l++) {
        const std::vector<long long> &keys = P->tree.sets[l];
        std::vector<int> ord(keys.size());
        for (size_t i = 0; i < ord.size(); i++) ord[i] = (int)i;
        std::sort(ord.begin(), ord.end(), [&](int a, int b) { return keys[a] < keys[b]; });
        rank[l].assign(keys.size(), 0);
        for (size_t r = 0; r < ord.size(); r++) rank[l][ord[r]] = (int)r;
    }
    for (int l = P->lmin; l <= P->lmax; l++) {
        LevelDev &L = P->lev[l];
        if (L.num_sr > 0) {
            long long T = L.num_sr;
            std::vector<int> beg(L.nb + 1), src(T), dst(T), key(T);
            std::vector<short> dir(T);
            FMM_CUDA_TRY(cudaMemcpy(beg.data(), L.sr_beg, sizeof(int) * (L.nb + 1), cudaMemcpyDeviceToHost));
            FMM_CUDA_TRY(cudaMemcpy(src.data(), L.sr_src, sizeof(int) * T, cudaMemcpyDeviceToHost));
            FMM_CUDA_TRY(cudaMemcpy(dir.data(), L.sr_dir, sizeof(short) * T, cudaMemcpyDeviceToHost));
            for (int b = 0; b < L.nb; b++)
                for (int t = beg[b]; t < beg[b + 1]; t++) {
                    dst[t] = b;
                    key[t] = dir[t];
                }
            std::vector<int> kw(P->dir_dist, P->dir_dist + NDIR);
            int st = upload_list(P, L.m2l, PASS_M2L, key, src, dst, NDIR, kw, L.p, rank[l], L.nb);
            if (st) return st;
        }
        if (l > P->lmin) {
            LevelDev &PL = P->lev[l - 1];
            std::vector<int> par(L.nb), key(L.nb), self(L.nb);
            std::vector<unsigned char> oct(L.nb);
            FMM_CUDA_TRY(cudaMemcpy(par.data(), L.parent, sizeof(int) * L.nb, cudaMemcpyDeviceToHost));
            FMM_CUDA_TRY(cudaMemcpy(oct.data(), L.octant, L.nb, cudaMemcpyDeviceToHost));
            for (int b = 0; b < L.nb; b++) {
                key[b] = oct[b];
                self[b] = b;
            }
            std::vector<int> kw(8, 0);
            int st = upload_list(P, L.m2m, PASS_M2M, key, self, par, 8, kw, PL.p, rank[l - 1], PL.nb);
            if (st) return st;
            st = upload_list(P, L.l2l, PASS_L2L, key, par, self, 8, kw, PL.p, rank[l], L.nb);
            if (st) return st;
        }
    }
    return FMM_OK;
}

// Columns and rows per unit of a pass, by timing on this plan's own list and tables (one right-hand side): the
// columns of pick_tile, half and a quarter of them (passes of few translations fill more SMs with narrower
// tiles), units of four rows, or of two (more units for the threads of a narrow tile).  Matvec results do not
// depend on the choice beyond the order of the FP32 atomic additions.
static int tune_list(Plan *P, int l, int which, RcrList &Lst)
{
    TileForm &f = Lst.form[FORM_FOLDED];
    if (f.tuned || Lst.key_beg.empty() || Lst.key_beg.back() == 0) return FMM_OK;
    std::vector<int2> cand;
    for (int tc = f.tc; tc >= 4 && 4 * tc >= f.tc; tc /= 2)
        for (int bal = 0; bal < 2; bal++) cand.push_back({tc, bal});
    cudaEvent_t a = nullptr, b = nullptr;
    float best = 1e30f;
    int2 pick = cand[0];
    int rc = FMM_OK;
    auto timed = [&](float *ms) -> int {
        FMM_CUDA_TRY(cudaEventRecord(a, P->stream));
        if (int e = launch_pass32(P, l, which, 1, P->stream)) return e;
        FMM_CUDA_TRY(cudaEventRecord(b, P->stream));
        FMM_CUDA_TRY(cudaEventSynchronize(b));
        FMM_CUDA_TRY(cudaEventElapsedTime(ms, a, b));
        return FMM_OK;
    };
    if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) {
        fmm_set_error("tile tuning: %s", cudaGetErrorString(cudaGetLastError()));
        rc = FMM_ERR_CUDA;
    }
    const int dense = Lst.td.on;
    Lst.td.on = 0;
    for (auto &c : cand) {
        f.tc = c.x;
        f.bal = c.y;
        f.items_nrhs = 0;
        float tot = 0.f;
        for (int rep = 0; rep < 4 && rc == FMM_OK; rep++) {
            float ms = 0.f;
            rc = timed(&ms);
            if (rep > 0) tot += ms;
        }
        if (rc != FMM_OK) break;
        if (tot < best) {
            best = tot;
            pick = c;
        }
    }
    Lst.td.on = dense;
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
    f.tc = pick.x;
    f.bal = pick.y;
    f.items_nrhs = 0;
    f.tuned = rc == FMM_OK;
    return rc;
}

// The tile shapes of a plan's passes, at plan creation.  Passes that run in the dense tensor-core form are left to
// scenes (dense_too), which run all passes on the tiles: with the widest tile and units of four rows instead of what
// timing picks there, 16 spheres of 2,420 triangles took 560 us for 482.
int tune_rcr_tiles(Plan *P, bool dense_too)
{
    // FMMBEM_TILE_BAL=0/1/2 forces one shape on every pass, for tests: 0 the columns of pick_tile and
    // units of four rows, 1 units of two rows, 2 half the columns and units of two rows
    if (const char *env = dense_too ? nullptr : getenv("FMMBEM_TILE_BAL")) {
        const int bal = std::max(0, std::min(2, atoi(env)));
        for (int l = P->lmin; l <= P->lmax; l++)
            for (RcrList *R : {&P->lev[l].m2m, &P->lev[l].m2l, &P->lev[l].l2l})
                for (TileForm &f : R->form) {
                    f.bal = bal ? 1 : 0;
                    if (bal == 2) f.tc = std::max(4, f.tc / 2);
                    f.items_nrhs = 0;
                    f.tuned = true;
                }
        return FMM_OK;
    }
    for (int l = P->lmin; l <= P->lmax; l++) {
        LevelDev &L = P->lev[l];
        for (int which = PASS_M2M; which <= PASS_L2L; which++) {
            if (which != PASS_M2L && l == P->lmin) continue;
            RcrList &Lst = which == PASS_M2M ? L.m2m : which == PASS_M2L ? L.m2l : L.l2l;
            if (Lst.td.on && !dense_too) continue;
            if (int e = tune_list(P, l, which, Lst)) return e;
        }
    }
    return FMM_OK;
}
} // namespace fmm
