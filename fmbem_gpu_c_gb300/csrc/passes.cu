// The FMM matvec: P2M, translations, L2P + near field.  Templated on the arithmetic type: double
// for the plain path, float for the mixed-precision path.
//
// Every translation is rotation - coaxial - rotation (RCR) as in the reference
// (transMatsVecsMul_SR_rcr, translation.cu:1864-1961): rotate by (phi, theta, 0), apply the
// coaxial blocks for |t|, rotate back by (0, theta, phi).  The rotation matrix is
// e^{i m alpha} e^{-i m' gamma} H_n^{m'm}(beta) (translation.cu:1221-1235), so one real
// table H per direction serves both rotations and the phases are applied elementwise.
// The FP64 path, its float-float form (FMM_FLOAT2) and deterministic mixed plans run the
// translations of owner.cu (no atomics, bit-reproducible).  The mixed path runs the batched
// direction-grouped tiles of batched.cu, which add into the expansions with FP32 atomics, so
// mixed results vary in the last bits from run to run.
#include "plan.h"
#include "ff.cuh"
#include <algorithm>
#include <vector>
#include <type_traits>

namespace fmm {

__constant__ int c_dir_dist[NDIR];

template <typename T> struct Cx;
template <> struct Cx<double> { typedef double2 t; };
template <> struct Cx<float> { typedef float2 t; };

__device__ __forceinline__ void decode_nm(int i, int &n, int &m)
{
    int q = (int)sqrtf((float)i);
    while (q * q > i) q--;
    while ((q + 1) * (q + 1) <= i) q++;
    n = q;
    m = i - q * q - q;
}

__device__ __forceinline__ float2 to_c(double2 v, float) { return make_float2((float)v.x, (float)v.y); }
__device__ __forceinline__ double2 to_c(double2 v, double) { return v; }
__device__ __forceinline__ double2 to_d(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ double2 to_d(double2 v) { return v; }

// One RCR translation by a whole CTA.  x has pin^2 entries (zero padded to p); the result
// for n < pout is accumulated into sY.  H and ph are the direction's real rotation table
// (stride rot_size(pmax), prefix order p) and phases e^{i m phi} indexed m + pmax - 1.
__device__ void rcr_block(int p, int pmax, const double *__restrict__ H, const double2 *__restrict__ ph,
                          const double2 *__restrict__ Cc, const double2 *__restrict__ xin, int pin,
                          double2 *sX, double2 *sW1, double2 *sW2,
                          double2 *sY, int pout)
{
    const int pp = p * p, pin2 = pin * pin, tid = threadIdx.x, nt = blockDim.x, off = pmax - 1;
    for (int i = tid; i < pp; i += nt) {
        int n, m;
        decode_nm(i, n, m);
        double2 v = (i < pin2) ? xin[i] : mk2(0.0, 0.0);
        sX[i] = cmul(v, ph[m + off]);
    }
    __syncthreads();
    for (int i = tid; i < pp; i += nt) {
        int n, mp;
        decode_nm(i, n, mp);
        const double *col = H + rot_off(n) + (mp + n);
        const int w = 2 * n + 1, base = n * n;
        double ar = 0, ai = 0;
        for (int m = 0; m < w; m++) {
            double h = col[m * w];
            double2 v = sX[base + m];
            ar += h * v.x;
            ai += h * v.y;
        }
        sW1[i] = mk2(ar, ai);
    }
    __syncthreads();
    for (int i = tid; i < pp; i += nt) {
        int np, m;
        decode_nm(i, np, m);
        int am = m < 0 ? -m : m, sz = p - am;
        const double2 *col = Cc + coax_off(p, am) + (np - am);
        double ar = 0, ai = 0;
        for (int n = am; n < p; n++) {
            double2 c = col[(n - am) * sz];
            double2 v = sW1[n * n + n + m];
            ar += c.x * v.x - c.y * v.y;
            ai += c.x * v.y + c.y * v.x;
        }
        sW2[i] = mk2(ar, ai);
    }
    __syncthreads();
    const int po2 = min(p, pout) * min(p, pout);  // no outputs beyond the translation's order
    for (int i = tid; i < po2; i += nt) {
        int n, mp;
        decode_nm(i, n, mp);
        const double *col = H + rot_off(n) + (mp + n);
        const int w = 2 * n + 1, base = n * n;
        double ar = 0, ai = 0;
        for (int m = 0; m < w; m++) {
            double h = col[m * w];
            double2 v = sW2[base + m];
            ar += h * v.x;
            ai += h * v.y;
        }
        double2 e = ph[mp + off];
        // conj(e) * (ar + i ai)
        double2 y = sY[i];
        y.x += e.x * ar + e.y * ai;
        y.y += e.x * ai - e.y * ar;
        sY[i] = y;
    }
    __syncthreads();
}

// flip = 0: C_b[n,m] = ik sum_e x_e U_e[n,m] (element moments of R_n^{-m}).
// flip = 1 (transposed operator): the same with the table read at (n,-m); with U = Rv this
// is the multipole expansion ik sum_i y_i R_n^{-m}(y_i - c) of point sources at centroids.
// P2M of one leaf box (CTA) for a group of up to G right-hand sides (blockIdx.y): thread i takes
// coefficient i; the box's elements and their i k x_e are staged in shared memory once, so that
// the loads of U depend on shared memory only and can all be in flight together, and each U
// entry serves the whole group.  Each column's sum runs in the same order whatever the group.
// With x32 given, the CTA also writes its elements' x in FP32 there (every element lies in one
// leaf), for the gathers of the L2P + near-field pass: GB300 converts FP64 to FP32 at its FP64
// rate, and the near field would otherwise convert each x once per near pair.
// The blocks behind the leaf boxes zero the expansions that the translations add to (a memset per
// level and kind, one after another, was 5 us of a 50 us matvec on 320 triangles).
struct ZeroList {
    float4 *ptr[2 * (FMM_MAX_LEVEL + 2)];
    unsigned end[2 * (FMM_MAX_LEVEL + 2)];          // blocks up to and with this entry
    unsigned long long n[2 * (FMM_MAX_LEVEL + 2)];  // 16-byte words
    unsigned words;                                 // per block: 16 KB, more where that takes over 64 blocks per SM
    int count;
};

template <typename T, int G>
__global__ void p2m_kernel(int pl, const int *__restrict__ leaf_beg, const int *__restrict__ leaf_elem,
                           const typename Cx<T>::t *__restrict__ U, const double2 *__restrict__ x, double k,
                           typename Cx<T>::t *__restrict__ Cm, int flip, int nf, int nb, int nrhs,
                           float2 *__restrict__ x32, const __grid_constant__ ZeroList zero)
{
    typedef typename Cx<T>::t C;
    if ((int)blockIdx.x >= nb) {
        if (blockIdx.y) return;
        unsigned z = blockIdx.x - nb, first = 0;
        int i = 0;
        while (z >= zero.end[i]) first = zero.end[i++];
        const unsigned long long w0 = (unsigned long long)(z - first) * zero.words;
        for (unsigned long long w = w0 + threadIdx.x; w < min(w0 + zero.words, zero.n[i]); w += blockDim.x)
            zero.ptr[i][w] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    constexpr int MAXE = 64;
    __shared__ int s_e[MAXE];
    __shared__ C s_x[MAXE][G];
    const int b = blockIdx.x, ppl = pl * pl, r0 = blockIdx.y * G, ng = min(G, nrhs - r0);
    const int s0 = leaf_beg[b], ne = leaf_beg[b + 1] - s0;
    for (int q = threadIdx.x; q < ne * G; q += blockDim.x) {
        const int j = q / G, g = q % G, e = leaf_elem[s0 + j];
        if (g == 0 && j < MAXE) s_e[j] = e;
        const double2 xe = g < ng ? x[(size_t)(r0 + g) * nf + e] : make_double2(0.0, 0.0);
        if (j < MAXE) s_x[j][g] = mk2((T)(-k * xe.y), (T)(k * xe.x));  // i k x_e
        if (x32 && g < ng) x32[(size_t)e * nrhs + r0 + g] = make_float2((float)xe.x, (float)xe.y);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ppl; i += blockDim.x) {
        int q = i;
        if (flip) {
            int n, m;
            decode_nm(i, n, m);
            q = n * n + n - m;
        }
        T ar[G], ai[G];
#pragma unroll
        for (int g = 0; g < G; g++) ar[g] = ai[g] = 0;
#pragma unroll 4
        for (int j = 0; j < ne && j < MAXE; j++) {
            const C u = U[(size_t)s_e[j] * ppl + q];
#pragma unroll
            for (int g = 0; g < G; g++) {
                const C xe = s_x[j][g];
                ar[g] += xe.x * u.x - xe.y * u.y;
                ai[g] += xe.x * u.y + xe.y * u.x;
            }
        }
        // boxes with more than MAXE elements (none at the usual leaf occupancy): the rest directly
        for (int j = MAXE; j < ne; j++) {
            const int e = leaf_elem[s0 + j];
            const C u = U[(size_t)e * ppl + q];
#pragma unroll
            for (int g = 0; g < G; g++) {
                if (g >= ng) break;
                const double2 xd = x[(size_t)(r0 + g) * nf + e];
                const T xr = (T)(-k * xd.y), xi = (T)(k * xd.x);
                ar[g] += xr * u.x - xi * u.y;
                ai[g] += xr * u.y + xi * u.x;
            }
        }
#pragma unroll
        for (int g = 0; g < G; g++) {
            if (g >= ng) break;
            Cm[((size_t)b * nrhs + r0 + g) * ppl + i] = mk2(ar[g], ai[g]); // [box][rhs][p^2]
        }
    }
}

__global__ void to_float_kernel2(const double *in, float *out, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = (float)in[i];
}

// L2P + near field + identity for element e (one warp) and a group of up to G right-hand sides
// (blockIdx.y): the near row and the element's basis are loaded once for the group, the x
// gathers and the local expansions per right-hand side.  Each column's sums run in the same
// order whatever the group, so a column's result does not depend on nrhs.  T = float gathers
// the near field's x from x32, the FP32 copy P2M wrote (the same values as converting x here), a
// column group of an element together (with a column's entries together a 32-byte sector was read for
// each 8 bytes).
// The identity's FP64 arithmetic runs once for a block's 8 elements and all their columns, a lane each: an FP64
// instruction takes the pipe 16 cycles whatever lanes are on, and one lane per element and column was
// half of the kernel.  64 columns on the 200,000-triangle head 6.8 -> 3.4 ms, 16 on the 81,920-triangle
// sphere 0.85 -> 0.47 ms; what is left is the latency of the gathers (22 % of the issue slots used).
constexpr int L2P_WARPS = 8;
template <typename T, int G>
__global__ void __launch_bounds__(32 * L2P_WARPS) l2p_near_kernel(int nf, int pl, const int *__restrict__ elem_leaf, const typename Cx<T>::t *__restrict__ Dl,
                                const typename Cx<T>::t *__restrict__ Rv, const int *__restrict__ near_beg,
                                const int *__restrict__ near_col, const typename Cx<T>::t *__restrict__ nearv,
                                const double2 *__restrict__ x, const float2 *__restrict__ x32, double2 a,
                                double2 *__restrict__ y, int flip, int nb, int nrhs)
{
    typedef typename Cx<T>::t C;
    __shared__ C s_sum[L2P_WARPS][G];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e0 = blockIdx.x * L2P_WARPS, e = min(e0 + warp, nf - 1);
    const int r0 = blockIdx.y * G, ng = min(G, nrhs - r0);
    int ppl = pl * pl;
    const bool whole = ng == G && nrhs % 2 == 0;  // a group's columns of an element lie on 16 bytes
    T ar[G], ai[G];
#pragma unroll
    for (int g = 0; g < G; g++) ar[g] = ai[g] = 0;
    for (int s = near_beg[e] + lane; s < near_beg[e + 1]; s += 32) {
        const C v = nearv[s];
        const int col = near_col[s];
        if constexpr (sizeof(T) == 4 && G % 2 == 0) {
            if (whole) {
                const float4 *xc = reinterpret_cast<const float4 *>(x32 + (size_t)col * nrhs + r0);
                float4 xg[G / 2];
#pragma unroll
                for (int g = 0; g < G / 2; g++) xg[g] = xc[g];
#pragma unroll
                for (int g = 0; g < G; g += 2) {
                    const float4 xf = xg[g / 2];
                    ar[g] += v.x * xf.x - v.y * xf.y;
                    ai[g] += v.x * xf.y + v.y * xf.x;
                    ar[g + 1] += v.x * xf.z - v.y * xf.w;
                    ai[g + 1] += v.x * xf.w + v.y * xf.z;
                }
                continue;
            }
        }
#pragma unroll
        for (int g = 0; g < G; g++) {
            if (g >= ng) break;
            T xr, xi;
            if constexpr (sizeof(T) == 4) {
                const float2 xf = x32[(size_t)col * nrhs + r0 + g];
                xr = xf.x;
                xi = xf.y;
            } else {
                const double2 xd = x[(size_t)(r0 + g) * nf + col];
                xr = xd.x;
                xi = xd.y;
            }
            ar[g] += v.x * xr - v.y * xi;
            ai[g] += v.x * xi + v.y * xr;
        }
    }
    const C *R = Rv + (size_t)e * ppl;
    const size_t db = (size_t)elem_leaf[e] * nrhs; // [box][rhs][p^2]
    for (int i = lane; i < ppl; i += 32) {
        int q = i;
        if (flip) {
            int n, m;
            decode_nm(i, n, m);
            q = n * n + n - m;
        }
        const C r = R[q];
        // (columns past the last read the last one's: loads without a branch between them are in flight together)
        C d[G];
#pragma unroll
        for (int g = 0; g < G; g++) d[g] = Dl[(db + r0 + min(g, ng - 1)) * ppl + i];
#pragma unroll
        for (int g = 0; g < G; g++) {
            ar[g] += d[g].x * r.x - d[g].y * r.y;
            ai[g] += d[g].x * r.y + d[g].y * r.x;
        }
    }
#pragma unroll
    for (int g = 0; g < G; g++) {
        if (g >= ng) break;
        T sr = ar[g], si = ai[g];
        for (int o = 16; o > 0; o >>= 1) {
            sr += __shfl_xor_sync(0xffffffffu, sr, o);
            si += __shfl_xor_sync(0xffffffffu, si, o);
        }
        if (lane == g) s_sum[warp][g] = mk2(sr, si);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < L2P_WARPS * ng; q += 32 * L2P_WARPS) {
        const int w = q % L2P_WARPS, g = q / L2P_WARPS;
        if (e0 + w >= nf) continue;
        const size_t k = (size_t)(r0 + g) * nf + e0 + w;
        const double2 xe = x[k];
        const C s = s_sum[w][g];
        y[k] = make_double2(a.x * xe.x - a.y * xe.y + (double)s.x, a.x * xe.y + a.y * xe.x + (double)s.y);
    }
}

static void timer_begin(Plan *P, const char *name, cudaStream_t st = nullptr)
{
    if (P->profiling != 1 || P->ntimers >= MAX_TIMERS) return;
    Timer &t = P->timers[P->ntimers];
    t.name = name;
    cudaEventRecord(t.beg, st ? st : P->stream);
}
static void timer_end(Plan *P, cudaStream_t st = nullptr)
{
    if (P->profiling != 1 || P->ntimers >= MAX_TIMERS) return;
    cudaEventRecord(P->timers[P->ntimers].end, st ? st : P->stream);
    P->ntimers++;
}

static const char *pass_names[3][14] = {
    {"m2m_l0", "m2m_l1", "m2m_l2", "m2m_l3", "m2m_l4", "m2m_l5", "m2m_l6", "m2m_l7", "m2m_l8", "m2m_l9", "m2m_l10",
     "m2m_l11", "m2m_l12", "m2m_l13"},
    {"m2l_l0", "m2l_l1", "m2l_l2", "m2l_l3", "m2l_l4", "m2l_l5", "m2l_l6", "m2l_l7", "m2l_l8", "m2l_l9", "m2l_l10",
     "m2l_l11", "m2l_l12", "m2l_l13"},
    {"l2l_l0", "l2l_l1", "l2l_l2", "l2l_l3", "l2l_l4", "l2l_l5", "l2l_l6", "l2l_l7", "l2l_l8", "l2l_l9", "l2l_l10",
     "l2l_l11", "l2l_l12", "l2l_l13"}};
static void pass_begin(Plan *P, int which, int l) { timer_begin(P, pass_names[which][l]); }
static void pass_end(Plan *P) { timer_end(P); }

// ---------------------------------------------------------------- float-float tables (FMM_FLOAT2)
__global__ void ff_from_cplx_kernel(const double2 *__restrict__ in, float4 *__restrict__ out, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const ff a = ff_from(in[i].x), b = ff_from(in[i].y);
        out[i] = make_float4(a.hi, a.lo, b.hi, b.lo);
    }
}
static unsigned ew_grid(size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 152 * 16); }

// coaxial tables of order p (layout of coax_off; blockIdx.x = m, blockIdx.y = table) in
// float-float, every part twice (the operands of the packed instructions in owner.cu): two
// float4 per entry, (re hi, re hi, re lo, re lo) and the same of im; rows times row[n'] and
// columns times col[n] where given
__global__ void ff_coax_kernel(const double2 *__restrict__ in, float4 *__restrict__ out, int p, const double *__restrict__ row,
                               const double *__restrict__ col)
{
    const int m = blockIdx.x, sz = p - m;
    const size_t off = (size_t)blockIdx.y * coax_size(p) + coax_off(p, m);
    for (int i = threadIdx.x; i < sz * sz; i += blockDim.x) {
        const double f = row ? row[m + i % sz] * col[m + i / sz] : 1.0;
        const double2 c = in[off + i];
        const ff x = ff_from(c.x * f), y = ff_from(c.y * f);
        out[2 * (off + i)] = make_float4(x.hi, x.hi, x.lo, x.lo);
        out[2 * (off + i) + 1] = make_float4(y.hi, y.hi, y.lo, y.lo);
    }
}

// The float-float copies of the translation tables (phases, coaxial blocks; the rotations: owner.cu) and
// the expansions, made on first use.  Where the FP32 mixed tables are built, the FP32 exponent
// range holds them: plain, or scaled by degree as the FP32 ones (multipoles d_n M_n, locals
// L_n / d_n, the coaxial tables scaled to match, the leaf expansions scaled on the way in and
// out); elsewhere FMM_FLOAT2 runs FMM_FP64.
static int ensure_ff(Plan *P)
{
    if (P->ff_ready) return FMM_OK;
    if (!P->opt.build_mixed || !P->U32) {
        P->ff_ready = -1;
        return FMM_OK;
    }
    const size_t nph = (size_t)(NDIR + 16) * (2 * P->pmax - 1);
    FMM_CUDA_TRY(dev_alloc(P, (void **)&P->PHall_ff, sizeof(float4) * nph));
    ff_from_cplx_kernel<<<ew_grid(nph), 256, 0, P->stream>>>(P->PHsr64, P->PHall_ff, nph);
    // the scalings of the FP32 tables (gen_coax_tables): M2L 1/d^l both sides; M2M rows d^{l-1},
    // columns 1/d^l below the child order (0 above); L2L rows 1/d^l below the child order (0
    // above), columns d^{l-1}; per level on the device: d, 1/d, and 1/d below the level's order
    std::vector<double> sc;
    std::vector<size_t> sc_at(P->lmax + 1, 0);
    double *dsc = nullptr;
    if (P->scaled) {
        for (int l = P->lmin; l <= P->lmax; l++) {
            const std::vector<double> &d = P->dsc[l];
            sc_at[l] = sc.size();
            sc.insert(sc.end(), d.begin(), d.end());
            for (double v : d) sc.push_back(1.0 / v);
            for (int n = 0; n < (int)d.size(); n++) sc.push_back(n < P->lev[l].p ? 1.0 / d[n] : 0.0);
        }
        FMM_CUDA_TRY(cudaMalloc(&dsc, sizeof(double) * sc.size()));
    }
    auto tables = [&]() -> int {
        if (dsc) FMM_CUDA_TRY(cudaMemcpyAsync(dsc, sc.data(), sizeof(double) * sc.size(), cudaMemcpyHostToDevice, P->stream));
        for (int l = P->lmin; l <= P->lmax; l++) {
            LevelDev &L = P->lev[l];
            const size_t ne = (size_t)L.nb * L.p * L.p;
            const double *d = dsc ? dsc + sc_at[l] : nullptr, *inv = dsc ? d + P->dsc[l].size() : nullptr;
            const double *cut = dsc ? inv + P->dsc[l].size() : nullptr;
            FMM_CUDA_TRY(dev_alloc(P, (void **)&L.Csr_ff, 2 * sizeof(float4) * (NDIST * coax_size(L.p) + TABLE_PAD)));
            ff_coax_kernel<<<dim3(L.p, NDIST), 128, 0, P->stream>>>(L.Csr64, L.Csr_ff, L.p, inv, inv);
            if (l > P->lmin) {
                const int pp = P->lev[l - 1].p;
                const double *dp = dsc ? dsc + sc_at[l - 1] : nullptr;
                FMM_CUDA_TRY(dev_alloc(P, (void **)&L.Crr_ff, 2 * sizeof(float4) * (coax_size(pp) + TABLE_PAD)));
                ff_coax_kernel<<<dim3(pp, 1), 128, 0, P->stream>>>(L.Crr64, L.Crr_ff, pp, dp, cut);
                if (dsc) {
                    FMM_CUDA_TRY(dev_alloc(P, (void **)&L.CrrL_ff, 2 * sizeof(float4) * (coax_size(pp) + TABLE_PAD)));
                    ff_coax_kernel<<<dim3(pp, 1), 128, 0, P->stream>>>(L.Crr64, L.CrrL_ff, pp, cut, dp);
                }
            }
            FMM_CUDA_TRY(dev_alloc(P, (void **)&L.Cm_ff, sizeof(float4) * ne));
            FMM_CUDA_TRY(dev_alloc(P, (void **)&L.Dl_ff, sizeof(float4) * ne));
        }
        FMM_CUDA_TRY(cudaGetLastError());
        FMM_CUDA_TRY(cudaStreamSynchronize(P->stream));
        return FMM_OK;
    };
    const int rc = tables();
    cudaFree(dsc);
    if (rc) return rc;
    if (P->scaled) {
        const std::vector<double> &d = P->dsc[P->lmax];
        FMM_CUDA_TRY(dev_alloc(P, (void **)&P->dsc_leaf_dev, sizeof(double) * d.size()));
        FMM_CUDA_TRY(upload(P->dsc_leaf_dev, d.data(), sizeof(double) * d.size()));
    }
    FMM_CUDA_TRY(cudaGetLastError());
    P->ff_ready = 1;
    return FMM_OK;
}

static RcrPass make_pass(int p, int pin, int pout, int atomic, const float *H, int hstride, const float2 *PH,
                         int phstride, int phoff, const float2 *Cc, const float2 *src, float2 *dst, int nrhs, int nsrc,
                         int ndst)
{
    RcrPass ps;
    ps.p = p;
    ps.pin = pin;
    ps.pout = pout;
    ps.atomic = atomic;
    ps.nrhs = nrhs;
    ps.nsrc = nsrc;
    ps.ndst = ndst;
    ps.hstride = hstride;
    ps.phstride = phstride;
    ps.phoff = phoff;
    ps.H = H;
    ps.PH = PH;
    ps.Cc = Cc;
    ps.src = src;
    ps.dst = dst;
    ps.items = nullptr;
    ps.g_src = ps.g_dst = nullptr;
    ps.g_dir = nullptr;
    return ps;
}

// One batched FP32 pass of the mixed path for level l: PASS_M2M (level l into its parents),
// PASS_M2L (level l), PASS_L2L (parents into level l).
RcrList *pass32_desc(Plan *P, int l, int which, int nrhs, RcrPass &ps)
{
    const int pmax = P->pmax, rs = rot_size(pmax), w = 2 * pmax - 1;
    LevelDev &L = P->lev[l];
    if (which == PASS_M2L) {
        ps = make_pass(L.p, L.p, L.p, 1, P->Hsr32, rs, P->PHsr32, w, pmax - 1, L.Csr32, L.Cm32, L.Dl32, nrhs, L.nb, L.nb);
        ps.coax = L.Csr32p;
        return &L.m2l;
    }
    if (l <= P->lmin) return nullptr;
    LevelDev &PL = P->lev[l - 1];
    if (which == PASS_M2M) {
        ps = make_pass(PL.p, L.p, PL.p, 1, P->Hss32, rs, P->PHss32, w, pmax - 1, L.Crr32, L.Cm32, PL.Cm32, nrhs, L.nb,
                       PL.nb);
        ps.coax = L.Crr32p;
        return &L.m2m;
    }
    ps = make_pass(PL.p, PL.p, L.p, 0, P->Hrr32, rs, P->PHrr32, w, pmax - 1, L.Crr32L ? L.Crr32L : L.Crr32, PL.Dl32,
                   L.Dl32, nrhs, PL.nb, L.nb);
    ps.coax = L.Crr32Lp ? L.Crr32Lp : L.Crr32p;
    return &L.l2l;
}

int launch_pass32(Plan *P, int l, int which, int nrhs, cudaStream_t st)
{
    RcrPass ps;
    RcrList *Lst = pass32_desc(P, l, which, nrhs, ps);
    if (Lst && Lst->t3.on) return launch_tc3_pass(P, l, which, nrhs, st);
    if (Lst && Lst->td.on) return launch_tc_dense(P, l, which, nrhs, st);
    return Lst ? launch_rcr_pass(P, *Lst, ps, st) : FMM_OK;
}

// The expansions that the mixed path's translations add to, for nrhs columns: all multipoles above the
// leaves and all locals (each buffer has one coefficient to spare, so whole 16-byte words).
static ZeroList zero_list(const Plan *P, int nrhs)
{
    ZeroList z = {};
    unsigned end = 0;
    unsigned long long all = 0;
    for (int l = P->lmin; l <= P->lmax; l++) all += (unsigned long long)P->lev[l].nb * P->lev[l].p * P->lev[l].p * nrhs;
    z.words = (unsigned)std::max<unsigned long long>(1024, all / (152 * 64));
    for (int l = P->lmin; l <= P->lmax; l++)
        for (int c = l < P->lmax ? 0 : 1; c < 2; c++) {
            const LevelDev &L = P->lev[l];
            z.ptr[z.count] = reinterpret_cast<float4 *>(c ? L.Dl32 : L.Cm32);
            z.n[z.count] = ((unsigned long long)L.nb * L.p * L.p * nrhs + 1) / 2;
            end += (unsigned)((z.n[z.count] + z.words - 1) / z.words);
            z.end[z.count++] = end;
        }
    return z;
}

// The mixed path's translation passes for nrhs columns (into expansions that P2M zeroed): M2M up, the
// M2L of every level forked onto the side streams (one level's tail overlaps the next
// level's work), join, L2L down.  M2M and M2L add into zeroed expansions with atomics; L2L
// then adds the parents' locals top-down.
static int translate32_direct(Plan *P, int nrhs)
{
    const int lmin = P->lmin, lmax = P->lmax;
    cudaStream_t st = P->stream;
    if (P->profiling == 1) {
        cudaEventRecord(P->phase.beg, st);
        P->have_phase = 1;
    }
    for (int l = lmax; l > lmin; l--) {
        timer_begin(P, pass_names[PASS_M2M][l]);
        int e = launch_pass32(P, l, PASS_M2M, nrhs, st);
        if (e) return e;
        timer_end(P);
    }
    // every side stream waits on the fork, also one that gets no pass, so that all of them
    // join a graph capture
    FMM_CUDA_TRY(cudaEventRecord(P->fork_ev, st));
    for (int i = 0; i < P->nside; i++) FMM_CUDA_TRY(cudaStreamWaitEvent(P->side[i], P->fork_ev, 0));
    for (int l = lmin; l <= lmax; l++) {
        cudaStream_t sl = P->side[(l - lmin) % P->nside];
        timer_begin(P, pass_names[PASS_M2L][l], sl);
        int e = launch_pass32(P, l, PASS_M2L, nrhs, sl);
        if (e) return e;
        timer_end(P, sl);
        FMM_CUDA_TRY(cudaEventRecord(P->m2l_ev[l], sl));
    }
    // L2L into level l adds the parents' locals once level l's M2L (and the L2L above it) is
    // complete, so the top of the downward pass overlaps the M2L of the deeper levels
    FMM_CUDA_TRY(cudaStreamWaitEvent(st, P->m2l_ev[lmin], 0));
    for (int l = lmin + 1; l <= lmax; l++) {
        FMM_CUDA_TRY(cudaStreamWaitEvent(st, P->m2l_ev[l], 0));
        timer_begin(P, pass_names[PASS_L2L][l]);
        int e = launch_pass32(P, l, PASS_L2L, nrhs, st);
        if (e) return e;
        timer_end(P);
    }
    for (int i = 0; i < P->nside; i++) {
        FMM_CUDA_TRY(cudaEventRecord(P->join_ev[i], P->side[i]));
        FMM_CUDA_TRY(cudaStreamWaitEvent(st, P->join_ev[i], 0));
    }
    if (P->profiling == 1) cudaEventRecord(P->phase.end, st);
    return FMM_OK;
}

void drop_graph(Plan *P)
{
    if (P->graph_exec) cudaGraphExecDestroy(P->graph_exec);
    P->graph_exec = nullptr;
    P->graph_nrhs = 0;
    P->graph_seen = 0;
}

// Translation passes as a CUDA graph: the second call with the same number of columns
// captures them (the first has built the work items and set the kernels' attributes), later
// calls replay the graph, which saves the ~15 launches per matvec.  Per-pass
// profiling (mode 1) runs the passes directly so that each pass gets its own timer.
static int translate32(Plan *P, int nrhs)
{
    if (P->profiling == 1) return translate32_direct(P, nrhs);
    if (P->graph_exec && P->graph_nrhs == nrhs) {
        FMM_CUDA_TRY(cudaGraphLaunch(P->graph_exec, P->stream));
        return FMM_OK;
    }
    if (P->graph_seen != nrhs) {
        drop_graph(P);
        P->graph_seen = nrhs;
        return translate32_direct(P, nrhs);
    }
    cudaGraph_t g = nullptr;
    FMM_CUDA_TRY(cudaStreamBeginCapture(P->stream, cudaStreamCaptureModeThreadLocal));
    int e = translate32_direct(P, nrhs);
    cudaError_t ce = cudaStreamEndCapture(P->stream, &g);
    if (e) {
        if (g) cudaGraphDestroy(g);
        return e;
    }
    if (ce != cudaSuccess) {
        fmm_set_error("capturing the translation passes: %s", cudaGetErrorString(ce));
        return FMM_ERR_CUDA;
    }
    ce = cudaGraphInstantiate(&P->graph_exec, g, 0);
    cudaGraphDestroy(g);
    if (ce != cudaSuccess) {
        P->graph_exec = nullptr;
        fmm_set_error("instantiating the translation graph: %s", cudaGetErrorString(ce));
        return FMM_ERR_CUDA;
    }
    P->graph_nrhs = nrhs;
    FMM_CUDA_TRY(cudaGraphLaunch(P->graph_exec, P->stream));
    return FMM_OK;
}

// ffm2l (T = double only): the translations in float-float (FMM_FLOAT2)
template <typename T>
static int run_matvec_t(Plan *P, const double2 *x, double2 *y, int transpose, int nrhs, bool ffm2l = false)
{
    typedef typename Cx<T>::t C;
    const bool f64 = sizeof(T) == 8;
    // translations without atomics (owner.cu): the FP64 path, and the mixed path of deterministic plans
    const bool owner = f64 || P->opt.deterministic;
    const int lmax = P->lmax;
    cudaStream_t st = P->stream;
    P->ntimers = 0;
    P->have_total = 0;
    P->have_phase = 0;
    if (P->profiling) cudaEventRecord(P->total.beg, st);
    auto Cm = [&](int l) { return f64 ? (C *)P->lev[l].Cm64 : (C *)P->lev[l].Cm32; };
    auto Dl = [&](int l) { return f64 ? (C *)P->lev[l].Dl64 : (C *)P->lev[l].Dl32; };
    const C *U = f64 ? (const C *)P->U64 : (const C *)P->U32;
    const C *Rv = f64 ? (const C *)P->Rv64 : (const C *)P->Rv32;
    const C *nearv = f64 ? (const C *)P->near64 : (const C *)P->near32;
    LevelDev &LL = P->lev[lmax];
    float2 *x32 = f64 ? nullptr : P->x32;
    if (!f64 && (!x32 || P->x32_cap < nrhs)) {
        fmm_set_error("mixed matvec: FP32 input buffer missing");
        return FMM_ERR_CUDA;
    }

    timer_begin(P, "p2m");
    // the transposed operator swaps the roles of the element moments and the centroid basis
    // (index-flipped), keeps every translation, and uses the transposed near-field matrix
    const ZeroList zero = owner ? ZeroList{} : zero_list(P, nrhs);
    const unsigned blocks = LL.nb + (zero.count ? zero.end[zero.count - 1] : 0);
    if (nrhs == 1)
        p2m_kernel<T, 1><<<dim3(blocks, 1), 128, 0, st>>>(LL.p, P->leaf_beg, P->leaf_elem, transpose ? Rv : U, x, P->opt.k,
                                                      Cm(lmax), transpose, P->nf, LL.nb, 1, x32, zero);
    else
        p2m_kernel<T, 8><<<dim3(blocks, (nrhs + 7) / 8), 128, 0, st>>>(LL.p, P->leaf_beg, P->leaf_elem, transpose ? Rv : U, x,
                                                                   P->opt.k, Cm(lmax), transpose, P->nf, LL.nb, nrhs, x32,
                                                                   zero);
    timer_end(P);
    {
        int e = owner ? translate_owner(P, ffm2l ? OWN_FF : f64 ? OWN_FP64 : OWN_FP32, pass_begin, pass_end) : translate32(P, nrhs);
        if (e) return e;
    }
    timer_begin(P, "l2p_near");
    double2 a = make_double2(P->opt.a_re, P->opt.a_im);
    const C *nearT = f64 ? (const C *)P->nearT64 : (const C *)P->nearT32;
    {
        const int *nb_ = transpose ? P->nearT_beg : P->near_beg, *nc_ = transpose ? P->nearT_col : P->near_col;
        const C *nv_ = transpose ? nearT : nearv, *rv_ = transpose ? U : Rv;
        const unsigned gx = (unsigned)((P->nf + L2P_WARPS - 1) / L2P_WARPS);
        if (nrhs == 1)
            l2p_near_kernel<T, 1><<<dim3(gx, 1), 256, 0, st>>>(P->nf, LL.p, P->elem_leaf, Dl(lmax), rv_, nb_, nc_, nv_, x, x32,
                                                            a, y, transpose, LL.nb, 1);
        else
            l2p_near_kernel<T, 8><<<dim3(gx, (nrhs + 7) / 8), 256, 0, st>>>(P->nf, LL.p, P->elem_leaf, Dl(lmax), rv_, nb_,
                                                                         nc_, nv_, x, x32, a, y, transpose, LL.nb, nrhs);
    }
    timer_end(P);
    if (P->profiling) {
        cudaEventRecord(P->total.end, st);
        P->have_total = 1;
    }
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

// Dense operators for the tensor-core passes: T[c][i][j] (pout^2 x pin^2, FP64), the RCR
// translation of key keys[c] (M2L direction, M2M / L2L octant) applied to the unit source e_j, with
// its azimuthal phases left out (rotation by the polar angle, coaxial translation, rotation back);
// the translation of any key d with the same polar angle and distance is then
// diag(e^{-i m' phi_d}) T diag(e^{i m phi_d}).  One CTA per (operator, column).
__global__ void dense_rcr_kernel(int p, int pmax, int pin, int pout, const int *__restrict__ keys,
                                 const double *__restrict__ H, const double2 *__restrict__ Cc, int coax_per_dir,
                                 double2 *__restrict__ T)
{
    extern __shared__ unsigned char smraw[];
    const int P2 = p * p, c = blockIdx.x, d = keys[c], j = blockIdx.y, rs = rot_size(pmax), w = 2 * pmax - 1;
    const int pi2 = pin * pin, po2 = pout * pout;
    double2 *sE = (double2 *)smraw, *sX = sE + P2, *sW1 = sX + P2, *sW2 = sW1 + P2, *sY = sW2 + P2, *sOne = sY + max(P2, po2);
    for (int i = threadIdx.x; i < P2; i += blockDim.x) sE[i] = make_double2(i == j ? 1.0 : 0.0, 0.0);
    for (int i = threadIdx.x; i < po2; i += blockDim.x) sY[i] = make_double2(0.0, 0.0);
    for (int i = threadIdx.x; i < w; i += blockDim.x) sOne[i] = make_double2(1.0, 0.0);
    __syncthreads();
    const double2 *cb = Cc + (coax_per_dir ? (size_t)c_dir_dist[d] * coax_size(p) : 0);
    rcr_block(p, pmax, H + (size_t)d * rs, sOne, cb, sE, pin, sX, sW1, sW2, sY, pout);
    for (int i = threadIdx.x; i < po2; i += blockDim.x) T[((size_t)c * po2 + i) * pi2 + j] = sY[i];
}

int gen_dense_rcr(Plan *P, int l, int which, const int *keys, int nkeys, double2 *T)
{
    const LevelDev &L = P->lev[l];
    int p, pin, pout;
    const double *H;
    const double2 *Cc;
    if (which == PASS_M2L) {
        p = pin = pout = L.p;
        H = P->Hsr64;
        Cc = L.Csr64;
    } else {
        const int pp = P->lev[l - 1].p;  // the RCR order of M2M / L2L is the parent's
        p = pp;
        pin = which == PASS_M2M ? L.p : pp;
        pout = which == PASS_M2M ? pp : L.p;
        H = which == PASS_M2M ? P->Hss64 : P->Hrr64;
        Cc = L.Crr64;
    }
    size_t sm = ((size_t)4 * p * p + std::max(p, pout) * std::max(p, pout) + 2 * P->pmax) * sizeof(double2);
    if (sm > 48 * 1024) FMM_CUDA_TRY(cudaFuncSetAttribute(dense_rcr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    dense_rcr_kernel<<<dim3(nkeys, pin * pin), 128, sm, P->stream>>>(p, P->pmax, pin, pout, keys, H, Cc, which == PASS_M2L ? 1 : 0,
                                                                   T);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

int set_dir_dist(const int *dd)
{
    FMM_CUDA_TRY(cudaMemcpyToSymbol(c_dir_dist, dd, sizeof(int) * NDIR));
    return FMM_OK;
}

// The FP32 expansions hold rhs_cap32 right-hand sides, level by level ([box][rhs][p^2]).
static int ensure_rhs32(Plan *P, int nrhs)
{
    if (nrhs > P->x32_cap) {
        cudaFree(P->x32);
        P->x32 = nullptr;
        P->device_bytes -= sizeof(float2) * (size_t)P->nf * P->x32_cap;
        P->x32_cap = 0;
        FMM_CUDA_TRY(dev_alloc(P, (void **)&P->x32, sizeof(float2) * (size_t)P->nf * nrhs));
        P->x32_cap = nrhs;
    }
    if (nrhs <= P->rhs_cap32) return FMM_OK;
    drop_graph(P); // the captured passes address the old expansions
    for (int l = P->lmin; l <= P->lmax; l++) {
        LevelDev &L = P->lev[l];
        size_t n = (size_t)L.nb * L.p * L.p;
        cudaFree(L.Cm32);
        cudaFree(L.Dl32);
        L.Cm32 = nullptr;
        L.Dl32 = nullptr;
        P->device_bytes -= 2 * sizeof(float2) * (n * P->rhs_cap32 + 1);
        FMM_CUDA_TRY(dev_alloc(P, (void **)&L.Cm32, sizeof(float2) * (n * nrhs + 1)));
        FMM_CUDA_TRY(dev_alloc(P, (void **)&L.Dl32, sizeof(float2) * (n * nrhs + 1)));
    }
    P->rhs_cap32 = nrhs;
    P->buf_gen++;
    return FMM_OK;
}

int run_matvec(Plan *P, const double2 *x, double2 *y, int precision, int transpose, int nrhs)
{
    if (transpose && !P->nearT_beg) {
        fmm_set_error("transposed near field not built");
        return FMM_ERR_ARG;
    }
    if (precision == FMM_MIXED) {
        if (!P->U32) {
            fmm_set_error("%s", P->mixed_note);
            return FMM_ERR_ARG;
        }
        int st = ensure_rhs32(P, nrhs);
        if (st) return st;
        if (!P->opt.deterministic) return run_matvec_t<float>(P, x, y, transpose, nrhs);
        // the translations without atomics take one right-hand side
        for (int r = 0; r < nrhs; r++) {
            st = run_matvec_t<float>(P, x + (size_t)r * P->nf, y + (size_t)r * P->nf, transpose, 1);
            if (st) return st;
        }
        return FMM_OK;
    }
    bool ffm2l = false;
    if (precision == FMM_FLOAT2) {
        int st = ensure_ff(P);
        if (st) return st;
        ffm2l = P->ff_ready > 0;
    }
    for (int r = 0; r < nrhs; r++) {
        int st = run_matvec_t<double>(P, x + (size_t)r * P->nf, y + (size_t)r * P->nf, transpose, 1, ffm2l);
        if (st) return st;
    }
    return FMM_OK;
}

__global__ void gather_kernel(const double2 *src, const long long *perm, long long n, double2 *dst)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = src[perm[i]];
}

__global__ void conj_kernel(const double2 *x, double2 *y, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        y[i] = make_double2(x[i].x, -x[i].y);
}

void launch_conj(Plan *P, const double2 *x, double2 *y, size_t n)
{
    conj_kernel<<<(unsigned)std::min<size_t>((n + 255) / 256, 152 * 8), 256, 0, P->stream>>>(x, y, n);
}

// Near-field matrix transposed (CSR by source element), built on first use of the
// transposed operator: (A^T y)_j collects A_ij y_i over the targets i near j.
// The transpose of the near-field pattern: row beginnings tb and columns tc by source
// element, and for each transposed entry the position of the same pair in the forward CSR.
static int near_transpose_pattern(Plan *P, std::vector<int> &tb, std::vector<int> &tc, std::vector<long long> &perm)
{
    long long nnz = P->num_near;
    std::vector<int> beg(P->nf + 1), col(nnz);
    FMM_CUDA_TRY(cudaMemcpy(beg.data(), P->near_beg, sizeof(int) * (P->nf + 1), cudaMemcpyDeviceToHost));
    FMM_CUDA_TRY(cudaMemcpy(col.data(), P->near_col, sizeof(int) * nnz, cudaMemcpyDeviceToHost));
    std::vector<int> fill(P->nf, 0);
    tb.assign(P->nf + 1, 0);
    tc.resize(nnz);
    perm.resize(nnz);
    for (long long s = 0; s < nnz; s++) tb[col[s] + 1]++;
    for (int j = 0; j < P->nf; j++) tb[j + 1] += tb[j];
    for (int i = 0; i < P->nf; i++)
        for (int s = beg[i]; s < beg[i + 1]; s++) {
            int j = col[s];
            long long pos = tb[j] + fill[j]++;
            tc[pos] = i;
            perm[pos] = s;
        }
    return FMM_OK;
}

// valsT = the near-field values `vals` (forward CSR order) in the transposed CSR order
int near_transpose_values(Plan *P, const double2 *vals, double2 *valsT)
{
    std::vector<int> tb, tc;
    std::vector<long long> perm;
    int st = near_transpose_pattern(P, tb, tc, perm);
    if (st) return st;
    long long nnz = P->num_near;
    long long *perm_dev = nullptr;
    FMM_CUDA_TRY(cudaMalloc(&perm_dev, sizeof(long long) * std::max<long long>(1, nnz)));
    FMM_CUDA_TRY(upload(perm_dev, perm.data(), sizeof(long long) * nnz));
    gather_kernel<<<152 * 8, 256, 0, P->stream>>>(vals, perm_dev, nnz, valsT);
    FMM_CUDA_TRY(cudaGetLastError());
    FMM_CUDA_TRY(cudaStreamSynchronize(P->stream));
    cudaFree(perm_dev);
    return FMM_OK;
}

int build_transpose(Plan *P)
{
    if (P->nearT_beg) return FMM_OK;
    long long nnz = P->num_near;
    std::vector<int> tb, tc;
    std::vector<long long> perm;
    int st = near_transpose_pattern(P, tb, tc, perm);
    if (st) return st;
    long long *perm_dev = nullptr;
    FMM_CUDA_TRY(cudaMalloc(&perm_dev, sizeof(long long) * std::max<long long>(1, nnz)));
    FMM_CUDA_TRY(upload(perm_dev, perm.data(), sizeof(long long) * nnz));
    FMM_CUDA_TRY(dev_alloc(P, (void **)&P->nearT_beg, sizeof(int) * (P->nf + 1)));
    FMM_CUDA_TRY(dev_alloc(P, (void **)&P->nearT_col, sizeof(int) * std::max<long long>(1, nnz)));
    FMM_CUDA_TRY(dev_alloc(P, (void **)&P->nearT64, sizeof(double2) * std::max<long long>(1, nnz)));
    FMM_CUDA_TRY(upload(P->nearT_beg, tb.data(), sizeof(int) * (P->nf + 1)));
    FMM_CUDA_TRY(upload(P->nearT_col, tc.data(), sizeof(int) * nnz));
    gather_kernel<<<152 * 8, 256, 0, P->stream>>>(P->near64, perm_dev, nnz, P->nearT64);
    FMM_CUDA_TRY(cudaGetLastError());
    if (P->U32) {
        FMM_CUDA_TRY(dev_alloc(P, (void **)&P->nearT32, sizeof(float2) * std::max<long long>(1, nnz)));
        int blocks = 152 * 8;
        to_float_kernel2<<<blocks, 256, 0, P->stream>>>((const double *)P->nearT64, (float *)P->nearT32, 2 * (size_t)nnz);
        FMM_CUDA_TRY(cudaGetLastError());
    }
    FMM_CUDA_TRY(cudaStreamSynchronize(P->stream));
    cudaFree(perm_dev);
    return FMM_OK;
}


} // namespace fmm
