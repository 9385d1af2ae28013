// fmm_vjp: reverse-mode derivative of a far-field objective with respect to the vertex
// positions (the adjoint path; the reference has none).
//
// With A(V) x = b(V) (b the plane wave at the centroids) and p = F(V) x the scattered field at
// fixed exterior points, a cotangent pbar of p (dJ = 2 Re pbar^H dp) gives
//     dJ/dV = 2 Re[ pbar^H (dF/dV) x ] + 2 Re[ mu^T (db/dV - (dA/dV) x) ],
// where mu = conj(lambda) solves A^T mu = F^T conj(pbar) (the adjoint system A^H lambda =
// F^H pbar, conjugated).  dA/dV is the derivative of the operator this library applies: the
// octree, truncation orders and box centres are held fixed and A is split as the matvec
// splits it:
//   near pairs (i, j)     direct quadrature, differentiated pair by pair;
//   far pairs, target i   sum_j A_ij x_j = sum_nm D_i[nm] R_n^m(c_i - C_i) with D the leaf
//                         local of the forward pass on x: differentiate in c_i;
//   far pairs, source j   sum_i mu_i A_ij = sum_nm Psi_j[nm] U_j[n,-m] with Psi the leaf local
//                         of the transposed pass on mu (U_j[n,-m] integrates R_n^m over T_j):
//                         differentiate the integral over T_j in its vertices.
// Every local derivative is exact to rounding, and taken in reverse: the objective's weight is known
// before a quadrature point is evaluated, so a point adds real vectors to the gradients by the
// source's vertices, normal and area and the target's centroid and normal (a few operations more
// than its value), and the vertices follow by the chain rule once per pair.  The basis is
// evaluated through u = (x + i y)/r and polynomials in z/r (Q_n^m = st^m q_n^m), which stays
// smooth on the z-axis where (theta, phi) do not.
//
// What bounds it: the FP64 pipe (per point a sincos, a reciprocal square root and some 40
// multiply-adds; the near pairs of a Burton-Miller plan have 24 edge points per segment beside 7
// or 9 on the face).  On the 5,120-triangle head (498,000 near pairs, admittance, Burton-Miller)
// against forward-mode dual numbers with 9 to 18 slots: near pairs 111 -> 5.5 ms, source side
// of the far pairs 22 -> 0.9, far points 7.8 -> 0.3, target side 2.1 -> 0.3, the whole fmm_vjp
// with its adjoint solve 163 -> 27 ms.
#include "plan.h"
#include <algorithm>
#include <vector>

namespace fmm {

// copies of the regular rules of tables.cu (rule_tables), uploaded on first use
__constant__ double v_rule_bary[2][16 * 3];
__constant__ double v_rule_w[2][16];
__constant__ int v_rule_n[2];
// the 8-point Gauss rule on [-1, 1] of the Burton-Miller edge integrals (tables.cu)
constexpr int V_LINE_PTS = 8;
__constant__ double v_line_x[V_LINE_PTS], v_line_w[V_LINE_PTS];

static int upload_legendre();

static int upload_vjp_rules()
{
    static int dev_done = -1;
    int dev = 0;
    FMM_CUDA_TRY(cudaGetDevice(&dev));
    if (dev_done == dev) return FMM_OK;
    double bary[2][48], w[2][16];
    int n[2];
    rule_tables(bary, w, n);
    FMM_CUDA_TRY(cudaMemcpyToSymbol(v_rule_bary, bary, sizeof(bary)));
    FMM_CUDA_TRY(cudaMemcpyToSymbol(v_rule_w, w, sizeof(w)));
    FMM_CUDA_TRY(cudaMemcpyToSymbol(v_rule_n, n, sizeof(n)));
    double lx[V_LINE_PTS], lw[V_LINE_PTS];
    line_rule(V_LINE_PTS, lx, lw);
    FMM_CUDA_TRY(cudaMemcpyToSymbol(v_line_x, lx, sizeof(lx)));
    FMM_CUDA_TRY(cudaMemcpyToSymbol(v_line_w, lw, sizeof(lw)));
    int st = upload_legendre();
    if (st) return st;
    dev_done = dev;
    return FMM_OK;
}

// Number of equal segments of an edge of length len seen from distance dist, as in tables.cu; the
// numbers follow from the values and are held fixed by the derivative.
__device__ __forceinline__ int edge_segments_v(double len, double dist)
{
    double m = ceil(len / fmax(dist, 1e-12 * len));
    return m > 64.0 ? 64 : (int)m;
}

constexpr int VJP_PMAX = 24; // largest leaf order (plus one for gradient expansions) handled here

// factors of the recurrence in degree of q_n^m (Q_n^m = st^m q_n^m): q_n = a (ct q_{n-1} - b q_{n-2});
// q_m^m and the factor of q_{m+1}^m = sqrt(2m+3) ct q_m^m
__constant__ double v_leg_a[VJP_PMAX * VJP_PMAX], v_leg_b[VJP_PMAX * VJP_PMAX];
__constant__ double v_leg_mm[VJP_PMAX], v_leg_s[VJP_PMAX];

static int upload_legendre()
{
    double la[VJP_PMAX * VJP_PMAX] = {}, lb[VJP_PMAX * VJP_PMAX] = {}, mm[VJP_PMAX], ls[VJP_PMAX];
    double cmm = 0.28209479177387814; // q_0^0 = 1/sqrt(4 pi)
    for (int m = 0; m < VJP_PMAX; m++) {
        if (m > 0) cmm *= sqrt((2.0 * m + 1.0) / (2.0 * m));
        mm[m] = cmm;
        ls[m] = sqrt(2.0 * m + 3.0);
        for (int n = m + 2; n < VJP_PMAX; n++) {
            la[n * VJP_PMAX + m] = sqrt((4.0 * n * n - 1.0) / ((double)n * n - (double)m * m));
            lb[n * VJP_PMAX + m] = sqrt(((n - 1.0) * (n - 1.0) - (double)m * m) / (4.0 * (n - 1.0) * (n - 1.0) - 1.0));
        }
    }
    FMM_CUDA_TRY(cudaMemcpyToSymbol(v_leg_a, la, sizeof(la)));
    FMM_CUDA_TRY(cudaMemcpyToSymbol(v_leg_b, lb, sizeof(lb)));
    FMM_CUDA_TRY(cudaMemcpyToSymbol(v_leg_mm, mm, sizeof(mm)));
    FMM_CUDA_TRY(cudaMemcpyToSymbol(v_leg_s, ls, sizeof(ls)));
    return FMM_OK;
}

// f_e(v) = sum_{n < P, |m| <= n} coef[e][n^2+n+m] R_n^m(v), R_n^m = j_n(kr) q_n^|m|(z/r) u^m
// (u^{-m} read as conj(u)^m), and (GRAD) its gradient, for NE expansions at one point.  The sums over
// n are taken at fixed m for the value and its derivatives by r and by z/r; the derivative by u
// follows from the powers of u.
template <int NE, bool GRAD>
__device__ void eval_expansions(int P, double k, const double *v, const double2 *const *coef, double2 *val,
                                double2 (*grd)[3])
{
    const double r = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]), ri = 1.0 / r, ct = v[2] * ri;
    const double2 u = make_double2(v[0] * ri, v[1] * ri);
    double jn[VJP_PMAX + 1];
    sph_jn_array(P + 1, k * r, jn);
    double2 F[NE], Fr[NE], Fc[NE], Gp[NE], Gm[NE];
#pragma unroll
    for (int e = 0; e < NE; e++) F[e] = Fr[e] = Fc[e] = Gp[e] = Gm[e] = make_double2(0.0, 0.0);
    double2 um = make_double2(1.0, 0.0), um1 = make_double2(0.0, 0.0);
    auto add = [](double2 &a, double f, double2 c) {
        a.x = fma(f, c.x, a.x);
        a.y = fma(f, c.y, a.y);
    };
    for (int m = 0; m < P; m++) {
        if (m > 0) {
            um1 = um;
            um = cmul(um, u);
        }
        double2 Ap[NE], Am[NE], Arp[NE], Arm[NE], Acp[NE], Acm[NE];
#pragma unroll
        for (int e = 0; e < NE; e++) Ap[e] = Am[e] = Arp[e] = Arm[e] = Acp[e] = Acm[e] = make_double2(0.0, 0.0);
        double q2 = 0.0, q1 = 0.0, d2 = 0.0, d1 = 0.0;
        for (int n = m; n < P; n++) {
            double q, d;
            if (n == m) {
                q = v_leg_mm[m];
                d = 0.0;
            } else if (n == m + 1) {
                d = v_leg_s[m] * q1;
                q = d * ct;
            } else {
                const double a = v_leg_a[n * VJP_PMAX + m], b = v_leg_b[n * VJP_PMAX + m];
                q = a * (ct * q1 - b * q2);
                d = a * (q1 + ct * d1 - b * d2);
            }
            q2 = q1;
            q1 = q;
            d2 = d1;
            d1 = d;
            const double t0 = jn[n] * q;
            const double tr = GRAD ? (n * ri * jn[n] - k * jn[n + 1]) * q : 0.0, tc = GRAD ? jn[n] * d : 0.0;
#pragma unroll
            for (int e = 0; e < NE; e++) {
                const double2 cp = coef[e][n * n + n + m];
                add(Ap[e], t0, cp);
                if (GRAD) {
                    add(Arp[e], tr, cp);
                    add(Acp[e], tc, cp);
                }
                if (m > 0) {
                    const double2 cm = coef[e][n * n + n - m];
                    add(Am[e], t0, cm);
                    if (GRAD) {
                        add(Arm[e], tr, cm);
                        add(Acm[e], tc, cm);
                    }
                }
            }
        }
        // a u^m + b conj(u)^m
        auto both = [&](double2 &s, double2 a, double2 b) {
            s.x += (a.x + b.x) * um.x - (a.y - b.y) * um.y;
            s.y += (a.x - b.x) * um.y + (a.y + b.y) * um.x;
        };
#pragma unroll
        for (int e = 0; e < NE; e++) {
            both(F[e], Ap[e], Am[e]);
            if (GRAD) {
                both(Fr[e], Arp[e], Arm[e]);
                both(Fc[e], Acp[e], Acm[e]);
                add(Gp[e], m, cmul(Ap[e], um1));
                add(Gm[e], m, cconjmul(um1, Am[e]));
            }
        }
    }
#pragma unroll
    for (int e = 0; e < NE; e++) {
        val[e] = F[e];
        if (GRAD) {
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const double ra = v[a] * ri, ca = ((a == 2 ? 1.0 : 0.0) - ct * ra) * ri;
                // d u / d v_a and its conjugate
                const double2 ua = make_double2(((a == 0 ? 1.0 : 0.0) - u.x * ra) * ri, ((a == 1 ? 1.0 : 0.0) - u.y * ra) * ri);
                double2 g = cadd(cscale(Fr[e], ra), cscale(Fc[e], ca));
                g = cadd(g, cmul(Gp[e], ua));
                grd[e][a] = cadd(g, cconjmul(ua, Gm[e]));
            }
        }
    }
}

// grad phi and its derivatives H[b][a] = d_a d_b phi from the values and gradients of the
// derivative expansions d/dz, d+ and d- (d/dx +- i d/dy)
__device__ __forceinline__ void cartesian(const double2 *val, const double2 (*grd)[3], double2 *g, double2 (*H)[3])
{
    auto xy = [](double2 p, double2 m, double2 &x, double2 &y) {
        x = make_double2(0.5 * (p.x + m.x), 0.5 * (p.y + m.y));
        y = make_double2(0.5 * (p.y - m.y), -0.5 * (p.x - m.x));
    };
    xy(val[1], val[2], g[0], g[1]);
    g[2] = val[0];
    for (int a = 0; a < 3; a++) {
        xy(grd[1][a], grd[2][a], H[0][a], H[1][a]);
        H[2][a] = grd[0][a];
    }
}

// ----------------------------------------------------------------------------- pairs, in reverse
__device__ __forceinline__ double re_mul(double2 a, double2 b) { return a.x * b.x - a.y * b.y; }

// G = exp(ikr)/(4 pi r), h = G'/r (grad G = h d) and e = h'/r (grad h = e d) at distance r: the
// phase (c, s), the factors of r and kr, from which only real parts of products with complex
// weights are taken: w exp(ikr) first, then the polynomials in ikr.
struct Radial {
    double c, s, kr, f, fh, fe;
};
__device__ __forceinline__ Radial radial(double k, double r2)
{
    Radial o;
    const double ri = rsqrt(r2), ri2 = ri * ri;
    o.kr = k * (r2 * ri);
    sincos(o.kr, &o.s, &o.c);
    o.f = ri * (1.0 / (4.0 * FMM_PI));
    o.fh = o.f * ri2;
    o.fe = o.fh * ri2;
    return o;
}
// w exp(ikr), and Re(w G), Re(w h), Re(w e) from it
__device__ __forceinline__ double2 turned(const Radial &o, double2 w)
{
    return make_double2(w.x * o.c - w.y * o.s, w.x * o.s + w.y * o.c);
}
__device__ __forceinline__ double re_g(const Radial &o, double2 z) { return o.f * z.x; }
__device__ __forceinline__ double re_h(const Radial &o, double2 z) { return -o.fh * (z.x + o.kr * z.y); }
__device__ __forceinline__ double re_e(const Radial &o, double2 z)
{
    return o.fe * ((3.0 - o.kr * o.kr) * z.x + 3.0 * o.kr * z.y);
}

// the unnormalised normal N = u x v of a triangle (u = v0 - v2, v = v1 - v2) and its length
struct Tri {
    double u[3], v[3], N[3], J;
};
__device__ __forceinline__ Tri tri_of(const double *nd)
{
    Tri t;
    for (int a = 0; a < 3; a++) {
        t.u[a] = nd[a] - nd[6 + a];
        t.v[a] = nd[3 + a] - nd[6 + a];
    }
    t.N[0] = t.u[1] * t.v[2] - t.u[2] * t.v[1];
    t.N[1] = t.u[2] * t.v[0] - t.u[0] * t.v[2];
    t.N[2] = t.u[0] * t.v[1] - t.u[1] * t.v[0];
    t.J = sqrt(t.N[0] * t.N[0] + t.N[1] * t.N[1] + t.N[2] * t.N[2]);
    return t;
}
__device__ __forceinline__ double dot3(const double *a, const double *b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
// s += f (a x b)
__device__ __forceinline__ void cross_add(double *s, double f, const double *a, const double *b)
{
    s[0] += f * (a[1] * b[2] - a[2] * b[1]);
    s[1] += f * (a[2] * b[0] - a[0] * b[2]);
    s[2] += f * (a[0] * b[1] - a[1] * b[0]);
}
// gradients by N and J to the vertices
__device__ __forceinline__ void normal_to_nodes(const Tri &t, double *gN, double gJ, double *gs)
{
    for (int a = 0; a < 3; a++) gN[a] += gJ / t.J * t.N[a];
    double gu[3] = {0, 0, 0}, gv[3] = {0, 0, 0};
    cross_add(gu, 1.0, t.v, gN);
    cross_add(gv, 1.0, gN, t.u);
    for (int a = 0; a < 3; a++) {
        gs[a] += gu[a];
        gs[3 + a] += gv[a];
        gs[6 + a] -= gu[a] + gv[a];
    }
}

// The gradient of Re[ w0 (b I0 + c I1) + w1 (b I2 + c (k^2 (ny.nh) I0 - L)) ] over the element nd:
// I0, I1, I2 the integrals of G, dG/dn_x and dG/dn_y by the regular rule, L the edge integral
// of the regularised hypersingular kernel (tables.cu: elem_integrals_fused, hyper_edges; the numbers
// of edge segments follow from the values, as there, and are held fixed).  w0b = w0 b etc.; BM:
// with the w1 terms.  gs: by the vertices; gy, gny: by the target's point and unit normal (added).
template <bool BM>
__device__ __forceinline__ void pair_grad(double k, const double *nd, const double *y, const double *ny, int rule,
                                          double2 w0b, double2 w0c, double2 w1b, double2 w1c, double *gs, double *gy,
                                          double *gny)
{
    const Tri t = tri_of(nd);
    const double dn = BM ? dot3(ny, t.N) / t.J : 0.0;
    const double2 A0 = BM ? make_double2(w0b.x + k * k * dn * w1c.x, w0b.y + k * k * dn * w1c.y) : w0b;
    double gN[3] = {0, 0, 0}, gJ = 0.0, gdn = 0.0;
    for (int i = 0; i < 9; i++) gs[i] = 0.0;
    const int nq = v_rule_n[rule];
    for (int q = 0; q < nq; q++) {
        const double *bb = &v_rule_bary[rule][3 * q], wq = v_rule_w[rule][q];
        double d[3];
        for (int a = 0; a < 3; a++) d[a] = bb[0] * nd[a] + bb[1] * nd[3 + a] + bb[2] * nd[6 + a] - y[a];
        const Radial f = radial(k, dot3(d, d));
        const double2 z0 = turned(f, A0), z1 = turned(f, w0c);
        const double dN = dot3(d, t.N), a1h = re_h(f, z1);
        // by d: along d, along N and (BM) along ny
        double along = t.J * re_h(f, z0) + re_e(f, z1) * dN, a2h = 0.0, dny = 0.0;
        if (BM) {
            const double2 z2 = turned(f, w1b);
            dny = dot3(d, ny);
            a2h = -re_h(f, z2);
            along -= t.J * re_e(f, z2) * dny;
            gdn += wq * re_g(f, turned(f, w1c));
        }
        gJ += wq * (re_g(f, z0) + a2h * dny);
        for (int a = 0; a < 3; a++) {
            double D = along * d[a] + a1h * t.N[a];
            if (BM) {
                D += t.J * a2h * ny[a];
                gny[a] += wq * t.J * a2h * d[a];
            }
            D *= wq;
            gN[a] += wq * a1h * d[a];
            gs[a] += bb[0] * D;
            gs[3 + a] += bb[1] * D;
            gs[6 + a] += bb[2] * D;
        }
    }
    for (int a = 0; a < 3; a++) gy[a] -= gs[a] + gs[3 + a] + gs[6 + a];
    if (BM) {
        if (w1c.x != 0.0 || w1c.y != 0.0) {
            // -w1 c L: along an edge d = a - s t, and d . (t x ny) = a . (t x ny)
            for (int e = 0; e < 3; e++) {
                const double *va = nd + 3 * e, *vb = nd + 3 * ((e + 1) % 3);
                double tt[3], av[3], tn[3] = {0, 0, 0};
                for (int a = 0; a < 3; a++) {
                    tt[a] = vb[a] - va[a];
                    av[a] = y[a] - va[a];
                }
                cross_add(tn, 1.0, tt, ny);
                const double t2 = dot3(tt, tt), at = dot3(av, tt), len = sqrt(t2);
                const double sc = fmin(fmax(at / t2, 0.0), 1.0);
                const double e0 = av[0] - sc * tt[0], e1 = av[1] - sc * tt[1], e2 = av[2] - sc * tt[2];
                const int nseg = edge_segments_v(len, sqrt(e0 * e0 + e1 * e1 + e2 * e2));
                double hs = 0.0, es = 0.0, ess = 0.0, esss = 0.0;  // sums of -Re(w1c h), -Re(w1c e) s^0, s^1, s^2
                const double inv = 1.0 / nseg;
                for (int g = 0; g < nseg; g++)
                    for (int q = 0; q < V_LINE_PTS; q++) {
                        const double s = (g + 0.5 + 0.5 * v_line_x[q]) * inv, w = -0.5 * v_line_w[q] * inv;
                        const double d0 = av[0] - s * tt[0], d1 = av[1] - s * tt[1], d2 = av[2] - s * tt[2];
                        const Radial f = radial(k, d0 * d0 + d1 * d1 + d2 * d2);
                        const double2 z = turned(f, w1c);
                        const double he = w * re_e(f, z), hes = s * he;
                        hs += w * re_h(f, z);
                        es += he;
                        ess += hes;
                        esss += s * hes;
                    }
                const double an = dot3(av, tn);
                double ga[3], gt[3] = {0, 0, 0};
                for (int a = 0; a < 3; a++) ga[a] = hs * tn[a] + an * (es * av[a] - ess * tt[a]);
                cross_add(gt, hs, ny, av);
                cross_add(gny, hs, av, tt);
                for (int a = 0; a < 3; a++) {
                    gt[a] -= an * (ess * av[a] - esss * tt[a]);
                    gy[a] += ga[a];
                    gs[3 * e + a] -= ga[a] + gt[a];
                    gs[3 * ((e + 1) % 3) + a] += gt[a];
                }
            }
        }
        gdn *= k * k * t.J;
        for (int a = 0; a < 3; a++) {
            gny[a] += gdn / t.J * t.N[a];
            gN[a] += gdn / t.J * ny[a];
        }
        gJ -= gdn * dn / t.J;
    }
    normal_to_nodes(t, gN, gJ, gs);
}

__device__ __forceinline__ void load_tri_d(const double *V, const int *F, int e, double *nod)
{
    for (int t = 0; t < 3; t++)
        for (int a = 0; a < 3; a++) nod[3 * t + a] = V[3 * F[3 * e + t] + a];
}

__device__ __forceinline__ void add_vertex_grad(double *grad, const int *F, int e, const double *g9)
{
    for (int t = 0; t < 3; t++)
        for (int a = 0; a < 3; a++) atomicAdd(&grad[3 * F[3 * e + t] + a], g9[3 * t + a]);
}

// ----------------------------------------------------------------------------- VJP kernels
// The far-field operator F_kj = -int_{T_j} (b G + c dG/dn_x)(x, p_k) dS (fmm_far_field); a group of
// `grp` lanes (a power of two, at most a warp) takes an element and shares its points.
__device__ __forceinline__ double group_sum(double v, int grp)
{
    for (int o = grp / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// 2 Re[ sum_k conj(pbar_k) x_j dF_kj/dV_j ] for the vertices of element j; nb = -b, nc = -c
__global__ void vjp_farpts_kernel(const double *V, const int *F, int nf, double k, int rule, double2 nb, double2 nc,
                                  const double *pts, int npts, const double2 *pbar, const double2 *x, double *grad, int grp)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x, j = id / grp, l = id % grp;
    double g9[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (j < nf) {
        double nd[9];
        load_tri_d(V, F, j, nd);
        const double2 xj = x[j], z = make_double2(0.0, 0.0);
        for (int t = l; t < npts; t += grp) {
            const double2 pb = pbar[t];
            // w = 2 conj(pbar) x_j
            const double2 w = make_double2(2.0 * (pb.x * xj.x + pb.y * xj.y), 2.0 * (pb.x * xj.y - pb.y * xj.x));
            double gs[9], gy[3] = {0, 0, 0};
            pair_grad<false>(k, nd, pts + 3 * t, nullptr, rule, cmul(w, nb), cmul(w, nc), z, z, gs, gy, nullptr);
            for (int i = 0; i < 9; i++) g9[i] += gs[i];
        }
    }
    for (int i = 0; i < 9; i++) g9[i] = group_sum(g9[i], grp);
    if (j < nf && l == 0) add_vertex_grad(grad, F, j, g9);
}

// right-hand side of the conjugated adjoint system: rhs_j = sum_k F_kj conj(pbar_k)
__global__ void vjp_adjoint_rhs_kernel(const double *V, const int *F, int nf, double k, int rule, double2 nb, double2 nc,
                                       const double *pts, int npts, const double2 *pbar, double2 *rhs, int grp)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x, j = id / grp, l = id % grp;
    double2 acc = make_double2(0.0, 0.0);
    if (j < nf) {
        double nd[9];
        load_tri_d(V, F, j, nd);
        const Tri tr = tri_of(nd);
        const int nq = v_rule_n[rule];
        for (int t = l; t < npts; t += grp) {
            const double *y = pts + 3 * t;
            double2 I0 = make_double2(0.0, 0.0), I1 = I0;
            for (int q = 0; q < nq; q++) {
                const double *bb = &v_rule_bary[rule][3 * q], wq = v_rule_w[rule][q];
                double d[3];
                for (int a = 0; a < 3; a++) d[a] = bb[0] * nd[a] + bb[1] * nd[3 + a] + bb[2] * nd[6 + a] - y[a];
                const Radial f = radial(k, dot3(d, d));
                // G and h = -(1 - ikr) exp(ikr) / (4 pi r^3)
                I0 = cadd(I0, cscale(make_double2(f.c, f.s), wq * tr.J * f.f));
                I1 = cadd(I1, cscale(make_double2(f.c + f.kr * f.s, f.s - f.kr * f.c), -wq * dot3(d, tr.N) * f.fh));
            }
            const double2 f = cadd(cmul(nb, I0), cmul(nc, I1));
            acc = cadd(acc, cconjmul(pbar[t], f));
        }
    }
    acc.x = group_sum(acc.x, grp);
    acc.y = group_sum(acc.y, grp);
    if (j < nf && l == 0) rhs[j] = acc;
}

// 2 Re[ mu_i db_i/dV ] with b_i = exp(i k dir.c_i), c_i the centroid (1/3 per vertex)
__global__ void vjp_rhs_kernel(const double *V, const int *F, int nf, double k, double dx, double dy, double dz,
                               const double2 *mu, double *grad)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x) {
        double nd[9], c[3];
        load_tri_d(V, F, i, nd);
        for (int a = 0; a < 3; a++) c[a] = nd[a] + (2.0 / 3.0) * (0.5 * (nd[3 + a] + nd[6 + a]) - nd[a]);
        double s, co;
        sincos(k * (dx * c[0] + dy * c[1] + dz * c[2]), &s, &co);
        // d b / d c_a = i k dir_a b ;  Re(mu * i k dir_a b) = -k dir_a Im(mu b)
        double2 m = mu[i];
        double imb = m.x * s + m.y * co;
        double d3[3] = {dx, dy, dz}, g9[9];
        for (int t = 0; t < 3; t++)
            for (int a = 0; a < 3; a++) g9[3 * t + a] = 2.0 * (-k * d3[a] * imb) / 3.0;
        add_vertex_grad(grad, F, i, g9);
    }
}

// near pairs i != j: -2 Re[ mu_i x_j dA_ij ], A_ij = b I0 + c I1 and (BM) alpha (b K'_ij + c N_ij), one
// thread per entry of the near-field matrix.  The source's vertices take their share at once; by
// the target's centroid and unit normal the sums over its row go to tgt[i][6].
template <bool BM>
__global__ void __launch_bounds__(128)
vjp_near_kernel(const double *V, const int *F, int nf, long long nnz, const int *__restrict__ near_beg,
                const int *__restrict__ near_col, double k, double2 bco, double2 cco, double2 alpha, int rule,
                const double2 *mu, const double2 *x, double *grad, double *tgt)
{
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const bool on = s < nnz;
    int i = 0;
    double t6[6] = {0, 0, 0, 0, 0, 0};
    if (on) {
        // row of entry s: the last i with near_beg[i] <= s
        int hi = nf;
        while (hi - i > 1) {
            const int mid = (i + hi) >> 1;
            if (near_beg[mid] <= s) i = mid; else hi = mid;
        }
        const int j = near_col[s];
        if (i != j) {
            double ndi[9], nd[9], y[3], ny[3];
            load_tri_d(V, F, i, ndi);
            load_tri_d(V, F, j, nd);
            for (int a = 0; a < 3; a++) y[a] = ndi[a] + (2.0 / 3.0) * (0.5 * (ndi[3 + a] + ndi[6 + a]) - ndi[a]);
            if (BM) {
                const Tri ti = tri_of(ndi);
                for (int a = 0; a < 3; a++) ny[a] = ti.N[a] / ti.J;
            }
            const double2 w = cscale(cmul(mu[i], x[j]), -2.0), w1 = BM ? cmul(w, alpha) : w;
            double gs[9];
            pair_grad<BM>(k, nd, y, ny, rule, cmul(w, bco), cmul(w, cco), cmul(w1, bco), cmul(w1, cco), gs, t6, t6 + 3);
            add_vertex_grad(grad, F, j, gs);
        }
    }
    // rows are longer than a warp's 32 entries on most meshes: one addition per warp and row
    constexpr int NT = BM ? 6 : 3;
    const int i0 = __shfl_sync(0xffffffffu, i, 0);
    if (__all_sync(0xffffffffu, !on || i == i0)) {
        for (int a = 0; a < NT; a++) t6[a] = group_sum(t6[a], 32);
        if ((threadIdx.x & 31) == 0 && on)
            for (int a = 0; a < NT; a++) atomicAdd(&tgt[6 * (size_t)i + a], t6[a]);
    } else if (on) {
        for (int a = 0; a < NT; a++) atomicAdd(&tgt[6 * (size_t)i + a], t6[a]);
    }
}

// The target sides of the near pairs (tgt: gradients by centroid and unit normal) to the vertices,
// and the self terms: b G (three sub-triangles at the centroid by the collapsed rule; dG/dn
// vanishes on the element's own plane, wherever its vertices are) and (BM) alpha c N_ii
// (K'_ii = 0), the Hadamard finite part -(1/4 pi) [sum over edges of hL int exp(ikr)/r^3 - 2 pi i k],
// hL = |u x t| with u from the centroid to the edge and t along it.  One thread per element and
// sub-triangle / edge.
__global__ void vjp_near_self_kernel(const double *V, const int *F, int nf, double k, double2 bco, double2 cco,
                                     double2 alpha, const double2 *mu, const double2 *x, const double *tgt, double *grad)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x, i = id / 3, e = id % 3, e1 = (e + 1) % 3;
    if (i >= nf) return;
    const bool hb = bco.x != 0.0 || bco.y != 0.0;
    const bool hn = (cco.x != 0.0 || cco.y != 0.0) && (alpha.x != 0.0 || alpha.y != 0.0);
    double nd[9], g9[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, gc[3] = {0, 0, 0}, c[3];
    load_tri_d(V, F, i, nd);
    if (e == 0) {
        const double *g = tgt + 6 * (size_t)i;
        const Tri tr = tri_of(nd);
        // unit normal n = N / J: dJ/dN = n, so by N: (g - (g.n) n) / J
        double n[3], gN[3];
        for (int a = 0; a < 3; a++) n[a] = tr.N[a] / tr.J;
        const double gn = dot3(g + 3, n);
        for (int a = 0; a < 3; a++) {
            gN[a] = (g[3 + a] - gn * n[a]) / tr.J;
            gc[a] = g[a];
        }
        normal_to_nodes(tr, gN, 0.0, g9);
    }
    const double2 w = cscale(cmul(mu[i], x[i]), -2.0), z = make_double2(0.0, 0.0);
    double va[3], vb[3], ga[3] = {0, 0, 0}, gb[3] = {0, 0, 0};
    for (int a = 0; a < 3; a++) {
        c[a] = nd[a] + (2.0 / 3.0) * (0.5 * (nd[3 + a] + nd[6 + a]) - nd[a]);
        va[a] = nd[3 * e + a];
        vb[a] = nd[3 * e1 + a];
    }
    if (hb) {
        const double sub[9] = {va[0], va[1], va[2], vb[0], vb[1], vb[2], c[0], c[1], c[2]};
        double gs[9], gy[3] = {0, 0, 0};
        pair_grad<false>(k, sub, c, nullptr, 0, cmul(w, bco), z, z, z, gs, gy, nullptr);
        for (int a = 0; a < 3; a++) {
            ga[a] += gs[a];
            gb[a] += gs[3 + a];
            gc[a] += gs[6 + a] + gy[a];
        }
    }
    if (hn) {
        const double2 w1 = cscale(cmul(cmul(w, alpha), cco), -1.0 / (4.0 * FMM_PI));
        double u[3], t[3], uc[3] = {0, 0, 0}, gu[3] = {0, 0, 0}, gt[3] = {0, 0, 0};
        for (int a = 0; a < 3; a++) {
            u[a] = va[a] - c[a];
            t[a] = vb[a] - va[a];
        }
        cross_add(uc, 1.0, u, t);
        const double hL = sqrt(dot3(uc, uc)), len = sqrt(dot3(t, t));
        const int nseg = edge_segments_v(len, hL / len);
        // p = exp(ikr)/r^3, p'/r = exp(ikr) (ikr - 3)/r^5
        double ps = 0.0, es = 0.0, ess = 0.0, esss = 0.0;
        for (int g = 0; g < nseg; g++)
            for (int q = 0; q < V_LINE_PTS; q++) {
                const double s = (g + 0.5 + 0.5 * v_line_x[q]) / nseg, wl = 0.5 * v_line_w[q] / nseg;
                double d[3];
                for (int a = 0; a < 3; a++) d[a] = u[a] + s * t[a];
                const Radial f = radial(k, dot3(d, d));
                const double2 zw = turned(f, w1);
                const double f3 = wl * (4.0 * FMM_PI) * f.fh, f5 = wl * (4.0 * FMM_PI) * f.fe;
                const double pe = -f5 * (3.0 * zw.x + f.kr * zw.y);
                ps += f3 * zw.x;
                es += pe;
                ess += s * pe;
                esss += s * s * pe;
            }
        cross_add(gu, ps / hL, t, uc);
        cross_add(gt, ps / hL, uc, u);
        for (int a = 0; a < 3; a++) {
            gu[a] += hL * (es * u[a] + ess * t[a]);
            gt[a] += hL * (ess * u[a] + esss * t[a]);
            ga[a] += gu[a] - gt[a];
            gb[a] += gt[a];
            gc[a] -= gu[a];
        }
    }
    for (int t = 0; t < 3; t++)
        for (int a = 0; a < 3; a++)
            g9[3 * t + a] += gc[a] / 3.0 + (t == e ? ga[a] : 0.0) + (t == e1 ? gb[a] : 0.0);
    add_vertex_grad(grad, F, i, g9);
}

// far pairs, target side: -2 Re[ mu_i d/dc_i sum_nm D_i[nm] R_n^m(c_i - C) ], 1/3 per vertex
__global__ void vjp_far_target_kernel(const double *V, const int *F, int nf, int pl, double k, const int *elem_leaf,
                                      const double *box_ctr, const double2 *D, const double2 *mu, double *grad)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x) {
        double nd[9];
        load_tri_d(V, F, i, nd);
        int b = elem_leaf[i];
        double v[3];
        for (int a = 0; a < 3; a++) {
            double c = nd[a] + (2.0 / 3.0) * (0.5 * (nd[3 + a] + nd[6 + a]) - nd[a]);
            v[a] = c - box_ctr[3 * b + a];
        }
        const double2 *coef[1] = {D + (size_t)b * pl * pl};
        double2 f[1], g[1][3];
        eval_expansions<1, true>(pl, k, v, coef, f, g);
        double2 m = mu[i], w = make_double2(-m.x, -m.y);
        double g9[9];
        for (int a = 0; a < 3; a++) {
            double gc = 2.0 * re_mul(w, g[0][a]) / 3.0;
            for (int q = 0; q < 3; q++) g9[3 * q + a] = gc;
        }
        add_vertex_grad(grad, F, i, g9);
    }
}

// Burton-Miller far pairs, target side: -2 Re[ mu_i alpha d/dV (n_i . grad phi(c_i)) ] with
// phi = sum_nm D_i[nm] R_n^m(. - C), grad phi from its derivative expansions (Dz, Dp, Dm)
__global__ void vjp_far_target_bm_kernel(const double *V, const int *F, int nf, int pl, double k, double2 alpha,
                                         const int *elem_leaf, const double *box_ctr, const double2 *Dz,
                                         const double2 *Dp, const double2 *Dm, const double2 *mu, double *grad)
{
    const int po = pl + 1;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x) {
        double nd[9], v[3], n[3], gc[3], gn[3], gN[3], g9[9];
        load_tri_d(V, F, i, nd);
        int b = elem_leaf[i];
        const Tri tr = tri_of(nd);
        for (int a = 0; a < 3; a++) {
            v[a] = nd[a] + (2.0 / 3.0) * (0.5 * (nd[3 + a] + nd[6 + a]) - nd[a]) - box_ctr[3 * b + a];
            n[a] = tr.N[a] / tr.J;
        }
        const double2 *coef[3] = {Dz + (size_t)b * po * po, Dp + (size_t)b * po * po, Dm + (size_t)b * po * po};
        double2 e[3], de[3][3], g[3], H[3][3];
        eval_expansions<3, true>(po, k, v, coef, e, de);
        cartesian(e, de, g, H);
        // f = n . grad phi(c)
        const double2 w = cscale(cmul(mu[i], alpha), -2.0);
        for (int a = 0; a < 3; a++) {
            gc[a] = re_mul(w, H[0][a]) * n[0] + re_mul(w, H[1][a]) * n[1] + re_mul(w, H[2][a]) * n[2];
            gn[a] = re_mul(w, g[a]);
        }
        const double q = dot3(gn, n);
        for (int a = 0; a < 3; a++) {
            gN[a] = (gn[a] - q * n[a]) / tr.J;
            for (int t = 0; t < 3; t++) g9[3 * t + a] = gc[a] / 3.0;
        }
        normal_to_nodes(tr, gN, 0.0, g9);
        add_vertex_grad(grad, F, i, g9);
    }
}

// 2 Re[ mu_i d/dV alpha i k (d.n_i) exp(i k d.c_i) ]: the Burton-Miller term of the plane-wave
// right-hand side
__global__ void vjp_rhs_bm_kernel(const double *V, const int *F, int nf, double k, double dx, double dy, double dz,
                                  double2 alpha, const double2 *mu, double *grad)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x) {
        double nd[9], c[3], n[3], gN[3], g9[9];
        const double dv[3] = {dx, dy, dz};
        load_tri_d(V, F, i, nd);
        const Tri tr = tri_of(nd);
        for (int a = 0; a < 3; a++) {
            c[a] = nd[a] + (2.0 / 3.0) * (0.5 * (nd[3 + a] + nd[6 + a]) - nd[a]);
            n[a] = tr.N[a] / tr.J;
        }
        double sn, cs;
        sincos(k * dot3(dv, c), &sn, &cs);
        // b = i k alpha (d.n) e^{ik d.c}: by n i k alpha e d, by c i k b d
        const double2 z = cmul(cscale(cmul(mu[i], alpha), 2.0 * k), make_double2(-sn, cs));  // 2 mu alpha i k e
        const double dn = dot3(dv, n), gc = -k * dn * z.y, gn = z.x, gq = gn * dn;
        for (int a = 0; a < 3; a++) {
            gN[a] = (gn * dv[a] - gq * n[a]) / tr.J;
            for (int t = 0; t < 3; t++) g9[3 * t + a] = gc * dv[a] / 3.0;
        }
        normal_to_nodes(tr, gN, 0.0, g9);
        add_vertex_grad(grad, F, i, g9);
    }
}

// Coefficients of the derivatives of a regular expansion sum Psi[nm] R_n^m of order pl as
// expansions of order pl + 1 (from the G&D recurrences of dR/dz and (d/dx +- i d/dy) R):
//   dz  : k [ a(n,m) Psi_{n+1}^m - a(n-1,m) Psi_{n-1}^m ]
//   d+  : k [ b(n,-m) Psi_{n-1}^{m-1} - b(n+1,m-1) Psi_{n+1}^{m-1} ]
//   d-  : k [ b(n,m) Psi_{n-1}^{m+1} - b(n+1,-m-1) Psi_{n+1}^{m+1} ]
__global__ void deriv_coef_kernel(int nb, int pl, double k, const double2 *Psi, double2 *Dz, double2 *Dp, double2 *Dm)
{
    int po = pl + 1, po2 = po * po;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < (size_t)nb * po2; idx += (size_t)gridDim.x * blockDim.x) {
        int b = (int)(idx / po2), i = (int)(idx % po2);
        int n = (int)sqrt((double)i);
        while (n * n > i) n--;
        while ((n + 1) * (n + 1) <= i) n++;
        int m = i - n * n - n;
        const double2 *S = Psi + (size_t)b * pl * pl;
        auto at = [&](int nn, int mm) -> double2 {
            if (nn < 0 || nn >= pl || mm > nn || mm < -nn) return make_double2(0.0, 0.0);
            return S[nn * nn + nn + mm];
        };
        double2 a1 = at(n + 1, m), a0 = at(n - 1, m);
        double ca1 = coefA(n, m), ca0 = coefA(n - 1, m);
        Dz[idx] = make_double2(k * (ca1 * a1.x - ca0 * a0.x), k * (ca1 * a1.y - ca0 * a0.y));
        double2 p0 = at(n - 1, m - 1), p1 = at(n + 1, m - 1);
        double cp0 = coefB(n, -m), cp1 = coefB(n + 1, m - 1);
        Dp[idx] = make_double2(k * (cp0 * p0.x - cp1 * p1.x), k * (cp0 * p0.y - cp1 * p1.y));
        double2 q0 = at(n - 1, m + 1), q1 = at(n + 1, m + 1);
        double cq0 = coefB(n, m), cq1 = coefB(n + 1, -m - 1);
        Dm[idx] = make_double2(k * (cq0 * q0.x - cq1 * q1.x), k * (cq0 * q0.y - cq1 * q1.y));
    }
}

// far pairs, source side: -2 Re[ x_j d/dV_j sum_q w_q (b phi(y_q) J + c grad phi(y_q) . N) ] with
// phi = sum_nm Psi_j[nm] R_n^m(. - C), grad phi and its gradient from its derivative expansions, and
// N = J nh the unnormalised normal; one thread per element and quadrature point
__global__ void __launch_bounds__(128)
vjp_far_source_kernel(const double *V, const int *F, int nf, int pl, double k, int rule, double2 bco, double2 cco,
                      const int *elem_leaf, const double *box_ctr, const double2 *Psi, const double2 *Dz,
                      const double2 *Dp, const double2 *Dm, const double2 *x, double *grad)
{
    const int po = pl + 1, nq = v_rule_n[rule], id = blockIdx.x * blockDim.x + threadIdx.x, q = id / nf, j = id % nf;
    if (q >= nq) return;
    double nd[9], v[3], gs[9], gN[3], gJ = 0.0;
    load_tri_d(V, F, j, nd);
    const int b = elem_leaf[j];
    const Tri tr = tri_of(nd);
    const double *bb = &v_rule_bary[rule][3 * q], wq = v_rule_w[rule][q];
    for (int a = 0; a < 3; a++) v[a] = bb[0] * nd[a] + bb[1] * nd[3 + a] + bb[2] * nd[6 + a] - box_ctr[3 * b + a];
    const double2 w = cscale(x[j], -2.0 * wq), wb = cmul(w, bco), wc = cmul(w, cco);
    const double2 *coef[3] = {Dz + (size_t)b * po * po, Dp + (size_t)b * po * po, Dm + (size_t)b * po * po};
    double2 e[3], de[3][3], g[3], H[3][3];
    eval_expansions<3, true>(po, k, v, coef, e, de);
    cartesian(e, de, g, H);
    if (bco.x != 0.0 || bco.y != 0.0) {
        const double2 *c1[1] = {Psi + (size_t)b * pl * pl};
        double2 phi[1];
        eval_expansions<1, false>(pl, k, v, c1, phi, nullptr);
        gJ = re_mul(wb, phi[0]);
    }
    for (int a = 0; a < 3; a++) {
        const double gy = tr.J * re_mul(wb, g[a]) + re_mul(wc, H[0][a]) * tr.N[0] + re_mul(wc, H[1][a]) * tr.N[1] +
                          re_mul(wc, H[2][a]) * tr.N[2];
        gN[a] = re_mul(wc, g[a]);
        for (int t = 0; t < 3; t++) gs[3 * t + a] = bb[t] * gy;
    }
    normal_to_nodes(tr, gN, gJ, gs);
    add_vertex_grad(grad, F, j, gs);
}

// g_beta[j] = i k ( (w_j - z_j) x_j - (alpha/2) mu_j x_j ): the admittance derivative per
// element (see fmm_vjp_admittance)
__global__ void vjp_admittance_kernel(int nf, double k, double2 alpha, const double2 *w, const double2 *z,
                                      const double2 *mu, const double2 *x, double2 *g)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nf; j += gridDim.x * blockDim.x) {
        double2 gb = cmul(csub(w[j], z[j]), x[j]);
        double2 ga = cmul(mu[j], x[j]);
        double2 t = csub(gb, cscale(cmul(alpha, ga), 0.5));
        g[j] = make_double2(-k * t.y, k * t.x);
    }
}

} // namespace fmm

using namespace fmm;

// lanes that share an element's far points: a power of two up to a warp
static int point_group(int npts)
{
    int g = 1;
    while (g < 32 && g < npts) g *= 2;
    return g;
}

static std::vector<double> leaf_centres(const Plan *P)
{
    const LevelDev &L = P->lev[P->lmax];
    std::vector<double> ctr(3 * (size_t)L.nb);
    double h = ldexp(1.0, -P->lmax), h2 = ldexp(1.0, -P->lmax - 1);
    for (int i = 0; i < L.nb; i++) {
        int x, y, z;
        box_xyz(P->tree.sets[P->lmax][i], P->lmax, &x, &y, &z);
        ctr[3 * i] = P->tree.d * (h * x + h2) + P->tree.pt_min[0];
        ctr[3 * i + 1] = P->tree.d * (h * y + h2) + P->tree.pt_min[1];
        ctr[3 * i + 2] = P->tree.d * (h * z + h2) + P->tree.pt_min[2];
    }
    return ctr;
}

namespace fmm {
int solve_transposed(Plan *P, const double2 *rhs_dev, double2 *x_dev, double tol, int maxit, int restart, int precision,
                     int *iters, double *relres);
}

extern "C" int fmm_vjp(fmm_plan *plan, const cuDoubleComplex *x, const double *dir, const double *pts, int npts,
                       const cuDoubleComplex *pbar, double tol, int precision, double *grad, cuDoubleComplex *lambda)
{
    Plan *P = (Plan *)plan;
    if (!P || !x || !pts || npts < 1 || !pbar || !grad || !(tol > 0)) { fmm_set_error("fmm_vjp: invalid argument"); return FMM_ERR_ARG; }
    if (precision != FMM_FP64 && precision != FMM_MIXED) { fmm_set_error("fmm_vjp: unknown precision"); return FMM_ERR_ARG; }
    if (P->pleaf + 1 > VJP_PMAX) { fmm_set_error("fmm_vjp: leaf order %d above %d", P->pleaf, VJP_PMAX - 1); return FMM_ERR_ARG; }

    int nf = P->nf, nv = P->nv, pl = P->pleaf, lmax = P->lmax;
    int nbl = P->lev[lmax].nb;
    cudaStream_t st = P->stream;
    int rc = build_transpose(P);
    if (rc) return rc;
    if ((rc = upload_vjp_rules())) return rc;
    size_t loc = (size_t)nbl * pl * pl, locd = (size_t)nbl * (pl + 1) * (pl + 1);
    double2 *xd = nullptr, *pb = nullptr, *rhs = nullptr, *mu = nullptr, *tmp = nullptr, *D = nullptr, *Dz = nullptr, *Dp = nullptr,
            *Dm = nullptr;
    double *ptd = nullptr, *gd = nullptr, *ctr = nullptr, *tgt = nullptr;
    std::vector<double> hctr = leaf_centres(P);
#define VTRY(call)                                                                                              \
    do {                                                                                                        \
        cudaError_t e_ = (call);                                                                                \
        if (e_ != cudaSuccess) { fmm_set_error("fmm_vjp: %s: %s", #call, cudaGetErrorString(e_)); rc = FMM_ERR_CUDA; goto done; } \
    } while (0)
    VTRY(cudaMalloc(&xd, sizeof(double2) * nf));
    VTRY(cudaMalloc(&pb, sizeof(double2) * npts));
    VTRY(cudaMalloc(&rhs, sizeof(double2) * nf));
    VTRY(cudaMalloc(&mu, sizeof(double2) * nf));
    VTRY(cudaMalloc(&tmp, sizeof(double2) * nf));
    VTRY(cudaMalloc(&D, sizeof(double2) * loc));
    VTRY(cudaMalloc(&Dz, sizeof(double2) * locd));
    VTRY(cudaMalloc(&Dp, sizeof(double2) * locd));
    VTRY(cudaMalloc(&Dm, sizeof(double2) * locd));
    VTRY(cudaMalloc(&ptd, sizeof(double) * 3 * npts));
    VTRY(cudaMalloc(&gd, sizeof(double) * 3 * nv));
    VTRY(cudaMalloc(&ctr, sizeof(double) * hctr.size()));
    VTRY(cudaMalloc(&tgt, sizeof(double) * 6 * nf));
    VTRY(cudaMemcpyAsync(xd, x, sizeof(double2) * nf, cudaMemcpyDefault, st));
    VTRY(cudaMemcpyAsync(pb, pbar, sizeof(double2) * npts, cudaMemcpyDefault, st));
    VTRY(cudaMemcpyAsync(ptd, pts, sizeof(double) * 3 * npts, cudaMemcpyDefault, st));
    VTRY(cudaMemcpyAsync(ctr, hctr.data(), sizeof(double) * hctr.size(), cudaMemcpyHostToDevice, st));
    VTRY(cudaMemsetAsync(gd, 0, sizeof(double) * 3 * nv, st));
    VTRY(cudaMemsetAsync(mu, 0, sizeof(double2) * nf, st));
    VTRY(cudaMemsetAsync(tgt, 0, sizeof(double) * 6 * nf, st));
    {
        // elementwise kernels: small CTAs, so that a few thousand elements reach every SM
        const int T = 32, B = (nf + T - 1) / T, grp = point_group(npts), PB = (int)(((long long)nf * grp + 127) / 128);
        // adjoint system A^T mu = F^T conj(pbar)
        double2 nb = make_double2(-P->opt.b_re, -P->opt.b_im), nc = make_double2(-P->opt.c_re, -P->opt.c_im);
        vjp_adjoint_rhs_kernel<<<PB, 128, 0, st>>>(P->V_dev, P->F_dev, nf, P->opt.k, P->opt.rule, nb, nc, ptd, npts, pb,
                                                  rhs, grp);
        VTRY(cudaGetLastError());
        int it = 0;
        double rr = 0.0;
        rc = solve_transposed(P, rhs, mu, tol, 1000, 60, precision, &it, &rr);
        if (rc != FMM_OK && rc != FMM_ERR_NOT_CONVERGED) goto done;
        if (rc == FMM_ERR_NOT_CONVERGED) { fmm_set_error("fmm_vjp: adjoint GMRES stopped at %.3g > %.3g", rr, tol); goto done; }
        // forward leaf locals D (FP64 pass on x), then the transposed leaf locals Psi (on mu)
        if ((rc = run_matvec(P, xd, tmp, FMM_FP64, 0, 1))) goto done;
        VTRY(cudaMemcpyAsync(D, P->lev[lmax].Dl64, sizeof(double2) * loc, cudaMemcpyDeviceToDevice, st));
        if ((rc = run_matvec(P, mu, tmp, FMM_FP64, 1, 1))) goto done;
        deriv_coef_kernel<<<(unsigned)std::min<size_t>((locd + 255) / 256, 152 * 8), 256, 0, st>>>(nbl, pl, P->opt.k,
                                                                                                 P->lev[lmax].Dl64, Dz, Dp, Dm);
        double2 bco = make_double2(P->opt.b_re, P->opt.b_im), cco = make_double2(P->opt.c_re, P->opt.c_im);
        vjp_far_source_kernel<<<(unsigned)(((long long)nf * 9 + 127) / 128), 128, 0, st>>>(P->V_dev, P->F_dev, nf, pl, P->opt.k, P->opt.rule, bco, cco, P->elem_leaf,
                                               ctr, P->lev[lmax].Dl64, Dz, Dp, Dm, xd, gd);
        vjp_far_target_kernel<<<B, T, 0, st>>>(P->V_dev, P->F_dev, nf, pl, P->opt.k, P->elem_leaf, ctr, D, mu, gd);
        const double2 alpha = make_double2(P->opt.alpha_re, P->opt.alpha_im);
        const bool bm = alpha.x != 0.0 || alpha.y != 0.0;
        if (bm) {
            // target-side normal derivative of the far field: the derivative expansions of D
            // (Dz, Dp, Dm are free again once the source kernel above has run)
            deriv_coef_kernel<<<(unsigned)std::min<size_t>((locd + 255) / 256, 152 * 8), 256, 0, st>>>(nbl, pl, P->opt.k,
                                                                                                     D, Dz, Dp, Dm);
            vjp_far_target_bm_kernel<<<B, T, 0, st>>>(P->V_dev, P->F_dev, nf, pl, P->opt.k, alpha, P->elem_leaf, ctr, Dz,
                                                      Dp, Dm, mu, gd);
            if (dir)
                vjp_rhs_bm_kernel<<<B, T, 0, st>>>(P->V_dev, P->F_dev, nf, P->opt.k, dir[0], dir[1], dir[2], alpha, mu, gd);
        }
        const unsigned NB = (unsigned)((P->num_near + 127) / 128);
        if (bm)
            vjp_near_kernel<true><<<NB, 128, 0, st>>>(P->V_dev, P->F_dev, nf, P->num_near, P->near_beg, P->near_col, P->opt.k,
                                                      bco, cco, alpha, P->opt.rule, mu, xd, gd, tgt);
        else
            vjp_near_kernel<false><<<NB, 128, 0, st>>>(P->V_dev, P->F_dev, nf, P->num_near, P->near_beg, P->near_col, P->opt.k,
                                                       bco, cco, alpha, P->opt.rule, mu, xd, gd, tgt);
        vjp_near_self_kernel<<<(3 * nf + T - 1) / T, T, 0, st>>>(P->V_dev, P->F_dev, nf, P->opt.k, bco, cco, alpha, mu, xd, tgt, gd);
        vjp_farpts_kernel<<<PB, 128, 0, st>>>(P->V_dev, P->F_dev, nf, P->opt.k, P->opt.rule, nb, nc, ptd, npts, pb, xd, gd, grp);
        if (dir)
            vjp_rhs_kernel<<<B, T, 0, st>>>(P->V_dev, P->F_dev, nf, P->opt.k, dir[0], dir[1], dir[2], mu, gd);
        VTRY(cudaGetLastError());
        VTRY(cudaMemcpyAsync(grad, gd, sizeof(double) * 3 * nv, cudaMemcpyDefault, st));
        if (lambda) {
            // lambda = conj(mu)
            launch_conj(P, mu, tmp, nf);
            VTRY(cudaMemcpyAsync(lambda, tmp, sizeof(double2) * nf, cudaMemcpyDefault, st));
        }
        VTRY(cudaStreamSynchronize(st));
        rc = FMM_OK;
    }
done:
#undef VTRY
    for (void *q : {(void *)xd, (void *)pb, (void *)rhs, (void *)mu, (void *)tmp, (void *)D, (void *)Dz, (void *)Dp, (void *)Dm,
                    (void *)ptd, (void *)gd, (void *)ctr, (void *)tgt})
        if (q) cudaFree(q);
    return rc;
}

// Admittance derivative of the far-field objective of fmm_vjp.  For a locally reacting surface
// dp/dn = i k beta_j p on element j the operator is A = a I + (1 + alpha d/dn_y)(L B + c M), with
// B = diag(b_j), b_j = i k beta_j at the source elements and, with the Burton-Miller coupling,
// a_i = (1 + alpha b_i)/2 at the targets; the far field is F x = M x - L_far (B x).  So
//     dJ = 2 Re sum_j g_j dbeta_j,
//     g_j = i k [ x_j (w_j - z_j) - (alpha/2) conj(lambda_j) x_j ],
// w = (dF/db)^T conj(pbar) (the far-field operator with b = 1, c = 0), z = S^T conj(lambda) with
// S = (1 + alpha d/dn_y) L: one transposed FP64 FMM pass of the plan with its element tables and
// near-field matrix regenerated for (a, b, c) = (0, 1, 0), on temporary buffers that stand in for
// the plan's own during the pass.
extern "C" int fmm_vjp_admittance(fmm_plan *plan, const cuDoubleComplex *x, const double *pts, int npts,
                                  const cuDoubleComplex *pbar, const cuDoubleComplex *lambda, cuDoubleComplex *g_beta,
                                  double *dJ_dbeta)
{
    Plan *P = (Plan *)plan;
    if (!P || !x || !pts || npts < 1 || !pbar || !lambda || (!g_beta && !dJ_dbeta)) {
        fmm_set_error("fmm_vjp_admittance: invalid argument");
        return FMM_ERR_ARG;
    }
    int nf = P->nf, pl = P->pleaf;
    cudaStream_t st = P->stream;
    int rc = build_transpose(P);
    if (rc) return rc;
    size_t tbl = (size_t)nf * pl * pl;
    long long nnz = P->num_near;
    double2 *xd = nullptr, *mu = nullptr, *pb = nullptr, *w = nullptr, *z = nullptr, *U = nullptr, *Rv = nullptr,
            *nearL = nullptr, *nearTL = nullptr, *g = nullptr;
    double *ptd = nullptr;
    std::vector<double2> hg;
#define ATRY(call)                                                                                                 \
    do {                                                                                                           \
        cudaError_t e_ = (call);                                                                                   \
        if (e_ != cudaSuccess) { fmm_set_error("fmm_vjp_admittance: %s: %s", #call, cudaGetErrorString(e_)); rc = FMM_ERR_CUDA; goto done; } \
    } while (0)
    ATRY(cudaMalloc(&xd, sizeof(double2) * nf));
    ATRY(cudaMalloc(&mu, sizeof(double2) * nf));
    ATRY(cudaMalloc(&w, sizeof(double2) * nf));
    ATRY(cudaMalloc(&z, sizeof(double2) * nf));
    ATRY(cudaMalloc(&g, sizeof(double2) * nf));
    ATRY(cudaMalloc(&pb, sizeof(double2) * npts));
    ATRY(cudaMalloc(&ptd, sizeof(double) * 3 * npts));
    ATRY(cudaMalloc(&U, sizeof(double2) * tbl));
    ATRY(cudaMalloc(&Rv, sizeof(double2) * tbl));
    ATRY(cudaMalloc(&nearL, sizeof(double2) * (nnz + 1)));
    ATRY(cudaMalloc(&nearTL, sizeof(double2) * (nnz + 1)));
    ATRY(cudaMemcpyAsync(xd, x, sizeof(double2) * nf, cudaMemcpyDefault, st));
    ATRY(cudaMemcpyAsync(w, lambda, sizeof(double2) * nf, cudaMemcpyDefault, st));
    ATRY(cudaMemcpyAsync(pb, pbar, sizeof(double2) * npts, cudaMemcpyDefault, st));
    ATRY(cudaMemcpyAsync(ptd, pts, sizeof(double) * 3 * npts, cudaMemcpyDefault, st));
    launch_conj(P, w, mu, nf); // mu = conj(lambda)
    ATRY(cudaGetLastError());
    if ((rc = gen_operator_part(P, make_double2(1.0, 0.0), make_double2(0.0, 0.0), U, Rv, nearL))) goto done;
    if ((rc = near_transpose_values(P, nearL, nearTL))) goto done;
    {
        // z = S^T mu with the single-layer part standing in for the plan's operator
        double2 *sU = P->U64, *sN = P->near64, *sNT = P->nearT64;
        fmm_options so = P->opt;
        P->U64 = U;
        P->near64 = nearL;
        P->nearT64 = nearTL;
        P->opt.a_re = P->opt.a_im = 0.0;
        P->opt.b_re = 1.0;
        P->opt.b_im = 0.0;
        P->opt.c_re = P->opt.c_im = 0.0;
        rc = run_matvec(P, mu, z, FMM_FP64, 1, 1);
        cudaError_t e2 = cudaStreamSynchronize(st);
        P->U64 = sU;
        P->near64 = sN;
        P->nearT64 = sNT;
        P->opt = so;
        if (rc) goto done;
        ATRY(e2);
    }
    {
        const int T = 128, B = std::min((nf + T - 1) / T, 152 * 8);
        // w = (dF/db)^T conj(pbar): the far-field operator -int G of unit b
        const int grp = point_group(npts), PB = (int)(((long long)nf * grp + 127) / 128);
        vjp_adjoint_rhs_kernel<<<PB, 128, 0, st>>>(P->V_dev, P->F_dev, nf, P->opt.k, P->opt.rule, make_double2(-1.0, 0.0),
                                                  make_double2(0.0, 0.0), ptd, npts, pb, w, grp);
        vjp_admittance_kernel<<<B, T, 0, st>>>(nf, P->opt.k, make_double2(P->opt.alpha_re, P->opt.alpha_im), w, z, mu, xd, g);
        ATRY(cudaGetLastError());
        hg.resize(nf);
        ATRY(cudaMemcpyAsync(hg.data(), g, sizeof(double2) * nf, cudaMemcpyDeviceToHost, st));
        ATRY(cudaStreamSynchronize(st));
        if (g_beta) ATRY(cudaMemcpy(g_beta, hg.data(), sizeof(double2) * nf, cudaMemcpyDefault));
        if (dJ_dbeta) {
            double sr = 0.0, si = 0.0;
            for (int j = 0; j < nf; j++) { sr += hg[j].x; si += hg[j].y; }
            dJ_dbeta[0] = 2.0 * sr;  // dJ/dRe(beta) = 2 Re g
            dJ_dbeta[1] = -2.0 * si; // dJ/dIm(beta) = 2 Re(i g)
        }
        rc = FMM_OK;
    }
done:
#undef ATRY
    for (void *q : {(void *)xd, (void *)mu, (void *)pb, (void *)w, (void *)z, (void *)U, (void *)Rv, (void *)nearL,
                    (void *)nearTL, (void *)g, (void *)ptd})
        if (q) cudaFree(q);
    return rc;
}
