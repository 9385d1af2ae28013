// Batched translation passes of the mixed path on the 5th-generation tensor cores
// (tcgen05.mma, kind::tf32) as dense operators: the M2L of the levels whose operators are small
// enough to store densely (p <= 16, the levels that carry most translations) and, on request,
// the M2M and L2L of those levels.
//
// The translation of direction d is T_d = diag(e^{-i m' phi_d}) S_c diag(e^{i m phi_d}) (the RCR
// product of translation.cu:1864-1961 with its azimuthal phases taken out), where S_c (p^2 x p^2
// complex, formed once at plan time) depends only on the polar angle and the distance of d: the
// 316 M2L directions fall into 61 classes c of equal (dz, dx^2 + dy^2), the 8 octants of M2M and
// L2L into 2.  S_c moves along a vector of the x-z plane, so the reflection y -> -y (m -> -m)
// commutes with it: in the sums and differences x_m + x_-m, x_m - x_-m (m >= 0) of the phased
// source it falls into two blocks of p (p + 1) / 2 and p (p - 1) / 2 coefficients, half the
// products of the whole operator.  A tile is 128 translations of one class (times right-hand
// sides); the pass is the pair of real GEMMs
//     D[t][o] = sum_k A[t][k] B[o][k],   A = sums (differences) of the phased source, re and im,
//                                         B = the block, embedded as a real matrix,
// and the epilogue turns sums and differences back into m and -m and applies e^{-i m' phi} of the
// row's own direction.  (Levels with fewer translations keep the whole operator, a chunk's first and last four
// coefficients as the two operands, fold_pays().)  Split TF32 (3 products hi*hi + hi*lo + lo*hi of rounded 11-bit halves)
// gives close to FP32 accuracy.
//
// A persistent, warp-specialised kernel (one CTA per SM, 20 warps) runs over the tiles
// (128 translations x one range of output degrees):
//   warp 0     issues the MMAs (one thread) into a set of TMEM accumulators (of two, or the one) and
//              commits each K chunk to its stage's "empty" barrier, each tile to its
//              accumulators' "full" barrier;
//   warp 1     copies the operator's K chunks (hi and lo tiles of both blocks) with cp.async.bulk;
//   warps 2, 3 copy the source expansions, row by row, in pieces of whole degrees;
//   warps 4-11 (two per TMEM lane quarter, on alternate chunks; lane = row) read four coefficient
//              pairs (n, m), (n, -m) of their row, apply its phases, form sums and differences,
//              split them into TF32 hi / lo and write them to TMEM as the MMA's A operand;
//   warps 12-19 (two per quarter, each its groups of degrees) read the finished accumulators, form the
//              group's coefficients of their row in shared memory and add them into the destination
//              expansions, a row's group with one bulk reduction (single coefficients with atomics where it does
//              not lie on 16 bytes), overlapping the next tile's MMAs where there are two sets.
// Every wait has a time limit, after which the thread sets the plan's error flag and stops.
//
// What bounds it: 16 columns on the 81,920-triangle sphere, p = 14 (192,528 translations) 2.77 ms and
// p = 10 (650,304) 2.82 ms.  At p = 10 a tile takes 8,900 cycles, of which the MMAs need 4,400 (52 cycles
// each at N = 112 / 96, the full TF32 rate) and the reductions into L2 4,900 (20 bytes a cycle and SM is
// what the L2 takes from all of them); the issue slots are 71 % busy, a third of them with A's phases
// and splits.  At p = 14 (one set of accumulators) reading them out, 10,000 of 36,000 cycles, is not hidden.  Through L2
// go 10 and 14 TB/s, half of it at p = 14 and a third at p = 10 the operator, streamed again for every tile.  An earlier
// form, with the whole operator, A in shared memory and one atomic per 16 bytes of output, took 5.96
// and 5.58 ms (its load/store unit 80 % busy with rows read 16 bytes a lane, A's stores and the atomics).
// Orders up to 5 are bound by the epilogue's work per row: one group of all degrees, a tile each for the two warps of
// a quarter in turn, and rows on odd coefficients (odd p^2) as many at a time as the others (649,008 translations, one
// column: p = 4 115 -> 95 us, p = 5 216 -> 138, p = 9 414 -> 309, p = 10 274 -> 256).
// What made the difference: half the products; A through TMEM; source rows by cp.async, a row per
// instruction; outputs by bulk reductions, a row's group per instruction; the MMA's issue by one
// elected thread with operands in uniform registers (500 instead of 950 cycles per six MMAs).
#include "plan.h"
#include "tc_common.cuh"
#include "f32x2.cuh"
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

namespace fmm {

constexpr int TC_M = 128;               // translations per tile (MMA M)
constexpr int TC_KC = 8;                // K per chunk and block: four complex inputs (n, m >= 0)
constexpr int TC_RW = 2;                // warps that copy source rows
constexpr int TC_A0 = 2 + TC_RW, TC_AW = 8;  // source warps
constexpr int TC_E0 = TC_A0 + TC_AW, TC_EW = 8;  // epilogue warps
constexpr int TC_THREADS = 32 * (TC_E0 + TC_EW);
// orders up to 16: at p = 20 the dense form's rounding (FP32 accumulation of 300 split products
// per output) raised the iterations of the refined 64-column solve on the 200,000-triangle
// head-like body from 48 to 56, which cost more than its faster M2L saved
constexpr int TC_MAXP = 16;
constexpr int TC_SLOTS = 2;             // pieces of 128 rows in shared memory
constexpr int TC_STAGES = 6;            // stages of the operands, at most
constexpr int TC_ACOL = 4 * TC_KC;      // TMEM columns of an A stage: hi and lo of both blocks
constexpr size_t TC_SMEM_MAX = 232448;  // 227 KB of dynamic shared memory per CTA

struct TcPass {
    TcShape sh;
    const int4 *items;
    const int *g_src, *g_dst, *g_dir;    // per translation (class order): boxes and direction
    const float2 *PH;                    // phases e^{i m phi} of direction d at d phstride + phoff + m
    int phstride, phoff;
    int nrhs, P2, P2o, ntiles;           // P2 = pin^2, P2o = pout^2
    unsigned long long per;              // e / nrhs = e per >> shift for columns e < 2^31: per = 2^shift / nrhs, rounded
    int shift;                           // up, 2^(shift - 31) >= nrhs
    const float *B;
    const float2 *src;
    float2 *dst;
    int *err;
};

static __host__ __device__ __forceinline__ int up16(int n) { return (n + 15) / 16 * 16; }

// stride of a row of `coefs` coefficients in shared memory, one to spare: 16-byte steps, an odd number
static int tc_stride(int coefs) { return 16 * (((8 * coefs + 8 + 15) / 16) | 1); }
static size_t tc_smem_bytes(const TcShape &g)
{
    return (size_t)g.nst * g.bstage + (size_t)TC_SLOTS * TC_M * g.row_stride + (size_t)TC_EW * 32 * g.epi_stride +
           (2 * (TC_SLOTS + g.nst) + 4) * 8 + 16;
}

// The pass's shape for source order pin and destination order pout.
// Inputs, folded: the pairs (n, m >= 0), degree by degree, in pieces of whole degrees (a row's copy), each
// piece in chunks of four; the cut with the fewest chunks.  Not folded: the coefficients in their order,
// eight a chunk (two steps of the MMA's K one after another).
// Outputs: ranges of degrees, each two blocks of MMA columns (rounded up to 16, at most 256).  Where
// all degrees take at most 208 columns (p <= 10), two sets of accumulators and three A stages fit
// into the 512 of TMEM, and the epilogue overlaps the next tile's MMAs; beyond, one set of up to 416 columns
// (the cut with the fewest): forming A once for all of a row's outputs saves more than the
// overlap would (17.5 against 17.8 ms for 16 columns on the 81,920-triangle sphere, 1.13 against 1.17 ms for
// one on a 27,380-triangle body with p = 16 and 12).  Without the fold a chunk's operator takes twice the
// room, so there are always ranges of at most 208 columns and two sets.
// Pieces and groups as large as shared memory allows.
static bool tc_shape(int pin, int pout, int fold, TcShape &g)
{
    if (pin < 4 || pin > TC_MAXP || pout < 4 || pout > TC_MAXP) return false;
    auto tri = [](int n) { return n * (n + 1) / 2; };
    auto cut = [](int p, auto cost, std::vector<int> &at) {  // cost(a, b) < 0: degrees [a, b) do not fit
        std::vector<int> best(p + 1, 1 << 30), from(p + 1, 0);
        best[0] = 0;
        for (int b = 1; b <= p; b++)
            for (int a = 0; a < b; a++) {
                const int c = cost(a, b);
                if (c >= 0 && best[a] + c < best[b]) best[b] = best[a] + c, from[b] = a;
            }
        at.clear();
        for (int b = p; b > 0; b = from[b]) at.push_back(from[b]);
        std::reverse(at.begin(), at.end());
        at.push_back(p);
    };
    std::vector<int> at;
    auto sums = [&](int a, int b) { return up16(2 * (tri(b) - tri(a))); };
    auto diffs = [&](int a, int b) { return up16(std::max(2 * (tri(b - 1) - tri(a - 1)), 16)); };
    g.fold = fold;
    g.sets = !fold || sums(0, pout) + diffs(0, pout) <= 208 ? 2 : 1;
    const int most_columns = fold ? 416 : 208, parts = fold ? 1 : 2;
    cut(pout, [&](int a, int b) {
        const int w = sums(a, b) + diffs(a, b);
        return w > most_columns || sums(a, b) > 256 ? -1 : w + 8;
    }, at);
    g.nsub = (int)at.size() - 1;
    if (g.nsub > TC_MAXSUB) return false;
    g.setw = 0;
    for (int i = 0; i < g.nsub; i++) {
        TcSub &s = g.sub[i];
        s.beg = at[i];
        s.end = at[i + 1];
        s.nP = sums(s.beg, s.end);
        s.nQ = diffs(s.beg, s.end);
        g.setw = std::max(g.setw, s.nP + s.nQ);
    }
    g.bstage = parts * 2 * TC_KC * 4 * g.setw;
    static const int sizes[][2] = {{53, 36}, {53, 32}, {36, 36}, {36, 32}, {31, 31}};  // a degree of p <= 16 has up to 31
    for (auto &size : sizes) {
        const int piece = size[0], group = size[1];
        g.nch = g.row_stride = 0;
        if (fold) {
            cut(pin, [&](int a, int b) { return b * b - a * a > piece ? -1 : 64 * ((tri(b) - tri(a) + 3) / 4) + 1; }, at);
        } else {  // runs of whole chunks
            at.clear();
            for (int c = 0; c < pin * pin; c += piece / 8 * 8) at.push_back(c);
            at.push_back(pin * pin);
        }
        g.npiece = (int)at.size() - 1;
        if (g.npiece > TC_MAXPIECE) continue;
        for (int i = 0; i < g.npiece; i++) {
            const int a = at[i], b = at[i + 1], c0 = fold ? a * a : a, cnt = fold ? b * b - c0 : b - a;
            const int nc = fold ? (tri(b) - tri(a) + 3) / 4 : (cnt + 7) / 8;
            g.piece[i] = {c0, cnt, g.nch, g.nch + nc};
            g.row_stride = std::max(g.row_stride, tc_stride(cnt));
            if (g.nch + nc > TC_MAXCH) return false;
            int k = 4 * g.nch;
            if (fold) {
                for (int n = a; n < b; n++)
                    for (int m = 0; m <= n; m++) g.tab[k++] = {8 * (n * n + n + m - c0), 8 * (n * n + n - m - c0), 8 * m, 0};
                while (k < 4 * (g.nch + nc)) g.tab[k++] = {0, 0, 0, TC_PAD};  // coefficient 0 of the piece against a zero operator
            } else {
                for (; k < 4 * (g.nch + nc); k++) {
                    const int lo = 8 * (k / 4) + k % 4, hi = lo + 4;
                    auto order = [](int i) { int n = 0; while ((n + 1) * (n + 1) <= i) n++; return i - n * n - n; };
                    g.tab[k] = {lo < b ? 8 * (lo - c0) : 0, hi < b ? 8 * (hi - c0) : 0, lo < b ? 8 * order(lo) : 0, hi < b ? 8 * order(hi) : 0};
                }
            }
            g.nch += nc;
        }
        g.epi_stride = tc_stride(group);
        for (int i = 0; i < g.nsub; i++) {
            // groups of degrees of the epilogue, few of them and few that start on an odd coefficient (all degrees in
            // one where it holds them), and the warp of a quarter that takes each (the larger first, to the warp
            // with less; with two sets of accumulators the warps change roles from tile to tile)
            TcSub &s = g.sub[i];
            const int all = s.end * s.end - s.beg * s.beg;
            const int most = all <= group ? group : std::min(group, std::max(2 * s.end - 1, all / 2 + 8));
            cut(s.end - s.beg, [&](int a, int b) {
                a += s.beg, b += s.beg;
                return b * b - a * a > most ? -1 : 3 + 2 * (a & 1);
            }, at);
            s.ngrp = (int)at.size() - 1;
            for (int k = 0; k <= s.ngrp; k++) s.grp[k] = (unsigned char)(s.beg + at[k]);
            auto coefs = [&](int k) { return s.grp[k + 1] * s.grp[k + 1] - s.grp[k] * s.grp[k]; };
            std::vector<int> order(s.ngrp);
            for (int k = 0; k < s.ngrp; k++) order[k] = k;
            std::sort(order.begin(), order.end(), [&](int a, int b) { return coefs(a) > coefs(b); });
            int load[2] = {0, 0};
            s.second = 0;
            for (int k : order) {
                const int w = load[1] < load[0];
                load[w] += coefs(k);
                s.second |= (unsigned)w << k;
            }
        }
        const int room = (512 - g.sets * g.setw) / TC_ACOL;
        for (g.nst = std::min(TC_STAGES, room); g.nst > 3 && tc_smem_bytes(g) > TC_SMEM_MAX; g.nst--) {}
        if (g.nst >= 3 && tc_smem_bytes(g) <= TC_SMEM_MAX) {
            g.cls_floats = 0;
            for (int i = 0; i < g.nsub; i++) {
                g.sub[i].boff = g.cls_floats;
                g.cls_floats += parts * g.nch * 2 * TC_KC * (g.sub[i].nP + g.sub[i].nQ);
            }
            return true;
        }
    }
    return false;
}

__device__ __forceinline__ void tc_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_bulk(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tc_reduce(float2 *dst, uint32_t src, uint32_t bytes)
{
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void tc_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// one split product: A in TMEM, B in shared memory (low half of its descriptor; K-adjacent core
// matrices 128 bytes apart, groups of 8 rows 256)
constexpr uint32_t TC_DESC_LO = 128u >> 4 << 16, TC_DESC_HI = 256u >> 4 | 1u << 14;
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t add)
{
    asm volatile("{\n\t.reg .pred q;\n\t.reg .b64 bd;\n\tmov.b64 bd, {%2, %5};\n\tsetp.ne.b32 q, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], bd, %3, q;\n\t}" ::"r"(d),
                 "r"(a), "r"(b), "r"(idesc), "r"(add), "r"(TC_DESC_HI));
}

__device__ __forceinline__ void tc_ld16(uint32_t (&v)[16], uint32_t ta)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                   "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(ta));
}

__device__ __forceinline__ void tc_st32(uint32_t ta, const uint32_t (&v)[32])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
                 "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(ta),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                 "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
                 "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
                 "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
                 : "memory");
}

// a ring of stages: index and phase parity
struct Ring {
    int i = 0, par = 0;
    __device__ __forceinline__ void next(int n)
    {
        if (++i == n) {
            i = 0;
            par ^= 1;
        }
    }
};

// a row of a tile: its expansion's index box nrhs + rhs (< 0: none) and its direction
struct TileRow {
    int row = -1, dir = 0;
};

// the same looked up ahead: what the row is made of, as loaded
struct RowAhead {
    int box = 0, rhs = -1, dir = 0;
};
__device__ __forceinline__ RowAhead row_ahead(const TcPass &ps, int4 it, int r, const int *box)
{
    RowAhead o;
    if (r < it.z) {
        const int e = it.y + r, t = (int)(((unsigned long long)e * ps.per) >> ps.shift);
        o.box = __ldg(box + t);
        o.rhs = e - t * ps.nrhs;
        o.dir = __ldg(ps.g_dir + t);
    }
    return o;
}
__device__ __forceinline__ TileRow row_now(const TcPass &ps, const RowAhead &a)
{
    TileRow o;
    if (a.rhs >= 0) {
        o.row = a.box * ps.nrhs + a.rhs;
        o.dir = a.dir;
    }
    return o;
}

__device__ __forceinline__ TileRow tile_row(const TcPass &ps, int4 it, int r, const int *box)
{
    TileRow o;
    if (r < it.z) {
        const int e = it.y + r, t = (int)(((unsigned long long)e * ps.per) >> ps.shift);
        o.row = box[t] * ps.nrhs + (e - t * ps.nrhs);
        o.dir = ps.g_dir[t];
    }
    return o;
}

// What is copied of the cnt coefficients from c0 on of expansion `row` (P2 coefficients each; none where it is
// negative): n words of 16 bytes from the from-th on; with an odd first coefficient the one before it too.
struct RowCopy {
    unsigned long long from;
    int n;
};
__host__ __device__ __forceinline__ RowCopy row_copy(int row, int P2, int c0, int cnt)
{
    const unsigned long long e = (unsigned long long)(unsigned)row * (unsigned)P2 + (unsigned)c0;
    return RowCopy{e >> 1, row < 0 ? 0 : (cnt + (int)(e & 1) + 1) >> 1};
}

// Up to eight coefficient pairs (m = 0..last) of a degree from the columns of their sums (from p on) and
// differences (from q on, none for m = 0 where `first`) to y[m], y[-m] of the lane's row; columns past the last
// pair's are not used.
template <bool FOLD>
__device__ __forceinline__ void unfold(uint32_t p, uint32_t q, int last, const float2 (&f)[8], float2 *y, bool first)
{
    uint32_t u[16], w[16];
    tc_ld16(u, p);
    tc_ld16(w, q);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; j++) {
        if (j > last) break;
        const float sr = __uint_as_float(u[2 * j]), si = __uint_as_float(u[2 * j + 1]);
        if (first && j == 0) {
            y[0] = make_float2(sr, si);
            continue;
        }
        const float dr = __uint_as_float(w[2 * j]), di = __uint_as_float(w[2 * j + 1]);
        const float pr = FOLD ? sr + dr : sr, pi = FOLD ? si + di : si, mr = FOLD ? sr - dr : dr, mi = FOLD ? si - di : di;
        const int m = first ? j : j + 8;
        y[m] = make_float2(pr * f[j].x + pi * f[j].y, pi * f[j].x - pr * f[j].y);
        y[-m] = make_float2(mr * f[j].x - mi * f[j].y, mr * f[j].y + mi * f[j].x);
    }
}

// WIDE: source expansions of 64 GB and more, whose 16-byte words take more than 32 bits to count (a third
// exchange per row; in all passes it would cost 0.5 to 2 %).
template <bool FOLD, bool WIDE>
__global__ void __launch_bounds__(TC_THREADS, 1) tc_dense_kernel(const __grid_constant__ TcPass ps)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const TcShape &sh = ps.sh;
    const int nst = sh.nst, nsub = sh.nsub;
    unsigned char *rows = smem + (size_t)nst * sh.bstage;
    unsigned char *epi = rows + (size_t)TC_SLOTS * TC_M * sh.row_stride;
    uint64_t *bars = reinterpret_cast<uint64_t *>(epi + (size_t)TC_EW * 32 * sh.epi_stride);
    uint64_t *rfull = bars, *rempty = rfull + TC_SLOTS, *full = rempty + TC_SLOTS, *empty = full + nst, *accf = empty + nst,
             *acce = accf + 2;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(acce + 2);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 32) {
        auto init = [](uint64_t *b, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n)); };
        for (int i = 0; i < TC_SLOTS; i++) {
            init(rfull + i, 32 * TC_RW);  // row copies
            init(rempty + i, TC_AW);   // source warps
        }
        for (int i = 0; i < nst; i++) {
            init(full + i, 5);         // source warps of the chunk, one per lane quarter; operator copy
            init(empty + i, 1);        // MMA commit
        }
        for (int i = 0; i < 2; i++) {
            init(accf + i, 1);         // MMA commit
            init(acce + i, TC_EW);     // epilogue warps
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tslot, tmem_a = tmem + (uint32_t)(sh.sets * sh.setw);
    const int ntile = (ps.ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    // the CTA's i-th tile: its item and range of output degrees; where the grid is a multiple of the
    // ranges (of uneven width), each round takes the next one, so that every CTA meets them all
    const int spin = gridDim.x % nsub == 0 ? 1 : 0;
    auto tile = [&](int i) { return ((int)blockIdx.x + i * (int)gridDim.x) / nsub; };
    auto range = [&](int i) -> const TcSub & { return sh.sub[((int)blockIdx.x + i * ((int)gridDim.x + spin)) % nsub]; };
    // its accumulators: set and phase parity
    const int two = sh.sets == 2;
    auto set_of = [&](int i) { return two ? i & 1 : 0; };
    auto set_par = [&](int i) { return two ? (i >> 1) & 1 : i & 1; };
    bool ok = true;

    if (warp == 0) {
        // ---------------------------------------------------------------- MMA issuer
        // An MMA's issue waits until the tensor core can take it, so what lies between two chunks' MMAs is
        // time lost to it: one thread, and little arithmetic.
        if (elect_one()) {
            Ring rs;
            const uint32_t b0 = (smem_u32(smem) >> 4) | TC_DESC_LO, bstep = (uint32_t)sh.bstage >> 4;
            for (int i = 0; i < ntile && ok; i++) {
                const TcSub &s = range(i);
                const int a = set_of(i);
                const uint32_t kind = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TC_M >> 4) << 24);
                const uint32_t i1 = kind | (uint32_t)(s.nP >> 3) << 17, i2 = kind | (uint32_t)(s.nQ >> 3) << 17;
                const uint32_t d1 = tmem + (uint32_t)(a * sh.setw), d2 = d1 + (uint32_t)s.nP;
                const uint32_t l1 = (uint32_t)(s.nP * TC_KC) >> 2, l2 = (uint32_t)(s.nQ * TC_KC) >> 2;
                ok = mbar_wait(smem_u32(acce + a), set_par(i) ^ 1);
                uint32_t add = 0;
                for (int c = 0; c < sh.nch && ok; c++, add = 1) {
                    ok = mbar_wait(smem_u32(full + rs.i), rs.par);
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint32_t at = tmem_a + (uint32_t)(rs.i * TC_ACOL), b1 = b0 + (uint32_t)rs.i * bstep, b2 = b1 + 2 * l1;
                    const uint32_t a2 = at + 2 * TC_KC;
                    tc_mma(d1, at, b1, i1, add);
                    tc_mma(d1, at, b1 + l1, i1, 1);
                    tc_mma(d1, at + TC_KC, b1, i1, 1);
                    if constexpr (FOLD) {
                        tc_mma(d2, a2, b2, i2, add);
                        tc_mma(d2, a2, b2 + l2, i2, 1);
                        tc_mma(d2, a2 + TC_KC, b2, i2, 1);
                    } else {
                        const uint32_t c1 = b2 + 2 * l2, c2 = c1 + 2 * l1;
                        tc_mma(d2, at, b2, i2, add);
                        tc_mma(d2, at, b2 + l2, i2, 1);
                        tc_mma(d2, at + TC_KC, b2, i2, 1);
                        tc_mma(d1, a2, c1, i1, 1);
                        tc_mma(d1, a2, c1 + l1, i1, 1);
                        tc_mma(d1, a2 + TC_KC, c1, i1, 1);
                        tc_mma(d2, a2, c2, i2, 1);
                        tc_mma(d2, a2, c2 + l2, i2, 1);
                        tc_mma(d2, a2 + TC_KC, c2, i2, 1);
                    }
                    tc_commit(smem_u32(empty + rs.i));
                    rs.next(nst);
                }
                if (ok) tc_commit(smem_u32(accf + a));
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- operator copies
        if (lane == 0) {
            Ring rs;
            for (int i = 0; i < ntile && ok; i++) {
                const TcSub &s = range(i);
                const uint32_t fl = (uint32_t)((FOLD ? 2 : 4) * TC_KC * (s.nP + s.nQ));
                const float *B = ps.B + (size_t)ps.items[tile(i)].x * sh.cls_floats + s.boff;
                for (int c = 0; c < sh.nch; c++, B += fl) {
                    ok = mbar_wait(smem_u32(empty + rs.i), rs.par ^ 1);
                    if (!ok) break;
                    const uint32_t bar = smem_u32(full + rs.i);
                    tc_expect(bar, 4 * fl);
                    tc_bulk(smem_u32(smem + (size_t)rs.i * sh.bstage), B, 4 * fl, bar);
                    rs.next(nst);
                }
            }
        }
    } else if (warp < TC_A0) {
        // ---------------------------------------------------------------- source rows
        // A warp's rows one after another, a lane per 16 bytes (a bulk copy per row, issued by each row's
        // lane, took 80 cycles a row).  A row that starts on an odd coefficient is copied from
        // the one before on, one of odd length to the one after (the expansions are allocated
        // with one coefficient to spare).
        constexpr int NR = TC_M / TC_RW / 32;  // rows per lane
        const int r0 = (warp - 2) * 32 * NR;
        Ring rr;
        // rows are looked up a tile ahead, items two
        auto item = [&](int i) { return i < ntile ? ps.items[tile(i)] : make_int4(0, 0, 0, 0); };
        RowAhead next[NR];
        int4 it = item(0);
#pragma unroll
        for (int j = 0; j < NR; j++) next[j] = row_ahead(ps, it, r0 + lane + 32 * j, ps.g_src);
        it = item(1);
        for (int i = 0; i < ntile && ok; i++) {
            int at[NR];
#pragma unroll
            for (int j = 0; j < NR; j++) {
                at[j] = row_now(ps, next[j]).row;
                next[j] = row_ahead(ps, it, r0 + lane + 32 * j, ps.g_src);
            }
            it = item(i + 2);
            for (int pc = 0; pc < sh.npiece; pc++) {
                const int c0 = sh.piece[pc].c0, cnt = sh.piece[pc].cnt;
                ok = mbar_wait_warp(smem_u32(rempty + rr.i), rr.par ^ 1);
                if (!ok) break;
                uint32_t slot = smem_u32(rows + (size_t)(rr.i * TC_M + r0) * sh.row_stride) + 16 * lane;
                const char *src = reinterpret_cast<const char *>(ps.src) + 16 * lane;
#pragma unroll
                for (int j = 0; j < NR; j++) {
                    const RowCopy own = row_copy(at[j], ps.P2, c0, cnt);  // of the lane's own row
                    const uint32_t low = (uint32_t)own.from, high = (uint32_t)(own.from >> 32);
                    for (int k0 = 0; k0 < 32; k0 += 8) {
                        typename std::conditional<WIDE, unsigned long long, uint32_t>::type from[8];
                        int n[8];
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            from[k] = __shfl_sync(0xffffffffu, low, k0 + k);
                            if constexpr (WIDE) from[k] |= (unsigned long long)__shfl_sync(0xffffffffu, high, k0 + k) << 32;
                            n[k] = __shfl_sync(0xffffffffu, own.n, k0 + k);
                        }
#pragma unroll
                        for (int k = 0; k < 8; k++, slot += sh.row_stride)
                            asm volatile("{\n\t.reg .pred q;\n\tsetp.lt.s32 q, %2, %3;\n\t@q cp.async.cg.shared.global [%0], [%1], 16;\n\t}" ::"r"(slot),
                                         "l"(src + 16ull * from[k]), "r"(lane), "r"(n[k]));
                    }
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(rfull + rr.i)) : "memory");
                rr.next(TC_SLOTS);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp < TC_E0) {
        // ---------------------------------------------------------------- A operand
        const int quarter = warp & 3, grp = (warp - TC_A0) >> 2, r = 32 * quarter + lane;
        const uint32_t ta0 = tmem_a + ((uint32_t)(quarter * 32) << 16);
        Ring rr, rs;
        int turn = 0;
        TileRow next;
        if (ntile > 0) next = tile_row(ps, ps.items[tile(0)], r, ps.g_src);
        for (int i = 0; i < ntile && ok; i++) {
            const TileRow cur = next;
            // the next tile's row: its item now, its box and direction after the first piece, so
            // that neither lookup stalls the chunks
            const int4 itn = i + 1 < ntile ? ps.items[tile(i + 1)] : make_int4(0, 0, 0, 0);
            const unsigned char *ph = reinterpret_cast<const unsigned char *>(ps.PH + (size_t)cur.dir * ps.phstride + ps.phoff);
            const int base = cur.row >= 0 ? (int)(((long long)cur.row * ps.P2) & 1) : 0;
            for (int pc = 0; pc < sh.npiece && ok; pc++) {
                const int c0 = sh.piece[pc].c0, ce = sh.piece[pc].end;
                ok = mbar_wait_warp(smem_u32(rfull + rr.i), rr.par);
                if (!ok) break;
                const unsigned char *x = rows + (size_t)(rr.i * TC_M + r) * sh.row_stride + 8 * ((base + c0) & 1);
                // the coefficients and phases of a chunk are read before the one before it is stored
                float2 f[4], xp[4], xm[4], fm[FOLD ? 1 : 4];
                auto load = [&](int c) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const TcIn &w = sh.tab[4 * c + j];
                        f[j] = __ldg(reinterpret_cast<const float2 *>(ph + w.m));
                        if constexpr (!FOLD) fm[j] = __ldg(reinterpret_cast<const float2 *>(ph + w.mn));
                        xp[j] = *reinterpret_cast<const float2 *>(x + w.pos);
                        xm[j] = *reinterpret_cast<const float2 *>(x + w.neg);
                    }
                };
                int c = sh.piece[pc].beg + (turn ^ grp);
                if (c < ce) load(c);
                if (turn != grp) rs.next(nst);
                for (; c < ce; c += 2) {
                    uint32_t v[32];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float s[4];
                        if constexpr (FOLD) {  // x_m e + x_-m e*, x_m e - x_-m e*
                            const float sr = xp[j].x + xm[j].x, si = xp[j].y + xm[j].y, dr = xp[j].x - xm[j].x, di = xp[j].y - xm[j].y;
                            s[0] = sr * f[j].x - di * f[j].y, s[1] = si * f[j].x + dr * f[j].y;
                            s[2] = dr * f[j].x - si * f[j].y, s[3] = di * f[j].x + sr * f[j].y;
                        } else {
                            s[0] = xp[j].x * f[j].x - xp[j].y * f[j].y, s[1] = xp[j].x * f[j].y + xp[j].y * f[j].x;
                            s[2] = xm[j].x * fm[j].x - xm[j].y * fm[j].y, s[3] = xm[j].x * fm[j].y + xm[j].y * fm[j].x;
                        }
#pragma unroll
                        for (int k = 0; k < 4; k += 2) {
                            const float h0 = tf32_round(s[k]), h1 = tf32_round(s[k + 1]);
                            const float2 lo = f2_parts(f2_sub(f2_pack(s[k], s[k + 1]), f2_pack(h0, h1)));
                            const int o = k * TC_KC + 2 * j;
                            v[o] = __float_as_uint(h0);
                            v[o + 1] = __float_as_uint(h1);
                            v[o + TC_KC] = __float_as_uint(tf32_round(lo.x));
                            v[o + TC_KC + 1] = __float_as_uint(tf32_round(lo.y));
                        }
                    }
                    if (c + 2 < ce) load(c + 2);
                    ok = mbar_wait_warp(smem_u32(empty + rs.i), rs.par ^ 1);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    tc_st32(ta0 + (uint32_t)(rs.i * TC_ACOL), v);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(full + rs.i));
                    rs.next(nst);
                    if (c + 1 < ce) rs.next(nst);
                }
                turn ^= (ce - sh.piece[pc].beg) & 1;
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(rempty + rr.i));
                rr.next(TC_SLOTS);
                if (pc == 0) next = tile_row(ps, itn, r, ps.g_src);
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue
        const int quarter = warp & 3, eh = (warp - TC_E0) >> 2;
        const int es = sh.epi_stride;
        float2 *st = reinterpret_cast<float2 *>(epi + ((warp - TC_E0) * 32 + lane) * es);
        const uint32_t st0 = smem_u32(epi + (warp - TC_E0) * 32 * es);
        for (int i = 0; i < ntile && ok; i++) {
            const int a = set_of(i);
            const TcSub &s = range(i);
            const TileRow tr = tile_row(ps, ps.items[tile(i)], quarter * 32 + lane, ps.g_dst);
            // the row's phases, m = 0..7 and 8..15 (the tables hold 2 pmax - 1 >= 2 p - 1 of a direction)
            const float2 *ph = ps.PH + (size_t)tr.dir * ps.phstride + ps.phoff;
            float2 f0[8], f1[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                f0[j] = j < s.end ? __ldg(ph + j) : make_float2(0.f, 0.f);
                f1[j] = j + 8 < s.end ? __ldg(ph + j + 8) : make_float2(0.f, 0.f);
            }
            const uint32_t tp = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(a * sh.setw), tq = tp + (uint32_t)s.nP;
            const int p0 = s.beg * (s.beg + 1) / 2, q0 = s.beg * (s.beg - 1) / 2;
            ok = mbar_wait_warp(smem_u32(accf + a), set_par(i));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const unsigned mine = ((two ? eh ^ (i & 1) : eh) ? s.second : ~s.second) & ((1u << s.ngrp) - 1);
            unsigned left = mine;
            while (left) {
                const int g = __ffs(left) - 1, na = s.grp[g], nb = s.grp[g + 1], c0 = na * na, cnt = nb * nb - c0;
                const long long e0 = (long long)tr.row * ps.P2o + c0;
                const int odd = (int)(e0 & 1);
                left &= left - 1;
                // the warp's last group is out of its staging
                if (elect_one()) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                __syncwarp();
                for (int n = na; n < nb; n++) {
                    float2 *y = st + odd + (n * n + n - c0);
                    const uint32_t pn = tp + (uint32_t)(2 * (n * (n + 1) / 2 - p0)), qn = tq + (uint32_t)(2 * (n * (n - 1) / 2 - q0)) - 2;
                    unfold<FOLD>(pn, qn, n, f0, y, true);
                    if (n >= 8) unfold<FOLD>(pn + 16, qn + 16, n - 8, f1, y, false);
                }
                if (!left) {  // the warp's last columns are read
                    asm volatile("tcgen05.fence::before_thread_sync;");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(acce + a));
                }
                // a row's group is added by a bulk reduction of what lies on 16 bytes, single coefficients at
                // the ends by its lane
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                float2 *o = ps.dst + e0;
                const int whole = (cnt - odd) & ~1;
                const uint32_t size = tr.row >= 0 ? 8u * (uint32_t)whole : 0u;
                const unsigned alike = __match_any_sync(0xffffffffu, size << 1 | (uint32_t)odd);
                if (alike == 0xffffffffu && size) {
                    const uint32_t from = st0 + 16 * odd;
                    for (int k0 = 0; k0 < 32; k0 += 8) {
                        int row[8];
#pragma unroll
                        for (int k = 0; k < 8; k++) row[k] = __shfl_sync(0xffffffffu, tr.row, k0 + k);
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < 8; k++)
                                tc_reduce(ps.dst + (long long)row[k] * ps.P2o + (c0 + odd), from + (uint32_t)((k0 + k) * es), size);
                        }
                    }
                } else {  // (an odd p^2: every second row of destinations begins on an odd coefficient)
                    for (int k0 = 0; k0 < 32; k0 += 8) {
                        int row[8];
#pragma unroll
                        for (int k = 0; k < 8; k++) row[k] = __shfl_sync(0xffffffffu, tr.row, k0 + k);
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < 8; k++) {
                                const int odd_k = (int)(((unsigned)row[k] * (unsigned)ps.P2o + (unsigned)c0) & 1u);
                                const uint32_t size_k = 8u * (uint32_t)((cnt - odd_k) & ~1);
                                if (row[k] >= 0 && size_k)
                                    tc_reduce(ps.dst + (long long)row[k] * ps.P2o + (c0 + odd_k), st0 + (uint32_t)((k0 + k) * es) + 16 * odd_k, size_k);
                            }
                        }
                    }
                }
                if (elect_one()) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                if (tr.row >= 0) {
                    if (odd) atomicAdd(o, st[1]);
                    if (odd + whole < cnt) atomicAdd(o + cnt - 1, st[odd + cnt - 1]);
                }
            }
            if (mine == 0) {  // no group of this range is the warp's
                asm volatile("tcgen05.fence::before_thread_sync;");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(acce + a));
            }
        }
        if (elect_one()) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    if (!ok) *(volatile int *)ps.err = 1;
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// The blocks of a class's operator T, embedded as real matrices and split into TF32 hi / lo, in
// the order of the copies: class, output range, chunk, (sums hi, lo, differences hi, lo; without the
// fold outputs m hi, lo, outputs -m hi, lo of a chunk's first four inputs, then of its other four) in the core-matrix layout.  With P = x_m + x_-m, Q = x_m - x_-m of the inputs and y_+-m = S +- D of the
// outputs:  S = sum (T_m'm + T_m'-m) / 2 P (half of that for m = 0, where P = 2 x_0),
// D = sum (T_m'm - T_m'-m) / 2 Q.
// fout / fin (plans with scaled FP32 expansions, else null): per-degree factors of the
// destination and source coefficients, so that the operator maps the scaled expansions
// (multipoles d_n M_n, locals L_n / d_n of their own levels).
// Grid: (chunks, classes * output ranges).
__global__ void tc_split_kernel(const double2 *__restrict__ T, int pin, int pout, const __grid_constant__ TcShape sh,
                                const double *__restrict__ fout, const double *__restrict__ fin, float *__restrict__ B)
{
    const int c = blockIdx.x, cls = blockIdx.y / sh.nsub, P2i = pin * pin, P2o = pout * pout;
    const TcSub &s = sh.sub[blockIdx.y % sh.nsub];
    int c0 = 0;
    for (int i = 0; i < sh.npiece; i++)
        if (c >= sh.piece[i].beg && c < sh.piece[i].end) c0 = sh.piece[i].c0;
    const int parts = sh.fold ? 1 : 2, wide = s.nP + s.nQ;
    float *out = B + (size_t)cls * sh.cls_floats + s.boff + (size_t)c * parts * 2 * TC_KC * wide;
    for (int q = threadIdx.x; q < parts * wide * TC_KC; q += blockDim.x) {
        const int k = q % TC_KC, part = q / TC_KC / wide, row = q / TC_KC - part * wide, second = row >= s.nP;
        const int o = row - (second ? s.nP : 0);
        const TcIn w = sh.tab[4 * c + k / 2];
        // output o / 2 of the block: (n, m >= second), degree by degree
        int n = s.beg, j = o / 2;
        while (n < s.end && j > n - second) j -= n + 1 - second, n++;
        double v = 0.0;
        const int in = 8 * c + 4 * part + k / 2;  // (not folded) the coefficient
        if (n < s.end && (sh.fold ? w.mn != TC_PAD : in < P2i)) {
            const int m = j + second, ip = sh.fold ? c0 + w.pos / 8 : in, im = c0 + w.neg / 8;
            const double2 *row_m = T + ((size_t)cls * P2o + n * n + n + m) * P2i, *row_n = T + ((size_t)cls * P2o + n * n + n - m) * P2i;
            double2 t;
            if (sh.fold) {
                const double h = ip == im ? 0.25 : 0.5;
                t = second ? make_double2(h * (row_m[ip].x - row_m[im].x), h * (row_m[ip].y - row_m[im].y))
                           : make_double2(h * (row_m[ip].x + row_m[im].x), h * (row_m[ip].y + row_m[im].y));
            } else {
                t = (second ? row_n : row_m)[in];
            }
            v = (o & 1) == 0 ? ((k & 1) == 0 ? t.x : -t.y) : ((k & 1) == 0 ? t.y : t.x);
            if (fout) v *= fout[n] * fin[(int)sqrtf((float)ip + 0.5f)];
        }
        const float hi = tf32_round((float)v), lo = tf32_round((float)(v - (double)hi));
        float *blk = out + part * 2 * TC_KC * wide + (second ? 2 * TC_KC * s.nP : 0);
        blk[core_off(o, k, TC_KC) / 4] = hi;
        blk[(second ? s.nQ : s.nP) * TC_KC + core_off(o, k, TC_KC) / 4] = lo;
    }
}

// The list of a pass and its orders: M2L of level l, M2M of level l into its parents, L2L of
// the parents into level l.
static RcrList *dense_list(Plan *P, int l, int which, int &pin, int &pout)
{
    LevelDev &L = P->lev[l];
    if (which == PASS_M2L) {
        pin = pout = L.p;
        return &L.m2l;
    }
    if (l <= P->lmin) return nullptr;
    const int pp = P->lev[l - 1].p;
    pin = which == PASS_M2M ? L.p : pp;
    pout = which == PASS_M2M ? pp : L.p;
    return which == PASS_M2M ? &L.m2m : &L.l2l;
}

// Levels that run on sums and differences (T translations).  The fold halves the products and their rounding
// errors; at 100,000 translations and more it takes 0.45 against 0.51 ms (p = 14, 192,528 translations, one
// column) and less with more columns (17.5 against 19.5 ms for 16).  On smaller levels the
// gain is 10 to 20 us a pass, and refined
// solves, which run on bodies of that size, would stop at other steps: their stopping test sees the
// operator's error, and solutions would move by more than they differ from run to run (adjoint of a 5,120-triangle body
// at tol = 1e-8: 4e-9 against 1e-9).  The whole operator sums its products in the coefficients' order, eight at a
// time, hi hi, hi lo, lo hi, as it always has.
static bool fold_pays(int T) { return T >= 100000; }

static int build_tc_dense(Plan *P, int l, int which)
{
    int pin = 0, pout = 0;
    RcrList *Lst = dense_list(P, l, which, pin, pout);
    if (!Lst || Lst->key_beg.empty() || Lst->key_beg.back() == 0) return FMM_OK;
    TcDense &g = Lst->td;
    const char *env = getenv("FMMBEM_TENSOR_FOLD");
    const int fold = env ? atoi(env) != 0 : fold_pays(Lst->key_beg.back());
    if (!tc_shape(pin, pout, fold, g.sh)) return FMM_OK;
    const char *wide = getenv("FMMBEM_TENSOR_WIDE");  // 1: the kernel for 64 GB and more, for tests
    g.wide = wide && atoi(wide) != 0;
    g.pin = pin;
    g.pout = pout;
    const int nkeys = (int)Lst->key_beg.size() - 1, P2i = pin * pin, P2o = pout * pout;
    std::vector<int> rep;
    direction_classes(P, which, nkeys, g.cls_of_dir, rep);
    g.ncls = (int)rep.size();
    const size_t total = (size_t)g.ncls * g.sh.cls_floats;
    double2 *T = nullptr;
    int *rep_dev = nullptr;
    double *fdev = nullptr;
    auto fail = [&](cudaError_t e) {
        cudaFree(T);
        cudaFree(rep_dev);
        cudaFree(fdev);
        fmm_set_error("tensor-core pass tables: %s", cudaGetErrorString(e));
        return FMM_ERR_CUDA;
    };
    cudaError_t e = cudaMalloc(&T, sizeof(double2) * (size_t)g.ncls * P2o * P2i);
    if (e == cudaSuccess) e = cudaMalloc(&rep_dev, sizeof(int) * rep.size());
    if (e == cudaSuccess) e = upload(rep_dev, rep.data(), sizeof(int) * rep.size());
    if (e != cudaSuccess) return fail(e);
    int st = gen_dense_rcr(P, l, which, rep_dev, g.ncls, T);
    if (st) {
        cudaFree(T);
        cudaFree(rep_dev);
        return st;
    }
    // degree factors of the scaled expansions: M2L 1/d^l both sides; M2M d^{l-1} out, 1/d^l
    // in; L2L 1/d^l out, d^{l-1} in
    const double *fo = nullptr, *fi = nullptr;
    if (P->scaled) {
        const int pm = std::max(pin, pout);
        std::vector<double> h(2 * pm, 1.0);
        for (int n = 0; n < pm; n++) {
            const double inv = 1.0 / P->dsc[l][n], par = which == PASS_M2L ? 1.0 : P->dsc[l - 1][n];
            h[n] = which == PASS_M2M ? par : inv;           // out
            h[pm + n] = which == PASS_L2L ? par : inv;      // in
        }
        e = cudaMalloc(&fdev, sizeof(double) * h.size());
        if (e == cudaSuccess) e = upload(fdev, h.data(), sizeof(double) * h.size());
        if (e != cudaSuccess) return fail(e);
        fo = fdev;
        fi = fdev + pm;
    }
    e = dev_alloc(P, (void **)&g.B, sizeof(float) * total);
    if (e != cudaSuccess) return fail(e);
    g.B_bytes = sizeof(float) * total;
    tc_split_kernel<<<dim3(g.sh.nch, g.ncls * g.sh.nsub), 256, 0, P->stream>>>(T, pin, pout, g.sh, fo, fi, g.B);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(P->stream);
    cudaFree(T);
    cudaFree(rep_dev);
    cudaFree(fdev);
    T = nullptr;
    rep_dev = nullptr;
    fdev = nullptr;
    if (e != cudaSuccess) return fail(e);
    return FMM_OK;
}

__global__ void tc_permute_kernel(int n, const int *__restrict__ perm, const int *__restrict__ src,
                                  const int *__restrict__ dst, int *__restrict__ psrc, int *__restrict__ pdst)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int t = perm[i];
        psrc[i] = src[t];
        pdst[i] = dst[t];
    }
}

// The pass's translations in class order and the tiles over them, rebuilt when nrhs changes:
// where the expansions of nrhs columns are more than L2 keeps, the destination boxes are cut
// into Morton ranges first (as for the SIMT tiles); within a range, class by class, the runs
// of the class's keys one after another (each run sorted by destination).  Tiles are (class,
// first column, count) of at most 128 columns e = t nrhs + r.
static int ensure_td_items(RcrList &Lst, size_t ws, int nrhs, cudaStream_t st)
{
    TcDense &g = Lst.td;
    if (g.items_nrhs == nrhs) return FMM_OK;
    const int nkeys = (int)Lst.key_beg.size() - 1, T = Lst.key_beg.back(), nd = std::max(Lst.ndst_rank, 1);
    const size_t budget = 48u << 20;
    const long long nblk = std::min<long long>(nd, std::max<long long>(1, (long long)((ws + budget - 1) / budget)));
    std::vector<std::vector<int>> dirs(g.ncls);
    for (int d = 0; d < nkeys; d++) dirs[g.cls_of_dir[d]].push_back(d);
    std::vector<int> perm, pdir;
    std::vector<int4> items;
    perm.reserve(T);
    pdir.reserve(T);
    const int *rk = Lst.dst_rank.data();
    for (long long k = 0; k < nblk; k++) {
        const int lo = (int)(k * nd / nblk), hi = (int)((k + 1) * nd / nblk);
        for (int c = 0; c < g.ncls; c++) {
            const long long r0 = (long long)perm.size();
            for (int d : dirs[c]) {
                int a0 = Lst.key_beg[d], a1 = Lst.key_beg[d + 1];
                if (nblk > 1) {
                    a0 = (int)(std::lower_bound(rk + Lst.key_beg[d], rk + Lst.key_beg[d + 1], lo) - rk);
                    a1 = (int)(std::lower_bound(rk + Lst.key_beg[d], rk + Lst.key_beg[d + 1], hi) - rk);
                }
                for (int a = a0; a < a1; a++) {
                    perm.push_back(a);
                    pdir.push_back(d);
                }
            }
            const long long e0 = r0 * nrhs, e1 = (long long)perm.size() * nrhs;
            for (long long a = e0; a < e1; a += TC_M)
                items.push_back(make_int4(c, (int)a, (int)std::min<long long>(TC_M, e1 - a), 0));
        }
    }
    if ((int)perm.size() != T) {
        fmm_set_error("tensor-core pass: the class order covers %d of %d translations", (int)perm.size(), T);
        return FMM_ERR_ARG;
    }
    if (!g.src && T > 0) {
        FMM_CUDA_TRY(cudaMalloc(&g.src, sizeof(int) * T));
        FMM_CUDA_TRY(cudaMalloc(&g.dst, sizeof(int) * T));
        FMM_CUDA_TRY(cudaMalloc(&g.dir, sizeof(int) * T));
    }
    if (T > 0) {
        int *perm_dev = nullptr;
        FMM_CUDA_TRY(cudaMalloc(&perm_dev, sizeof(int) * T));
        cudaError_t e = upload(perm_dev, perm.data(), sizeof(int) * T);
        if (e == cudaSuccess) e = upload(g.dir, pdir.data(), sizeof(int) * T);
        if (e == cudaSuccess) {
            tc_permute_kernel<<<(T + 255) / 256, 256, 0, st>>>(T, perm_dev, Lst.src, Lst.dst, g.src, g.dst);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        cudaFree(perm_dev);
        if (e != cudaSuccess) { fmm_set_error("tensor-core pass lists: %s", cudaGetErrorString(e)); return FMM_ERR_CUDA; }
    }
    if (items.size() > g.items_cap) {
        if (g.items) cudaFree(g.items);
        g.items = nullptr;
        FMM_CUDA_TRY(cudaMalloc(&g.items, sizeof(int4) * items.size()));
        g.items_cap = items.size();
    }
    if (!items.empty()) FMM_CUDA_TRY(upload(g.items, items.data(), sizeof(int4) * items.size()));
    g.n_items = (int)items.size();
    g.items_nrhs = nrhs;
    return FMM_OK;
}

int launch_tc_dense(Plan *P, int l, int which, int nrhs, cudaStream_t st)
{
    int pin = 0, pout = 0;
    RcrList *Lst = dense_list(P, l, which, pin, pout);
    if (!Lst || Lst->key_beg.empty() || Lst->key_beg.back() == 0) return FMM_OK;
    TcDense &g = Lst->td;
    RcrPass rp;
    pass32_desc(P, l, which, nrhs, rp);
    const size_t ws = ((size_t)rp.nsrc * pin * pin + (size_t)rp.ndst * pout * pout) * sizeof(float2) * nrhs;
    int e = ensure_td_items(*Lst, ws, nrhs, st);
    if (e) return e;
    TcPass ps;
    ps.sh = g.sh;
    ps.items = g.items;
    ps.g_src = g.src;
    ps.g_dst = g.dst;
    ps.g_dir = g.dir;
    ps.PH = rp.PH;
    ps.phstride = rp.phstride;
    ps.phoff = rp.phoff;
    ps.nrhs = nrhs;
    ps.shift = 31;
    while (1ll << (ps.shift - 31) < nrhs) ps.shift++;
    ps.per = ((1ull << ps.shift) + nrhs - 1) / nrhs;
    ps.P2 = pin * pin;
    ps.P2o = pout * pout;
    ps.ntiles = g.n_items * g.sh.nsub;
    ps.B = g.B;
    ps.src = rp.src;
    ps.dst = rp.dst;
    ps.err = P->tc_err;
    const size_t sm = tc_smem_bytes(g.sh);
    const bool wide = g.wide || (size_t)rp.nsrc * nrhs * ps.P2 >= (size_t)1 << 33;
    const auto kernel = g.sh.fold ? (wide ? tc_dense_kernel<true, true> : tc_dense_kernel<true, false>)
                                  : (wide ? tc_dense_kernel<false, true> : tc_dense_kernel<false, false>);
    static size_t attr[4] = {0, 0, 0, 0};
    e = raise_smem_limit((const void *)kernel, sm, &attr[(g.sh.fold ? 1 : 0) + (wide ? 2 : 0)]);
    if (e) return e;
    // persistent: one CTA per SM (its shared memory and 512 TMEM columns take the SM)
    static int nsm = 0;
    if (!nsm) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (nsm <= 0) nsm = 152;
    }
    kernel<<<std::min(ps.ntiles, nsm), TC_THREADS, sm, st>>>(ps);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

// The bounded wait on its own: an mbarrier that expects one arrival nobody makes is waited on
// with a limit of `cycles` (out[0] = 1 if that wait gave up), then completed and waited on again
// (out[1] = 1 if that wait saw the phase complete).
__global__ void wait_probe_kernel(long long cycles, int *out)
{
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x != 0) return;
    const uint32_t b = smem_u32(&bar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b));
    out[0] = mbar_wait_limit(b, 0, cycles) ? 0 : 1;
    mbar_arrive(b);
    out[1] = mbar_wait_limit(b, 0, cycles) ? 1 : 0;
}

} // namespace fmm

extern "C" int fmm_selftest_bounded_wait(int device, int *gave_up, int *completed)
{
    using namespace fmm;
    if (!gave_up || !completed) { fmm_set_error("fmm_selftest_bounded_wait: null argument"); return FMM_ERR_ARG; }
    FMM_CUDA_TRY(cudaSetDevice(device));
    int *d = nullptr, h[2] = {0, 0};
    FMM_CUDA_TRY(cudaMalloc(&d, sizeof(h)));
    wait_probe_kernel<<<1, 32>>>(2000000LL, d);  // ~1 ms at 2 GHz
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) { fmm_set_error("fmm_selftest_bounded_wait: %s", cudaGetErrorString(e)); return FMM_ERR_CUDA; }
    *gave_up = h[0];
    *completed = h[1];
    return FMM_OK;
}

namespace fmm {

// The error flag lies in host memory that the device can write: a call reads it after its stream's
// synchronization.  (A copy from the device, with its own synchronization, was 8 us of the 59 us of a mixed
// matvec on 320 triangles.)
int ensure_tc_err(Plan *P)
{
    if (P->tc_err) return FMM_OK;
    FMM_CUDA_TRY(cudaHostAlloc((void **)&P->tc_err_host, sizeof(int), cudaHostAllocMapped));
    *P->tc_err_host = 0;
    FMM_CUDA_TRY(cudaHostGetDevicePointer((void **)&P->tc_err, P->tc_err_host, 0));
    return FMM_OK;
}

// The caller has synchronized the stream of the passes.
int check_tc_error(Plan *P)
{
    if (P->tc_err_host && *(volatile int *)P->tc_err_host) {
        fmm_set_error("tensor-core M2L: a wait on its MMA barriers gave up");
        return FMM_ERR_CUDA;
    }
    return FMM_OK;
}

// M2L levels that run dense (order p <= 16, T translations, nb boxes).  Large levels: the dense form is the faster
// one (16 columns on the 81,920-triangle sphere: p = 10, 650,304 translations 2.8 ms against 9.3 on the SIMT
// tiles; p = 14, 192,528 translations 2.8 against 6.0).  Small ones: the SIMT tiles are, by little (one column, tiles
// against dense: T = 2,504 p = 9 12 against 18 us, p = 14 18 against 24; T = 10,592 p = 9 18 against 20, p = 14 37
// against 41, p = 16 45 against 59).  The line lies where slower tiles used to lose: a level keeps
// its form and with it its rounding (TF32 halves against FP32), since a body's results
// would move by up to eleven times what two runs differ by (44 columns on a 3,380-triangle sphere, orders 18, 16).
// Dense from 2,000 translations on at p = 6..14 (at p = 11, 13, 14 from 4,000 on where they spread over more than
// the 64 boxes of level 2: thin bodies, few directions with many translations each), from 10,000 on at p = 15 and
// 9,500 at p = 16.
static bool dense_pays(int p, int T, int nb)
{
    if (p < 6) return T >= 20000;
    if (p == 11 || p == 13 || p == 14) return T >= (nb > 64 ? 4000 : 2000);
    return T >= (p <= 14 ? 2000 : p == 15 ? 10000 : 9500);
}

// Builds the dense split operators of the passes that run on the tensor cores: the M2L levels of
// order <= 16 that dense_pays() names.  FMMBEM_TENSOR_M2L (M2L) and FMMBEM_TENSOR_M2M (M2M and
// L2L, where both orders are <= 16) = 0 keep the SIMT tiles, = 1 take the tensor cores wherever
// they apply; FMMBEM_TENSOR_FOLD = 0 or 1 overrides fold_pays().  M2M and L2L stay on the SIMT tiles unless FMMBEM_TENSOR_M2M is set: their dense
// form is about ten times less accurate on the 81,920-triangle sphere (mixed against FP64
// 8.9e-7 against 7.7e-8), which costs the refined solves more iterations than it saves.
int tune_tc_dense(Plan *P)
{
    const char *env_l = getenv("FMMBEM_TENSOR_M2L"), *env_m = getenv("FMMBEM_TENSOR_M2M");
    const int mode_l = env_l ? atoi(env_l) : -1, mode_m = env_m ? atoi(env_m) : 0;
    if (mode_l == 0 && mode_m == 0) return FMM_OK;
    for (int l = P->lmin; l <= P->lmax; l++)
        for (int which = PASS_M2M; which <= PASS_L2L; which++) {
            const int mode = which == PASS_M2L ? mode_l : mode_m;
            if (mode == 0) continue;
            int pin = 0, pout = 0;
            RcrList *Lst = dense_list(P, l, which, pin, pout);
            if (!Lst || Lst->key_beg.empty() || Lst->key_beg.back() == 0) continue;
            if (mode != 1 && !dense_pays(pin, Lst->key_beg.back(), P->lev[l].nb)) continue;
            int rc = ensure_tc_err(P);
            if (rc == FMM_OK) rc = build_tc_dense(P, l, which);
            if (rc) return rc;
            Lst->td.on = Lst->td.B ? 1 : 0;  // (orders beyond the dense form have no operators)
        }
    return FMM_OK;
}

} // namespace fmm
