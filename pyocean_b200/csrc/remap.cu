// FP64 conservative vertical remap (PCM / PLM / PPM_H4) of water columns on B200.
//
// Reference: core/vertical/remap.py — remap_column :306-397, reconstruct :234-294, _average :297-303,
// _remap_columns :400-415 (one call per field there; here every field of the stack in one launch).
//
// Mapping.  Columns of up to SG_LAYERS layers are remapped with their layers side by side (remap_segments_body below) where
// that is faster (remap_form).  Deeper ones, large batches of domains and large planes of few layers: one thread owns one column and NF fields of it; consecutive threads take
// consecutive i, so each per-layer load or store of a warp is one contiguous 256-byte segment of the (k, j, i) arrays (a warp per column
// would touch 8 bytes of every 32-byte sector instead).  The column is processed in one pass (remap_core.cuh,
// remap_column_stream): a 6-cell register window builds each source cell's polynomial from its neighbours and the
// cell is integrated at once over the targets it overlaps; no column array is stored, thickness-only factors are
// computed once for all NF fields.  Columns whose target thicknesses are not all >= 0 (outside the sweep's
// domain) are marked with a sentinel in their first output layer and finished by a second launch with the
// reference's array formulation (remap_column_general); the second launch reads one value per column otherwise.
// Both paths give the reference's numbers bit for bit (-fmad=false, reference expression order).
#include <cmath>

#include "common.cuh"
#include "fct_args.cuh"
#include "exactdiv.cuh"
#include "remap_core.cuh"
#include "remap_io.cuh"

// Launch bounds of the streaming remap; POCEAN_REMAP_CTAS (resident CTAs per SM) sets its register budget.  Fitted to 5
// CTAs (20 warps) per SM: 10 % faster than ptxas's choice (128 registers with spills, 4 CTAs), 6 % faster than 6 CTAs,
// measured at 512 x 512 x 50 with two fields.
#ifndef POCEAN_REMAP_CTAS
#define POCEAN_REMAP_CTAS 5
#endif
// One field per thread (NF = 1: a lone or odd field, one-tracer domains of a batch) has fewer registers to keep:
// fitted to 7 CTAs per SM, 15 % faster than 5 (1.30 against 1.53 ms for two single-field remaps at 512 x 512 x 50)
// and than 6 or 8.
#ifndef POCEAN_REMAP1_CTAS
#define POCEAN_REMAP1_CTAS 7
#endif
#define REMAP_BOUNDS __launch_bounds__(128, NF == 1 ? POCEAN_REMAP1_CTAS : POCEAN_REMAP_CTAS)

namespace po {
namespace remap {

// One column c of NF fields m0 .. m0+NF-1: f_src (nfields, n0, plane) -> out (nfields, n1, plane).
template <int NF, typename IX>
__device__ __forceinline__ void remap_stream_body(const double* __restrict__ h_src, const double* __restrict__ f_src,
                                                  const double* __restrict__ h_tgt, const uint8_t* __restrict__ wet,
                                                  int n0, int n1, i64 plane, int m0, int scheme,
                                                  double* __restrict__ out, i64 c)
{
    if (sizeof(IX) == 4) {
        ColumnIO32<NF> io;
        io.h = h_src;
        io.t = h_tgt;
        io.c = (int)c;
        io.plane = (int)plane;
#pragma unroll
        for (int m = 0; m < NF; ++m) {
            io.u[m] = f_src + (i64)(m0 + m) * n0 * plane;
            io.o[m] = out + (i64)(m0 + m) * n1 * plane;
        }
        remap_column_io<NF>(io, wet[c] != 0, n0, n1, scheme);
    } else {
        ColumnIO<NF> io;
        io.h = h_src + c;
        io.t = h_tgt + c;
        io.plane = plane;
#pragma unroll
        for (int m = 0; m < NF; ++m) {
            io.u[m] = f_src + (i64)(m0 + m) * n0 * plane + c;
            io.o[m] = out + (i64)(m0 + m) * n1 * plane + c;
        }
        remap_column_io<NF>(io, wet[c] != 0, n0, n1, scheme);
    }
}

template <int NMAX>
__device__ __forceinline__ void remap_general_body(const double* __restrict__ h_src, const double* __restrict__ f_src,
                                                   const double* __restrict__ h_tgt, int n0, int n1, i64 plane,
                                                   int m, int scheme, double* __restrict__ out, i64 c)
{
    double* o = out + (i64)m * n1 * plane + c;
    if (__double_as_longlong(o[0]) != kRedo) return;
    ColumnIO<1> io;
    io.h = h_src + c;
    io.t = h_tgt + c;
    io.plane = plane;
    io.u[0] = f_src + (i64)m * n0 * plane + c;
    io.o[0] = o;
    rc::remap_column_general<NMAX>(io, 0, n0, n1, scheme);
}

template <int NF, typename IX>
__global__ void REMAP_BOUNDS remap_stream_kernel(const double* __restrict__ h_src,
                                                           const double* __restrict__ f_src,
                                                           const double* __restrict__ h_tgt,
                                                           const uint8_t* __restrict__ wet, int n0, int n1, i64 plane,
                                                           int field0, int scheme, double* __restrict__ out)
{
    const i64 c = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= plane) return;
    remap_stream_body<NF, IX>(h_src, f_src, h_tgt, wet, n0, n1, plane, field0 + (int)blockIdx.y * NF, scheme, out, c);
}

template <int NMAX>
__global__ void __launch_bounds__(128) remap_general_kernel(const double* __restrict__ h_src,
                                                            const double* __restrict__ f_src,
                                                            const double* __restrict__ h_tgt, int n0, int n1,
                                                            i64 plane, int scheme, double* __restrict__ out)
{
    const i64 c = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= plane) return;
    remap_general_body<NMAX>(h_src, f_src, h_tgt, n0, n1, plane, blockIdx.y, scheme, out, c);
}

// ---------------------------------------------------------------------------------------------------------------
// Remap with the layers of a column side by side, for columns of up to SG_LAYERS layers: a CTA takes SG_COLS columns of
// NF fields, the columns in shared memory, one thread per (column, layer) in turn.
//
// The sweep above keeps a column in one thread, whose chain of divisions and walks over the targets is what it waits
// for, and whose columns take different numbers of steps.  Here each stage is a loop over layers with no chain:
//   edges       running sums of the thicknesses (one thread per column, the reference's order);
//   raw edges, bounds, coefficients   the reconstruction, per interface and per cell;
//   targets     the target a cell ends in, by binary search (target edges are nondecreasing: every target thickness is
//               >= 0 here), the targets it leaves behind, and its thickest piece;
//   pieces      the integrals.  A cell that overlaps targets js .. je has je - js pieces besides its thickest, which
//               takes what they leave of its content (Hallberg), so the column's integrals number as its targets left
//               behind: integral r belongs to the cell that leaves target r, one thread each, all alike;
//   residuals   per cell, its integrals summed in the order of the targets;
//   contents    per target, its pieces summed in the order of the cells.
// Same arithmetic as the sweep, same results.  Two fields of 360 x 360 x 50 take 0.53 ms against 0.70 by the sweep, one of
// 150 x 121 x 30 38 us against 100, one of 64 x 64 x 20 13 us against 90; remap_form says where the sweep is faster.
constexpr int SG_COLS = 8;
constexpr int SG_THREADS = 256;                 // most threads of a CTA
constexpr int SG_LAYERS = 96;
constexpr uint8_t SG_NONE = 0xff;

__host__ __device__ constexpr size_t segment_smem(int nf, int n0, int n1)
{
    const int mx = n0 > n1 ? n0 : n1;
    return (size_t)SG_COLS * ((3 * n0 + n1 + 2 + nf * (4 * n0 + 1 + 2 * mx)) * sizeof(double) + 2 * n0 + n1 + 8);
}

// Threads of a CTA: the layers in rounds of at most 32 threads per column, of equal size to whole warps.
inline int segment_threads(int n0, int n1)
{
    const int mx = n0 > n1 ? n0 : n1, rounds = (mx + SG_THREADS / SG_COLS - 1) / (SG_THREADS / SG_COLS);
    const int slots = ((mx + rounds - 1) / rounds + 3) / 4 * 4;
    return SG_COLS * (slots < 8 ? 8 : slots);
}

template <int NMAX>
static __device__ __noinline__ void general_column(const double* h, const double* u, const double* t, double* o,
                                                   i64 plane, int n0, int n1, int scheme)
{
    ColumnIO<1> io;
    io.h = h;
    io.t = t;
    io.plane = plane;
    io.u[0] = u;
    io.o[0] = o;
    rc::remap_column_general<NMAX>(io, 0, n0, n1, scheme);
}

// Columns c0 .. c0 + SG_COLS - 1 of fields m0 .. m0 + NF - 1.  MARK: columns with a negative or NaN target thickness are left
// to a launch of their own, as by the sweep.
template <int NF, bool MARK>
__device__ __forceinline__ void remap_segments_body(double* sm, const double* __restrict__ h_src,
                                                    const double* __restrict__ f_src, const double* __restrict__ h_tgt,
                                                    const uint8_t* __restrict__ wet_in, int n0, int n1, i64 plane,
                                                    int m0, int scheme, double* __restrict__ out, i64 col0)
{
    __shared__ int s_active[SG_COLS], s_first[SG_COLS], s_last[SG_COLS], s_regular[SG_COLS];
    constexpr int W = SG_COLS;
    const int x = threadIdx.x % W, slot = threadIdx.x / W, SG_SLOTS = blockDim.x / W;
    const int mx = n0 > n1 ? n0 : n1;
    double* H = sm + x;                                        // row k of this column: H[k * W]
    double* A = H + n0 * W;                                    // source edges
    double* T = A + (n0 + 1) * W;                              // target edges
    double* Y = T + (n1 + 1) * W;                              // 1 / h
    double* F = Y + n0 * W;                                    // per field:
    const int fu = 0, fc0 = n0, fc1 = 2 * n0 + 1, fc2 = 3 * n0 + 1, fe0 = 4 * n0 + 1, fe1 = fe0 + mx, fn = fe1 + mx;
    uint8_t* JE = reinterpret_cast<uint8_t*>(F + NF * fn * W - x) + x;       // target a cell ends in (row i + 1)
    uint8_t* JT = JE + (n0 + 1) * W;                           // target of its thickest piece
    uint8_t* OWN = JT + n0 * W;                                // the cell that leaves a target behind
    auto at = [&](int m, int row) -> double& { return F[(m * fn + row) * W]; };

    const i64 c = col0 + x;
    const bool in = c < plane, wet = in && wet_in[c] != 0;
    const double* hs = h_src + c;
    const double* ht = h_tgt + c;
    const double* f = f_src + (i64)m0 * n0 * plane + c;
    double* o = out + (i64)m0 * n1 * plane + c;
    if (in && !wet) {                                          // remap.py:405-408
#pragma unroll
        for (int m = 0; m < NF; ++m)
            for (int k = slot; k < n1; k += SG_SLOTS)
                o[((i64)m * n1 + k) * plane] = n0 == n1 ? __ldg(f + ((i64)m * n0 + k) * plane) : nan("");
    }
    if (!__syncthreads_or(wet)) return;
    for (int k = slot; k < n0; k += SG_SLOTS) {
        H[k * W] = wet ? __ldg(hs + k * plane) : 0.0;
#pragma unroll
        for (int m = 0; m < NF; ++m) at(m, fu + k) = wet ? __ldg(f + ((i64)m * n0 + k) * plane) : 0.0;
    }
    for (int k = slot; k < n1; k += SG_SLOTS) T[(k + 1) * W] = wet ? __ldg(ht + k * plane) : 0.0;
    __syncthreads();
    // The first warp adds up the edges while the others begin the reconstruction by the scheme asked for, which needs
    // the thicknesses only (slots 4 on; the few columns that fall back to a lower scheme follow below).
    auto begin_reconstruction = [&](int sch, int first) {
        if (sch == rc::PPM_H4 && n0 >= 4) {                    // raw edge values of the interfaces, over c0
            for (int i = slot - first; i <= n0; i += SG_SLOTS - first) {
                if (i >= 2 && i <= n0 - 2) {
                    const rc::H4Weights w = rc::h4_weights(H[(i - 2) * W], H[(i - 1) * W], H[i * W], H[(i + 1) * W]);
                    const double y = shared_recip(w.den);
#pragma unroll
                    for (int m = 0; m < NF; ++m)
                        at(m, fc0 + i) = quotient(rc::h4_numerator(w, at(m, fu + i - 2), at(m, fu + i - 1),
                                                                   at(m, fu + i), at(m, fu + i + 1)), w.den, y);
                } else if (i == 0 || i == n0) {
                    const int s = i == 0 ? 1 : -1, b = i == 0 ? 0 : n0 - 1;
#pragma unroll 1
                    for (int m = 0; m < NF; ++m) {
                        double end, inner;
                        rc::end_values(rc::pmax(rc::H_NEGLECT_EDGE, H[b * W]),
                                       rc::pmax(rc::H_NEGLECT_EDGE, H[(b + s) * W]),
                                       rc::pmax(rc::H_NEGLECT_EDGE, H[(b + 2 * s) * W]),
                                       rc::pmax(rc::H_NEGLECT_EDGE, H[(b + 3 * s) * W]), at(m, fu + b),
                                       at(m, fu + b + s), at(m, fu + b + 2 * s), at(m, fu + b + 3 * s), end, inner);
                        at(m, fc0 + i) = end;
                        at(m, fc0 + i + s) = inner;
                    }
                }
            }
        } else if (sch == rc::PLM && n0 >= 3) {                // limited slopes, over e0
            for (int k = slot - first; k < n0; k += SG_SLOTS - first) {
                const bool inner = k > 0 && k < n0 - 1;
                const double r = inner ? rc::plm_ratio(H[(k - 1) * W], H[k * W], H[(k + 1) * W]) : 0.0;
#pragma unroll
                for (int m = 0; m < NF; ++m)
                    at(m, fe0 + k) = inner ? rc::plm_slope(r, at(m, fu + k - 1), at(m, fu + k), at(m, fu + k + 1)) : 0.0;
            }
        }
    };
    if (slot >= 4) {
        if (wet) begin_reconstruction(scheme, 4);
    } else if (slot == 0) {                                    // source edges, active cells
        int na = 0, fst = n0, lst = -1;
        double a = 0.0;
        A[0] = 0.0;
        for (int k = 0; k < n0; k += 4) {
            double h[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) h[q] = k + q < n0 ? H[(k + q) * W] : 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (h[q] > 0.0) {
                    ++na;
                    fst = k + q < fst ? k + q : fst;
                    lst = k + q;
                    a = a + h[q];
                }
                if (k + q < n0) A[(k + q + 1) * W] = a;
            }
        }
        s_active[x] = na;
        s_first[x] = fst;
        s_last[x] = lst;
    } else if (slot == 1) {                                    // target edges
        bool ok = true;
        double t = 0.0;
        T[0] = 0.0;
        for (int k = 1; k <= n1; k += 4) {
            double h[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) h[q] = k + q <= n1 ? T[(k + q) * W] : 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ok = ok && h[q] >= 0.0;
                t = t + h[q];
                if (k + q <= n1) T[(k + q) * W] = t;
            }
        }
        s_regular[x] = ok;
    }
    __syncthreads();
    const int na = s_active[x], fst = s_first[x], lst = s_last[x];
    const bool run = wet && s_regular[x] && na > 0;
    if (wet && !s_regular[x]) {                                // a negative or NaN target thickness
        if (slot < NF) {
            const double* fm = f + (i64)slot * n0 * plane;
            double* om = o + (i64)slot * n1 * plane;
            if (MARK) om[0] = __longlong_as_double(kRedo);
            else if (mx <= 64) general_column<64>(hs, fm, ht, om, plane, n0, n1, scheme);
            else general_column<SG_LAYERS>(hs, fm, ht, om, plane, n0, n1, scheme);
        }
    } else if (wet && !run) {                                  // no active cell (remap.py:375-381)
#pragma unroll
        for (int m = 0; m < NF; ++m) {
            double* om = o + (i64)m * n1 * plane;
            if (n0 == n1) {
                for (int k = slot; k < n1; k += SG_SLOTS) om[k * plane] = at(m, fu + k);
            } else {
                double mean = 0.0;
                for (int k = 0; k < n0; ++k) mean += at(m, fu + k) / n0;
                for (int k = slot; k < n1; k += SG_SLOTS) om[k * plane] = mean;
            }
        }
    }
    const int sch = rc::effective_scheme(na, scheme);
    const bool plm = run && sch == rc::PLM && n0 >= 3, ppm = run && sch == rc::PPM_H4 && n0 >= 4;
    if (run && sch != scheme) begin_reconstruction(sch, 0);
    if (run) {                                                 // the target each cell ends in
        for (int k = slot; k < n0; k += SG_SLOTS) {
            const double b = A[(k + 1) * W];
            int j = 0, len = n1 - 1;                           // the first of 0 .. n1-2 with t[j + 1] > b, else n1-1
            while (len > 0) {
                const int half = len >> 1;
                if (T[(j + half + 1) * W] <= b) {
                    j += half + 1;
                    len -= half + 1;
                } else {
                    len = half;
                }
            }
            JE[(k + 1) * W] = (uint8_t)j;
        }
    }
    __syncthreads();
    if (ppm) {                                                 // bounded edges of each cell
        for (int k = slot; k < n0; k += SG_SLOTS) {
            const int km = k > 0 ? k - 1 : 0, kp = k < n0 - 1 ? k + 1 : n0 - 1;
            const rc::BoundRatio br = rc::bound_ratio(H[km * W], H[k * W], H[kp * W]);
#pragma unroll
            for (int m = 0; m < NF; ++m) {
                const double um = at(m, fu + km), uc = at(m, fu + k), up = at(m, fu + kp);
                const double sl = rc::bound_slope(br, um, uc, up);
                at(m, fe0 + k) = rc::bound_edge(at(m, fc0 + k), um, uc, sl, -1.0);
                at(m, fe1 + k) = rc::bound_edge(at(m, fc0 + k + 1), up, uc, sl, 1.0);
            }
        }
    } else if (plm) {                                          // monotonized slopes, over e1
        for (int k = slot; k < n0; k += SG_SLOTS)
#pragma unroll
            for (int m = 0; m < NF; ++m)
                at(m, fe1 + k) = k == 0 || k == n0 - 1
                                     ? 0.0
                                     : rc::plm_monotonized(at(m, fu + k - 1), at(m, fu + k), at(m, fu + k + 1),
                                                           at(m, fe0 + k - 1), at(m, fe0 + k), at(m, fe0 + k + 1));
    }
    __syncthreads();
    if (run) {                                                 // coefficients; thickest piece; targets left behind
        for (int i = slot; i < n0; i += SG_SLOTS) {
            const double hi = H[i * W];
            if (!(hi > 0.0)) continue;
            Y[i * W] = shared_recip(hi);
            const bool inner = i >= 1 && i <= n0 - 2;
#pragma unroll
            for (int m = 0; m < NF; ++m) {
                const double uc = at(m, fu + i);
                double c0 = uc, c1 = 0.0, c2 = 0.0;
                if (inner && ppm) {
                    double el = at(m, fe0 + i), er = at(m, fe1 + i), er_m = at(m, fe1 + i - 1), el_p = at(m, fe0 + i + 1);
                    const double um = at(m, fu + i - 1), up = at(m, fu + i + 1);
                    rc::check_pair(er_m, el, um, uc);
                    rc::check_pair(er, el_p, uc, up);
                    rc::ppm_coef(um, uc, up, el, er, c0, c1, c2);
                } else if (inner && plm) {
                    rc::plm_coef(uc, at(m, fu + i + 1), at(m, fe1 + i), at(m, fe1 + i + 1), at(m, fe0 + i + 1), c0, c1);
                }
                at(m, fc0 + i) = c0;
                at(m, fc1 + i) = c1;
                at(m, fc2 + i) = c2;
            }
            const double a = A[i * W], b = a + hi;
            const int js = i == fst ? 0 : JE[i * W], je = JE[(i + 1) * W];
            int jt = SG_NONE;
            double thick = 0.0, tl = T[js * W];
            for (int j = js; j <= je; ++j) {
                const double th = T[(j + 1) * W];
                const double lo = tl > a ? tl : a, hi_t = j < n1 - 1 ? th : rc::pmax(th, b);
                const double L = (hi_t < b ? hi_t : b) - lo;
                if (L > thick) {
                    thick = L;
                    jt = j;
                }
                if (j < je) OWN[j * W] = (uint8_t)i;
                tl = th;
            }
            JT[i * W] = (uint8_t)jt;
        }
    }
    __syncthreads();
    const int jl = run ? JE[(lst + 1) * W] : -1;               // the target the column ends in
    if (run) {                                                 // the integrals; values of vanished targets
        for (int r = slot; r <= jl; r += SG_SLOTS) {
            const bool last = r == jl;                         // (no integral: the last vanished target's value only)
            if (last && r != n1 - 1) break;
            const int i = last ? (r > 0 ? OWN[(r - 1) * W] : fst) : OWN[r * W];
            const double a = A[i * W], hi = H[i * W], y = Y[i * W];
            if (!(__ldg(ht + r * plane) > 0.0)) {
                const double xi = quotient(T[r * W] - a, hi, y);
#pragma unroll
                for (int m = 0; m < NF; ++m)
                    o[((i64)m * n1 + r) * plane] = at(m, fc0 + i) + xi * (at(m, fc1 + i) + xi * at(m, fc2 + i));
            }
            if (last) break;
            const double b = a + hi;
            const int jt = JT[i * W], j = r < jt ? r : r + 1;  // (none: every j below it, every L <= 0)
            const double tl = T[j * W], th = T[(j + 1) * W];
            const double lo = tl > a ? tl : a, hi_t = j < n1 - 1 ? th : rc::pmax(th, b);
            const double up = hi_t < b ? hi_t : b, L = up - lo;
            if (L > 0.0) {
                const double xa = quotient(lo - a, hi, y), xb = quotient(up - a, hi, y);
#pragma unroll
                for (int m = 0; m < NF; ++m)
                    at(m, fe0 + r) = L * rc::average(at(m, fc0 + i), at(m, fc1 + i), at(m, fc2 + i), xa, xb);
            } else {
#pragma unroll
                for (int m = 0; m < NF; ++m) at(m, fe0 + r) = 0.0;
            }
        }
    }
    __syncthreads();
    if (run) {                                                 // what the integrals leave to the thickest piece
        for (int i = slot; i < n0; i += SG_SLOTS) {
            const double hi = H[i * W];
            if (!(hi > 0.0)) continue;
            const int js = i == fst ? 0 : JE[i * W], je = JE[(i + 1) * W];
#pragma unroll
            for (int m = 0; m < NF; ++m) {
                double s = 0.0;
                for (int r = js; r < je; ++r) s += at(m, fe0 + r);
                at(m, fe1 + i) = at(m, fu + i) * hi - s;
            }
        }
    }
    __syncthreads();
    if (run) {                                                 // contents
        for (int j = slot; j < n1; j += SG_SLOTS) {
            const double hgt = __ldg(ht + j * plane);
            if (hgt > 0.0) {
                double content[NF];
#pragma unroll
                for (int m = 0; m < NF; ++m) content[m] = 0.0;
                if (j <= jl) {
                    const int i1 = j < jl ? OWN[j * W] : lst;
                    for (int i = j > 0 ? OWN[(j - 1) * W] : fst; i <= i1; ++i) {
                        if (!(H[i * W] > 0.0)) continue;
                        const int jt = JT[i * W];
                        if (jt == SG_NONE) continue;
                        const int row = jt == j ? fe1 + i : fe0 + (j < jt ? j : j - 1);
#pragma unroll
                        for (int m = 0; m < NF; ++m) content[m] += at(m, row);
                    }
                }
                if (NF == 1) {
                    o[j * plane] = content[0] / hgt;
                } else {
                    const double y = shared_recip(hgt);
#pragma unroll
                    for (int m = 0; m < NF; ++m) o[((i64)m * n1 + j) * plane] = quotient(content[m], hgt, y);
                }
            } else if (!(j < jl || (j == n1 - 1 && jl == n1 - 1))) {
#pragma unroll
                for (int m = 0; m < NF; ++m) o[((i64)m * n1 + j) * plane] = at(m, fu + lst);   // never reached
            }
        }
    }
}

// CTAS (resident CTAs per SM, which sets the registers): 4; for one field of a column, whose shared memory leaves room for
// more up to about 60 layers, 5 (512 x 512 x 50: 653 us against 675 at 4; 320 x 320 x 75: 398 at 4, 440 at 5).
constexpr size_t SG_FIVE = 44 * 1024;
template <int NF, int CTAS, bool MARK>
__global__ void __launch_bounds__(SG_THREADS, CTAS) remap_segments_kernel(
    const double* __restrict__ h_src, const double* __restrict__ f_src, const double* __restrict__ h_tgt,
    const uint8_t* __restrict__ wet, int n0, int n1, i64 plane, int field0, int scheme, double* __restrict__ out)
{
    extern __shared__ double sm[];
    remap_segments_body<NF, MARK>(sm, h_src, f_src, h_tgt, wet, n0, n1, plane, field0 + (int)blockIdx.y * NF, scheme, out,
                                  (i64)blockIdx.x * SG_COLS);
}

// The same over every field of every domain of a batch (its advected stack, D.a.out -> D.rout).  A CTA goes through
// SG_BATCH_COLS columns of one domain, which its first thread finds.
constexpr int SG_BATCH_COLS = 32;
template <bool MARK>
__global__ void __launch_bounds__(SG_THREADS, 4) remap_segments_batched(const BatchDomain* __restrict__ doms,
                                                                       const int* __restrict__ off, int ndom)
{
    extern __shared__ double sm[];
    __shared__ int domain;
    if (threadIdx.x == 0) domain = find_domain(off, ndom, blockIdx.x);
    __syncthreads();
    const BatchDomain& D = doms[domain];
    const int n = D.a.s.n;
    const i64 plane = (i64)D.a.s.ny * D.a.s.nx;
    const int groups = (int)((plane + SG_BATCH_COLS - 1) / SG_BATCH_COLS), local = blockIdx.x - __ldg(off + domain);
    const int m = local / groups;
    i64 c = (i64)(local - m * groups) * SG_BATCH_COLS;
    for (const i64 end = c + SG_BATCH_COLS; c < end && c < plane; c += SG_COLS) {
        remap_segments_body<1, MARK>(sm, D.h_src, D.a.out, D.h_tgt, D.wet, n, n, plane, m, D.remap_scheme, D.rout, c);
        __syncthreads();
    }
}

// Batched remap of every domain's advected stack (D.a.out -> D.rout).  Mode: NF = 2 over field pairs (group g =
// fields 2g, 2g+1), or NF = 1 over single fields starting at `first` (the odd field left by the pairs, or all).
template <int NF>
__global__ void REMAP_BOUNDS remap_stream_batched(const BatchDomain* __restrict__ doms,
                                                            const int* __restrict__ off, int ndom, int odd_only)
{
    const int d = find_domain(off, ndom, blockIdx.x);
    const BatchDomain& D = doms[d];
    const Shape s = D.a.s;
    const i64 plane = (i64)s.ny * s.nx;
    const int cblocks = (int)((plane + 127) / 128);
    const int local = blockIdx.x - __ldg(off + d);
    const int g = local / cblocks;
    const i64 c = (i64)(local - g * cblocks) * 128 + threadIdx.x;
    if (c >= plane) return;
    const int m0 = NF == 2 ? 2 * g : (odd_only ? s.nt - 1 : g);
    // the batch bounds every field by 2^31 entries
    remap_stream_body<NF, int>(D.h_src, D.a.out, D.h_tgt, D.wet, s.n, s.n, plane, m0, D.remap_scheme, D.rout, c);
}

template <int NMAX>
__global__ void __launch_bounds__(128) remap_general_batched(const BatchDomain* __restrict__ doms,
                                                             const int* __restrict__ off, int ndom)
{
    const int d = find_domain(off, ndom, blockIdx.x);
    const BatchDomain& D = doms[d];
    const Shape s = D.a.s;
    const i64 plane = (i64)s.ny * s.nx;
    const int cblocks = (int)((plane + blockDim.x - 1) / blockDim.x);      // the columns of a CTA of `off`
    const int local = blockIdx.x - __ldg(off + d);
    const int m = local / cblocks;
    const i64 c = (i64)(local - m * cblocks) * blockDim.x + threadIdx.x;
    if (c >= plane) return;
    remap_general_body<NMAX>(D.h_src, D.a.out, D.h_tgt, s.n, s.n, plane, m, D.remap_scheme, D.rout, c);
}

// reconstruct (remap.py:234-294) of ncols columns of n cells: h, u (n, ncols), coef (n, ncols, 3); the scheme as
// given (PCM below 3 cells, PLM below 4 for PPM_H4, as there).
template <int NMAX>
__global__ void __launch_bounds__(128) reconstruct_kernel(const double* __restrict__ h, const double* __restrict__ u,
                                                          int n, i64 ncols, int scheme, double* __restrict__ coef)
{
    const i64 c = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncols) return;
    double hh[NMAX], uu[NMAX], c0[NMAX], c1[NMAX], c2[NMAX], e0[NMAX], e1[NMAX];
    for (int k = 0; k < n; ++k) {
        hh[k] = __ldg(h + (k * ncols + c));
        uu[k] = __ldg(u + (k * ncols + c));
    }
    rc::reconstruct_column(hh, uu, n, scheme, c0, c1, c2, e0, e1);
    for (int k = 0; k < n; ++k) {
        double* o = coef + 3 * (k * ncols + c);
        o[0] = c0[k];
        o[1] = c1[k];
        o[2] = c2[k];
    }
}

}  // namespace remap

// The most dynamic shared memory a side-by-side launch takes: columns of SG_LAYERS layers of one field; field pairs up to
// three CTAs an SM.
constexpr size_t SG_SMEM1 = remap::segment_smem(1, remap::SG_LAYERS, remap::SG_LAYERS), SG_SMEM2 = 72 * 1024;

// Whether the columns with a negative or NaN target thickness of `columns` (those of all fields) of up to n layers take a
// launch of their own.  Else a thread of their CTA does them while the others wait.  The launch costs 3 us, at this line 4 %
// of the remap; without it, 360 x 360 x 50 columns of two fields, one in a hundred of them such, take 2.24 ms instead of
// 0.96, all of them 15.1 instead of 1.5 (by the sweep 1.30 and 1.40), and 64 x 64 x 50 of one field 0.31 and 0.28 ms (by the
// sweep 0.49 and 0.29).
static bool irregular_launch(long long columns, int n) { return columns * n > 1000000; }

// Whether the sweep remaps `columns` columns faster than they are remapped side by side.  It holds a wave of columns at a
// time; a wave costs it the same whatever is in it but for the last, which costs between half and a whole one, while side by
// side the time is proportional to the columns, `ratio` times the sweep's for whole waves.
static bool sweep_pays(long long columns, long long wave, double ratio)
{
    const long long full = columns / wave;
    const double rest = (double)(columns - full * wave) / wave;
    return ratio * ((double)full + rest) > full + (rest > 0.0 ? 0.5 + 0.5 * rest : 0.0);
}

// The ratio falls with the layers n, since side by side each column has its barriers whatever its depth.  Side by side / by
// the sweep, measured for whole waves (1024 x 1024, 724 x 724 and 512 x 512 columns, PPM_H4, us):
//   field pairs     2 layers 380/136, 4 677/335, 8 880/661, 12 1099/976, 20 1785/1654, 30 685/703, 50 1096/1177;
//   single fields   2 layers 290/83, 4 419/196, 8 577/390, 12 734/593, 20 1175/1005, 30 480/435, 50 753/734, 96 1562/1422.
// Pairs above 70 layers, which go side by side as two single fields: 75 layers of 512 x 512 2274/1778, of 300 x 310 822/660,
// of 240 x 240 517/558, 309 x 309 (just over a wave) 835/974.
static double side_ratio(int nf, double n)
{
    if (nf == 2) return 0.87 + 3.6 / n;
    return n <= 64 ? 0.95 + 3.0 / n : 1.06;
}
constexpr double SIDE_RATIO_DEEP_PAIRS = 1.28;
constexpr long long SWEEP_WAVE1 = 148 * POCEAN_REMAP1_CTAS * 128, SWEEP_WAVE2 = 148 * POCEAN_REMAP_CTAS * 128;

// Whether a batch of `columns` column-fields of up to nmax layers is remapped with the layers of a column side by side:
// batches that the one-thread-per-column sweep leaves the chip idle for, unless they are shallow.  Larger ones
// take the sweep: their domains' depths differ, and the shared memory of the deepest one's columns leaves too few CTAs
// (24 domains of one tracer: a step's remap 1.98 ms by the sweep, 2.4 ms side by side; 8 domains of 48..160 cells: the
// two steps 1.71 ms by the sweep, 1.47 ms side by side).
bool remap_batch_segments(long long columns, int nmax)
{
    return nmax <= remap::SG_LAYERS && columns <= 150000 &&
           !(nmax <= 16 && sweep_pays(columns, SWEEP_WAVE1, side_ratio(1, nmax)));
}

// The launches of a remap: of field pairs and of single fields, each side by side or by the sweep, and the irregular
// columns'.  Side by side, two fields of a column share the work on its thicknesses while three CTAs fit an SM.
struct RemapForm {
    int pairs, singles;
    bool side_pairs, side_singles, general;
    int launches() const { return (pairs > 0) + (singles > 0) + general; }
};

static RemapForm remap_form(int n0, int n1, i64 plane, int nfields)
{
    const int mx = n0 > n1 ? n0 : n1;
    const double n = 0.5 * (n0 + n1);
    RemapForm f{nfields / 2, nfields % 2, false, false, true};
    if (mx > remap::SG_LAYERS) return f;
    const bool fit2 = remap::segment_smem(2, n0, n1) <= SG_SMEM2;
    f.side_pairs = f.pairs && !sweep_pays(plane * f.pairs, SWEEP_WAVE2, fit2 ? side_ratio(2, n) : SIDE_RATIO_DEEP_PAIRS);
    if (f.side_pairs && !fit2) {
        f.pairs = 0;
        f.singles = nfields;
        f.side_singles = true;
    } else {
        f.side_singles = f.singles && !sweep_pays(plane, SWEEP_WAVE1, side_ratio(1, n));
    }
    f.general = (f.pairs && !f.side_pairs) || (f.singles && !f.side_singles) ||
                irregular_launch((long long)plane * nfields, mx);
    return f;
}

// Columns of a batched remap CTA.
int remap_batched_columns(bool segments) { return segments ? remap::SG_BATCH_COLS : 128; }

// A kernel's static and dynamic shared memory together above the default limit (48 KB) has to be asked for.  The limit
// belongs to the kernel, not to the launch: every call asks for the same, so that no other thread's call lowers it between
// a call's request and its launch.
static cudaError_t allow_smem(const void* kernel, size_t most)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

// Kernel launches of remap_batched_launch for domains of these shapes (nt, nz, ny, nx).
int remap_batch_launches(const int* shapes, int ndom, int nf_mode)
{
    long long columns = 0, padded = 0;
    int nmax = 1;
    bool pairs = false, odd = false;
    for (int d = 0; d < ndom; ++d) {
        const int nt = shapes[4 * d];
        const long long plane = (long long)shapes[4 * d + 2] * shapes[4 * d + 3];
        columns += plane * nt;
        padded += (plane + remap::SG_BATCH_COLS - 1) / remap::SG_BATCH_COLS * remap::SG_BATCH_COLS * nt;
        nmax = shapes[4 * d + 1] > nmax ? shapes[4 * d + 1] : nmax;
        pairs = pairs || nt >= 2;
        odd = odd || nt % 2 == 1;
    }
    if (remap_batch_segments(columns, nmax)) return 1 + irregular_launch(padded, nmax);
    return (nf_mode == 2 ? (int)pairs + (int)odd : 1) + 1;
}

// nf_mode 2: field pairs (+ the odd field); nf_mode 1: every field on its own.  nmax: the batch's deepest column.
cudaError_t remap_batched_launch(const BatchDomain* doms, const int* off_dev, const int* off_host, int ndom, int nf_mode,
                                 int nmax, bool segments, cudaStream_t st)
{
    auto total = [&](int pass) { return (unsigned)off_host[pass * (ndom + 1) + ndom]; };
    auto offs = [&](int pass) { return off_dev + pass * (ndom + 1); };
    if (segments) {
        const size_t smem = remap::segment_smem(1, nmax, nmax);
        const bool mark = irregular_launch((long long)total(BP_RALL) * remap::SG_BATCH_COLS, nmax);
        const auto kernel = mark ? remap::remap_segments_batched<true> : remap::remap_segments_batched<false>;
        const cudaError_t e = allow_smem((const void*)kernel, SG_SMEM1);
        if (e != cudaSuccess) return e;
        kernel<<<total(BP_RALL), remap::SG_THREADS, smem, st>>>(doms, offs(BP_RALL), ndom);
        if (mark)
            remap::remap_general_batched<remap::SG_LAYERS>
                <<<total(BP_RALL), remap::SG_BATCH_COLS, 0, st>>>(doms, offs(BP_RALL), ndom);
        return cudaSuccess;
    }
    if (nf_mode == 2) {
        if (total(BP_RPAIR)) remap::remap_stream_batched<2><<<total(BP_RPAIR), 128, 0, st>>>(doms, offs(BP_RPAIR), ndom, 0);
        if (total(BP_RREM)) remap::remap_stream_batched<1><<<total(BP_RREM), 128, 0, st>>>(doms, offs(BP_RREM), ndom, 1);
    } else {
        remap::remap_stream_batched<1><<<total(BP_RALL), 128, 0, st>>>(doms, offs(BP_RALL), ndom, 0);
    }
    if (nmax <= 64) remap::remap_general_batched<64><<<total(BP_RALL), 128, 0, st>>>(doms, offs(BP_RALL), ndom);
    else if (nmax <= 128) remap::remap_general_batched<128><<<total(BP_RALL), 128, 0, st>>>(doms, offs(BP_RALL), ndom);
    else remap::remap_general_batched<256><<<total(BP_RALL), 128, 0, st>>>(doms, offs(BP_RALL), ndom);
    return cudaSuccess;
}

void remap_general_launch(const double* h_src, const double* f_src, const double* h_tgt, int n0, int n1, i64 plane,
                          int nfields, int scheme, double* out, cudaStream_t st)
{
    const dim3 g2((unsigned)((plane + 127) / 128), (unsigned)nfields);
    const int nm = n0 > n1 ? n0 : n1;
    if (nm <= 128)
        remap::remap_general_kernel<128><<<g2, 128, 0, st>>>(h_src, f_src, h_tgt, n0, n1, plane, scheme, out);
    else
        remap::remap_general_kernel<256><<<g2, 128, 0, st>>>(h_src, f_src, h_tgt, n0, n1, plane, scheme, out);
}

}  // namespace po

using namespace po;

extern "C" int pocean_remap_columns_f64(const double* h_src, const double* f_src, const double* h_tgt,
                                        const uint8_t* wet, int n0, int n1, int ny, int nx, int nfields, int scheme,
                                        double* out, void* stream)
{
    const char* fn = "pocean_remap_columns_f64";
    if (n0 < 1 || n1 < 1 || ny < 1 || nx < 1 || nfields < 1)
        return pocean_fail(POCEAN_EINVAL, "%s: sizes must be >= 1 (n0=%d n1=%d ny=%d nx=%d nfields=%d)", fn, n0, n1,
                           ny, nx, nfields);
    if (n0 > 256 || n1 > 256)
        return pocean_fail(POCEAN_EINVAL, "%s: at most 256 layers per column (n0=%d n1=%d)", fn, n0, n1);
    if (nfields > 65535) return pocean_fail(POCEAN_EINVAL, "%s: nfields=%d exceeds 65535", fn, nfields);
    if (scheme < POCEAN_PCM || scheme > POCEAN_PPM_H4)
        return pocean_fail(POCEAN_EINVAL, "%s: unknown scheme %d", fn, scheme);
    if (!h_src || !f_src || !h_tgt || !wet || !out) return pocean_fail(POCEAN_EINVAL, "%s: null pointer", fn);
    int rc = pocean_check_device();
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const i64 plane = (i64)ny * nx;
    const RemapForm form = remap_form(n0, n1, plane, nfields);
    const int pairs = form.pairs, singles = form.singles, threads = remap::segment_threads(n0, n1);
    const unsigned side = (unsigned)((plane + remap::SG_COLS - 1) / remap::SG_COLS), gx = (unsigned)((plane + 127) / 128);
    // 32-bit offsets within a field when every field (n0 or n1 layers of the plane) holds fewer than 2^31 entries
    const bool small = (i64)(n0 > n1 ? n0 : n1) * plane < (1ll << 31);
    if (pairs > 0 && form.side_pairs) {
        const auto kernel = form.general ? remap::remap_segments_kernel<2, 4, true> : remap::remap_segments_kernel<2, 4, false>;
        const cudaError_t e = allow_smem((const void*)kernel, SG_SMEM2);
        if (e != cudaSuccess) return pocean_fail(POCEAN_ECUDA, "%s: %s", fn, cudaGetErrorString(e));
        kernel<<<dim3(side, (unsigned)pairs), threads, remap::segment_smem(2, n0, n1), st>>>(
            h_src, f_src, h_tgt, wet, n0, n1, plane, 0, scheme, out);
    } else if (pairs > 0) {
        const auto kernel = small ? remap::remap_stream_kernel<2, int> : remap::remap_stream_kernel<2, i64>;
        kernel<<<dim3(gx, (unsigned)pairs), 128, 0, st>>>(h_src, f_src, h_tgt, wet, n0, n1, plane, 0, scheme, out);
    }
    if (singles > 0 && form.side_singles) {
        const size_t s1 = remap::segment_smem(1, n0, n1);
        const bool five = s1 <= remap::SG_FIVE;
        const auto kernel = form.general
                                ? (five ? remap::remap_segments_kernel<1, 5, true> : remap::remap_segments_kernel<1, 4, true>)
                                : (five ? remap::remap_segments_kernel<1, 5, false> : remap::remap_segments_kernel<1, 4, false>);
        const cudaError_t e = allow_smem((const void*)kernel, SG_SMEM1);
        if (e != cudaSuccess) return pocean_fail(POCEAN_ECUDA, "%s: %s", fn, cudaGetErrorString(e));
        kernel<<<dim3(side, (unsigned)singles), threads, s1, st>>>(h_src, f_src, h_tgt, wet, n0, n1, plane, 2 * pairs, scheme,
                                                                   out);
    } else if (singles > 0) {
        const auto kernel = small ? remap::remap_stream_kernel<1, int> : remap::remap_stream_kernel<1, i64>;
        kernel<<<dim3(gx, (unsigned)singles), 128, 0, st>>>(h_src, f_src, h_tgt, wet, n0, n1, plane, 2 * pairs, scheme, out);
    }
    if (form.general) remap_general_launch(h_src, f_src, h_tgt, n0, n1, plane, nfields, scheme, out, st);
    return pocean_check_launch(fn);
}

extern "C" int pocean_remap_launches(int n0, int n1, int ny, int nx, int nfields)
{
    if (n0 < 1 || n1 < 1 || ny < 1 || nx < 1 || nfields < 1) return 0;
    return remap_form(n0, n1, (i64)ny * nx, nfields).launches();
}

extern "C" int pocean_reconstruct_f64(const double* h, const double* u, int n, long long ncols, int scheme,
                                      double* coef, void* stream)
{
    const char* fn = "pocean_reconstruct_f64";
    if (n < 1 || ncols < 1)
        return pocean_fail(POCEAN_EINVAL, "%s: sizes must be >= 1 (n=%d ncols=%lld)", fn, n, ncols);
    if (n > 256) return pocean_fail(POCEAN_EINVAL, "%s: at most 256 cells per column (n=%d)", fn, n);
    if (ncols > (1ll << 40)) return pocean_fail(POCEAN_EINVAL, "%s: ncols=%lld too large", fn, ncols);
    if (scheme < POCEAN_PCM || scheme > POCEAN_PPM_H4)
        return pocean_fail(POCEAN_EINVAL, "%s: unknown scheme %d", fn, scheme);
    if (!h || !u || !coef) return pocean_fail(POCEAN_EINVAL, "%s: null pointer", fn);
    int rc = pocean_check_device();
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned g = (unsigned)((ncols + 127) / 128);
    if (n <= 64) remap::reconstruct_kernel<64><<<g, 128, 0, st>>>(h, u, n, (i64)ncols, scheme, coef);
    else if (n <= 128) remap::reconstruct_kernel<128><<<g, 128, 0, st>>>(h, u, n, (i64)ncols, scheme, coef);
    else remap::reconstruct_kernel<256><<<g, 128, 0, st>>>(h, u, n, (i64)ncols, scheme, coef);
    return pocean_check_launch(fn);
}
