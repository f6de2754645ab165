// The three WENO passes of the FCT step split into a face pass and a cell pass each (included by advect.cu).
//
// Face pass of stage s: one thread per cell (k, j, i), every tracer in turn, computes the west x-face and the south y-face
// of its cell (the last column / row also the east / north domain face) straight from global memory (the five upwind
// cells of a face, loaded in upwind order, overlap between neighbouring threads and are served by L1), with no shared
// memory and no barrier, so the pass runs
// at high occupancy and the two independent WENO5 chains of a thread overlap.  Cell pass of stage s: the stage
// update from the stored faces.  Faces per stage are stored once:
//   stage 1: S <- F0;  stage 2: T <- F1;  stage 3: S <- A = ((F0 + F1)/6 + 2 F2/3) - F_L,
// with (F0 + F1)/6 and 2 F2/3 formed by the same exact divisions as the reference.  Stage 3 has no cell pass: its
// face pass also forms the donor-cell solution c_L of its cell, recomputing the cheap donor fluxes F_L of the
// cell's east and north faces, so F_L is never stored.  The arithmetic of every face and
// update is the reference's (weno.cuh; sigma_baroclinic.py:265-321, 452-511), so results equal the reference's bit
// for bit.  Which reconstruction a face takes comes from the class pass; CTAs
// whose stencils stay inside the domain run without the edge and periodic cases (INNER).
#pragma once

namespace po {

// The stencil classes of the domain's faces, one byte per cell, in the buffer that R+ takes after the face passes.
__device__ __forceinline__ uint8_t* fct_classes(const StepArgs& a) { return reinterpret_cast<uint8_t*>(a.q1); }

// The stage's input field (stages 1: C; 2: c1; 3: c2).
template <int STAGE>
__device__ __forceinline__ const double* stage_field(const StepArgs& a)
{
    return STAGE == 1 ? a.C : (STAGE == 2 ? a.c1 : a.c2);
}

// Which reconstruction a face takes (sigma_baroclinic.py:204-233 `_wval`): 2 WENO5 (all five cells of its upwind
// stencil are valid), 1 WENO3 (the middle three are), 0 the upwind cell; valid = inside the domain (or wrapped) and ok.
// Two bits per direction of a face: bits 0-1 / 2-3 the west x-face of a cell for Q >= 0 / Q < 0, bits 4-5 / 6-7 its
// south y-face, bits 8-9 / 10-11 (the unlimited step's uint16 classes) its bottom z-face.
__device__ __forceinline__ unsigned stencil_class(bool a, bool b, bool c, bool d, bool e)
{
    return (b && c && d) ? (a && e ? 2u : 1u) : 0u;
}

// The classes of a face between cells f-1 and f from the validity of cells f-3 .. f+2.
__device__ __forceinline__ unsigned face_class(const bool* v)
{
    return stencil_class(v[0], v[1], v[2], v[3], v[4]) | stencil_class(v[5], v[4], v[3], v[2], v[1]) << 2;
}

__device__ __forceinline__ unsigned line_class(const uint8_t* __restrict__ ok, int st, int n, bool per, int f)
{
    bool v[6];
    if (f >= 3 && f + 2 < n) {
#pragma unroll
        for (int m = 0; m < 6; ++m) v[m] = __ldg(ok + (f - 3 + m) * st) != 0;
        return face_class(v);
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        int g = f - 3 + m;
        bool in = true;
        if (per) g = wrap(g, n); else in = g >= 0 && g < n;
        v[m] = in && __ldg(ok + (in ? g : 0) * st) != 0;
    }
    return face_class(v);
}

// Validity of four neighbouring cells as the bytes of a word (0xff valid, 0 not): cells i .. i+3 of a row of n cells,
// 0 outside the row (a periodic row wraps); i is a multiple of four.  `words`: rows start on words.  Other rows are read
// as the two words around the cells where both lie within the mask (lo .. hi), the cells beyond the row cleared; what is
// left (the wrapped ends, the mask's own ends) goes by bytes.
__device__ __forceinline__ unsigned ok4(const uint8_t* __restrict__ row, int n, bool per, int i, bool words,
                                        const uint8_t* lo, const uint8_t* hi)
{
    if (!per && (i < 0 || i >= n)) return 0u;
    unsigned w = 0;
    const uint8_t* p = row + i;
    const unsigned off = (unsigned)reinterpret_cast<uintptr_t>(p) & 3u;
    const uint8_t* q = p - off;
    if (words && i >= 0 && i + 4 <= n) {
        w = __ldg(reinterpret_cast<const unsigned*>(p));
    } else if (i >= 0 && (i + 4 <= n || !per) && q >= lo && q + 8 <= hi) {
        const unsigned* q4 = reinterpret_cast<const unsigned*>(q);
        w = __funnelshift_r(__ldg(q4), __ldg(q4 + 1), 8 * off);
        if (i + 4 > n) w &= (1u << (8 * (n - i))) - 1u;
    } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            int g = i + m;
            if (per) g = wrap(g, n);
            if (g >= 0 && g < n) w |= (unsigned)__ldg(row + g) << (8 * m);
        }
    }
    return __vcmpne4(w, 0u);
}

// The classes (see face_class) of four faces from the validity words of the cells f-3 .. f+2 of each.
__device__ __forceinline__ unsigned class4(const unsigned* v)
{
    const unsigned m = v[1] & v[2] & v[3], q = v[4] & v[3] & v[2];            // the middle three, Q >= 0 / Q < 0
    const unsigned a = m & v[0] & v[4], b = q & v[5] & v[1];                  // all five
    return (a & 0x02020202u) | (m & ~a & 0x01010101u) | (b & 0x08080808u) | (q & ~b & 0x04040404u);
}

// Class pass: works out the classes of every cell's two faces once for the three face passes and every tracer (they
// depend on ok alone), one byte per cell; the face passes used to load and test five ok bytes per stencil.  A thread
// takes four neighbouring cells, their validity in the bytes of a word; where nx is a multiple of four and ok starts
// on a word, rows are read and written by words.
// Bounded by instruction issue (71 %): 39 us at 512 x 512 x 50, where the face passes it serves went from 2.11 to 1.47 ms
// (with their shorter divisions and tracer loop).  64 uneven boxes: 1.06 ms with rows that start off a word read by bytes,
// 0.84 so; two or four rows a thread were within the noise of one.
__device__ __forceinline__ void class_body(const StepArgs& a, int k, int i, int j)
{
    const Shape s = a.s;
    const Flags fl(a.flags);
    if (i >= s.nx || j >= s.ny) return;
    const int pl = s.ny * s.nx;
    const uint8_t* ok = a.ok + plane_at(k, pl);
    const bool words = (s.nx & 3) == 0 && (reinterpret_cast<uintptr_t>(ok) & 3) == 0;
    const uint8_t* row = ok + j * s.nx;
    const uint8_t *lo = a.ok, *hi = a.ok + plane_at(s.n, pl);
    const unsigned w0 = ok4(row, s.nx, fl.per_x, i - 4, words, lo, hi), w1 = ok4(row, s.nx, fl.per_x, i, words, lo, hi),
                   w2 = ok4(row, s.nx, fl.per_x, i + 4, words, lo, hi);
    unsigned v[6];
    v[0] = __funnelshift_r(w0, w1, 8);                                        // cells i-3 .. i
    v[1] = __funnelshift_r(w0, w1, 16);
    v[2] = __funnelshift_r(w0, w1, 24);
    v[3] = w1;
    v[4] = __funnelshift_r(w1, w2, 8);
    v[5] = __funnelshift_r(w1, w2, 16);
    unsigned c = class4(v);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        int g = j - 3 + m;
        if (fl.per_y) g = wrap(g, s.ny);
        v[m] = m == 3 ? w1 : (g >= 0 && g < s.ny ? ok4(ok + g * s.nx, s.nx, false, i, words, lo, hi) : 0u);
    }
    c |= class4(v) << 4;
    uint8_t* out = fct_classes(a) + plane_at(k, pl) + (j * s.nx + i);
    if (words) {
        *reinterpret_cast<unsigned*>(out) = c;
        return;
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
        if (i + m < s.nx) out[m] = (uint8_t)(c >> (8 * m));
}

// Face value of an interior face from its class (the face lies between cells f-1 and f of a line of n cells `st`
// apart; o: the offset of cell f).  The cells are loaded in upwind order v1..v5, as the reference passes them to
// _wval: cells f-3 .. f+1 for Q >= 0, f+2 .. f-2 for Q < 0.  A class only counts cells inside the domain, so only a
// periodic line's stencil needs to wrap, at its ends (INNER: the face is at least three cells from them).
template <bool ZV, bool MIX, bool INNER>
__device__ __forceinline__ double face_value(const double* __restrict__ c, int o, int st, int n, bool per, int f,
                                             bool pos, unsigned cls)
{
    const int d = pos ? st : -st;
    int o3 = pos ? o - st : o, o1 = o3 - 2 * d, o2 = o3 - d, o4 = o3 + d, o5 = o4 + d;
    if (!INNER && per && (f < 3 || f + 2 >= n)) {
        const int ln = n * st, l0 = o - f * st;           // offsets of this line run from l0 to l0 + ln
        auto in = [&](int x) { x -= l0; return l0 + (((unsigned)x < (unsigned)ln) ? x : wrap(x, ln)); };
        o1 = in(o1); o2 = in(o2); o3 = in(o3); o4 = in(o4); o5 = in(o5);
    }
    if (cls == 2u) return weno5_any<ZV, MIX>(__ldg(c + o1), __ldg(c + o2), __ldg(c + o3), __ldg(c + o4), __ldg(c + o5));
    const double v3 = __ldg(c + o3);
    if (cls == 0u) return v3;
    return weno3_any<MIX>(__ldg(c + o2), v3, __ldg(c + o4));
}

// The stage's quantity of one face (S, T: the face arrays of this plane), read back for stages 3 and 4 here, after
// the face computation: holding them across the WENO chains cost registers, and at the face passes' 32-register
// budget the spills outweighed the overlap (2.2 % of advect_fct at 512 x 512 x 50).  The thirds and sixths
// of zeros (land and closed faces, still tracers) take their short form: through two divisions each they cost stage 3
// half as many instructions again.
template <int STAGE>
__device__ __forceinline__ double staged_flux(const double* S, const double* T, int fo, double F, double FL)
{
    if (STAGE <= 2) return F;
    const double H = div6_exact(S[fo] + T[fo]) + div3_exact(2.0 * F);
    return STAGE == 3 ? H - FL : H;               // 4, the unlimited step: the RK3 flux F_H = (F0 + F1)/6 + 2 F2/3
}

// Flux through a domain-edge face (west / south: SIDE 1, inflow for q > 0; east / north: -1): upstream on an open
// edge with the exterior on inflow, 0 on a closed one (sigma_baroclinic.py:283-297); c, e: the edge cell's value and
// its exterior's.
template <int SIDE>
__device__ __forceinline__ double edge_flux(bool open, double q, double c, double e)
{
    return open ? q * ((SIDE > 0 ? q > 0.0 : q < 0.0) ? e : c) : 0.0;
}

// Face pass of stage STAGE for cell (k, j, i) of tracers t0 .. t1-1.  Flux through the cell's west x-face and south
// y-face: WENO5 on interior faces, 0 where Q = 0; stage 3 also the donor flux F_L of C (sigma_baroclinic.py:277-297,
// 486-494).  The last column / row adds the east / north domain face; on a periodic axis that face is face 0, which
// the first column / row stores twice.  INNER: the cell is at least three cells from every domain edge, where none of
// that arises.
template <int STAGE, bool ZV, bool MIX, bool INNER>
__device__ __forceinline__ void faces_cell(const StepArgs& a, int t0, int t1, int k, int i, int j)
{
    const Shape s = a.s;
    const Flags fl(a.flags);
    const int pl = s.ny * s.nx, xpl = s.ny * (s.nx + 1), ypl = (s.ny + 1) * s.nx;
    const int o = j * s.nx + i, ox = o + j;
    const double* __restrict__ qx = a.Qx + plane_at(k, xpl);
    const double* __restrict__ qy = a.Qy + plane_at(k, ypl);
    const unsigned cls = __ldg(fct_classes(a) + plane_at(k, pl) + o);
    const double qw = __ldg(qx + ox), qs = __ldg(qy + o);
    const bool per_x = !INNER && fl.per_x, per_y = !INNER && fl.per_y;
    const bool last_x = !INNER && i == s.nx - 1, last_y = !INNER && j == s.ny - 1;
#pragma unroll 1
    for (int t = t0; t < t1; ++t) {
        const int p = t * s.n + k;
        const i64 pc = plane_at(p, pl), pu = plane_at(p, xpl), pv = plane_at(p, ypl);
        const double* __restrict__ c = stage_field<STAGE>(a) + pc;
        const double* __restrict__ c0 = a.C + pc;                    // the donor flux of stage 3
        double* sx = (STAGE == 2 ? a.Tx : a.Sx) + pu;
        double* sy = (STAGE == 2 ? a.Ty : a.Sy) + pv;
        const double* tx = a.Tx + pu;
        const double* ty = a.Ty + pv;
        if (STAGE == 3) {                              // read after the WENO chains
            prefetch(sx + ox);
            prefetch(tx + ox);
            prefetch(sy + o);
            prefetch(ty + o);
            prefetch(c0 + o);
            if (t == t0) {
                prefetch(a.V0 + plane_at(k, pl) + o);
                prefetch(a.V1 + plane_at(k, pl) + o);
            }
        }
        double fw = 0.0, lw = 0.0, fs = 0.0, ls = 0.0;
        // west x-face
        if (INNER || per_x || i >= 1) {
            if (qw != 0.0) {
                const bool pos = qw >= 0.0;
                fw = qw * face_value<ZV, MIX, INNER>(c, o, 1, s.nx, per_x, i, pos, (pos ? cls : cls >> 2) & 3u);
            }
            if (STAGE == 3) lw = qw * __ldg(c0 + (qw >= 0 ? (INNER || i >= 1 ? o - 1 : o + s.nx - 1) : o));
        } else {
            fw = edge_flux<1>(fl.open_w, qw, c[o], a.inflow ? a.inflow[pc + o] : c[o]);
            if (STAGE == 3) lw = edge_flux<1>(fl.open_w, qw, c0[o], a.inflow ? a.inflow[pc + o] : c0[o]);
        }
        const double aw = staged_flux<STAGE>(sx, tx, ox, fw, lw);
        sx[ox] = aw;
        if (per_x && i == 0) sx[ox + s.nx] = aw;
        // south y-face
        if (INNER || per_y || j >= 1) {
            if (qs != 0.0) {
                const bool pos = qs >= 0.0;
                fs = qs * face_value<ZV, MIX, INNER>(c, o, s.nx, s.ny, per_y, j, pos, (pos ? cls >> 4 : cls >> 6) & 3u);
            }
            if (STAGE == 3) ls = qs * __ldg(c0 + (qs >= 0 ? (INNER || j >= 1 ? o - s.nx : o + pl - s.nx) : o));
        } else {
            fs = edge_flux<1>(fl.open_s, qs, c[o], a.inflow ? a.inflow[pc + o] : c[o]);
            if (STAGE == 3) ls = edge_flux<1>(fl.open_s, qs, c0[o], a.inflow ? a.inflow[pc + o] : c0[o]);
        }
        const double as = staged_flux<STAGE>(sy, ty, o, fs, ls);
        sy[o] = as;
        if (per_y && j == 0) sy[o + pl] = as;
        // east / north domain faces of a closed or open axis
        double le = 0.0, ln = 0.0;
        if (last_x && !per_x) {
            const double q = __ldg(qx + (ox + 1));
            const double fe = edge_flux<-1>(fl.open_e, q, c[o], a.inflow ? a.inflow[pc + o] : c[o]);
            if (STAGE == 3) le = edge_flux<-1>(fl.open_e, q, c0[o], a.inflow ? a.inflow[pc + o] : c0[o]);
            sx[ox + 1] = staged_flux<STAGE>(sx, tx, ox + 1, fe, le);
        }
        if (last_y && !per_y) {
            const double q = __ldg(qy + (o + s.nx));
            const double fn = edge_flux<-1>(fl.open_n, q, c[o], a.inflow ? a.inflow[pc + o] : c[o]);
            if (STAGE == 3) ln = edge_flux<-1>(fl.open_n, q, c0[o], a.inflow ? a.inflow[pc + o] : c0[o]);
            sy[o + s.nx] = staged_flux<STAGE>(sy, ty, o + s.nx, fn, ln);
        }
        if (STAGE == 3) {
            // c_L = safe(q0 - dt div F_L, V1) of this cell (sigma_baroclinic.py:509-511): the donor fluxes of its
            // east and north faces are recomputed here (they are its neighbours' west and south faces), so F_L is
            // never stored and no separate cell pass runs.  c_L goes over c1, which no pass after stage 2 reads.
            const double cc = __ldg(c0 + o);
            if (!last_x || per_x) {
                const double q = __ldg(qx + (last_x ? ox + 1 - s.nx : ox + 1));
                le = q * (q >= 0 ? cc : __ldg(c0 + (last_x ? o + 1 - s.nx : o + 1)));
            }
            if (!last_y || per_y) {
                const double q = __ldg(qy + (last_y ? i : o + s.nx));
                ln = q * (q >= 0 ? cc : __ldg(c0 + (last_y ? i : o + s.nx)));
            }
            const double dl = le - lw + ln - ls;
            const i64 g = plane_at(k, pl);
            const double v0 = __ldg(a.V0 + g + o), v1 = __ldg(a.V1 + g + o);
            const double q0 = v0 * cc;
            const double q = 0.0 * q0 + 1.0 * (q0 - a.dt * dl);
            (a.c1 + pc)[o] = v1 > 0 ? q / v1 : cc;
        }
    }
}

// The cell's pass, with the domain-edge cases left out where the block of cells (TI x TJR from (i0, j0)) is at least
// three cells from every edge (85 % of the blocks at 512 x 512).
template <int STAGE, bool ZV, bool MIX, int TJR>
__device__ __forceinline__ void faces_body(const StepArgs& a, int t0, int t1, int k, int i0, int j0)
{
    const int i = i0 + threadIdx.x % TI, j = j0 + threadIdx.x / TI;
    if (i0 >= 3 && j0 >= 3 && i0 + TI + 2 <= a.s.nx && j0 + TJR + 2 <= a.s.ny) {
        faces_cell<STAGE, ZV, MIX, true>(a, t0, t1, k, i, j);
    } else if (i < a.s.nx && j < a.s.ny) {
        faces_cell<STAGE, ZV, MIX, false>(a, t0, t1, k, i, j);
    }
}

// Register budget of the face passes, as resident 256-thread blocks per SM (scaled for other block sizes): 7 for
// all three stages, which ptxas rounds to 32 registers and full occupancy (64 warps per SM; stages 1-2 and 3 spill
// a few values to L1).  Measured at 512 x 512 x 50: 2.0 % faster for advect_fct than 6 (40 registers), and 1.0 %
// faster than 32 registers for stages 1-2 with 40 for stage 3 or the reverse; 40 registers had been 8.5 % faster
// than ptxas's own choice (58 / 80 registers), whose lower occupancy left the FP64 chains and the loads exposed.
#ifndef POCEAN_FACES12_MINB
#define POCEAN_FACES12_MINB 7
#endif
#ifndef POCEAN_FACES3_MINB
#define POCEAN_FACES3_MINB 7
#endif
// The mixed-precision face passes (FP32 weights) hold FP32 copies beside the FP64 values: 7 blocks of 256 for stages 1
// and 2 and 6 (40 registers) for stage 3.  Four tracers of 512 x 512 x 75, the FCT step: 6.25 ms so, 6.52 with 7 for all,
// 6.25 with 6 for all, 6.47 with 6 and 5.
#ifndef POCEAN_FACES12_MINB_MIX
#define POCEAN_FACES12_MINB_MIX 7
#endif
#ifndef POCEAN_FACES3_MINB_MIX
#define POCEAN_FACES3_MINB_MIX 6
#endif
#define FACES12_BOUNDS(n) __launch_bounds__(n, (MIX ? POCEAN_FACES12_MINB_MIX : POCEAN_FACES12_MINB) * 256 / (n))
#define FACES3_BOUNDS(n) __launch_bounds__(n, (MIX ? POCEAN_FACES3_MINB_MIX : POCEAN_FACES3_MINB) * 256 / (n))
// The layer and the tracers t0 .. t1-1 of a single-domain face CTA: every tracer of layer blockIdx.z, or, where those
// CTAs would leave the chip idle (StepArgs::per_plane), the one tracer of plane blockIdx.z.
__device__ __forceinline__ void split_tracers(const StepArgs& a, int& k, int& t0, int& t1)
{
    if (a.per_plane) {
        split_plane(a.k0 * a.s.nt + blockIdx.z, a.s.nt, a.tdiv, k, t0);
        t1 = t0 + 1;
    } else {
        k = a.k0 + blockIdx.z;
        t0 = 0;
        t1 = a.s.nt;
    }
}

template <int STAGE, bool ZV, bool MIX, int TJR>
__device__ __forceinline__ void faces_plane(const StepArgs& a)
{
    int k, t0, t1;
    split_tracers(a, k, t0, t1);
    faces_body<STAGE, ZV, MIX, TJR>(a, t0, t1, k, blockIdx.x * TI, blockIdx.y * TJR);
}

template <int STAGE, bool ZV, bool MIX, int TJR>
__global__ void FACES12_BOUNDS(TI * TJR) fct_faces_kernel(StepArgs a)
{
    faces_plane<STAGE, ZV, MIX, TJR>(a);
}

template <bool ZV, bool MIX, int TJR>
__global__ void FACES3_BOUNDS(TI * TJR) fct_faces3_kernel(StepArgs a)
{
    faces_plane<3, ZV, MIX, TJR>(a);
}

template <int TJR>
__global__ void __launch_bounds__(TI * TJR) fct_class_kernel(StepArgs a)
{
    class_body(a, a.k0 + blockIdx.z, 4 * (blockIdx.x * TI + threadIdx.x % TI), blockIdx.y * TJR + threadIdx.x / TI);
}

// Where a batched CTA works: its domain's arguments, its layer k (and tracer t) and its TW x TH tile (bx, by).  PLANES:
// the domain's CTAs count tiles of the (t, k) planes (k-major: the cell passes); else tiles of the layers (t = 0).
struct BlockTile {
    int d, t, k, bx, by;
};

template <bool PLANES, int TW, int TH>
__device__ __forceinline__ BlockTile block_tile(const FctBatch& B)
{
    int lo = 0, hi = B.ndom - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (B.off[mid] <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    BlockTile bt;
    bt.d = lo;
    const Shape s = B.a[lo].s;
    const int tx = ceil_div(s.nx, TW), tiles = tx * ceil_div(s.ny, TH), local = blockIdx.x - B.off[lo];
    const int p = tile_div(local, B.per_layer[lo], tiles), rest = local - p * tiles;
    bt.t = 0;
    bt.k = p;
    if (PLANES) split_plane(p, s.nt, B.a[lo].tdiv, bt.k, bt.t);
    bt.by = tile_div(rest, B.per_row[lo], tx);
    bt.bx = rest - bt.by * tx;
    return bt;
}

template <int STAGE, bool ZV, bool MIX, int TJR>
__global__ void FACES12_BOUNDS(TI * TJR) fct_faces_batched(const __grid_constant__ FctBatch B)
{
    const BlockTile bt = block_tile<false, TI, TJR>(B);
    const StepArgs& a = B.a[bt.d];
    faces_body<STAGE, ZV, MIX, TJR>(a, 0, a.s.nt, bt.k, bt.bx * TI, bt.by * TJR);
}

template <bool ZV, bool MIX, int TJR>
__global__ void FACES3_BOUNDS(TI * TJR) fct_faces3_batched(const __grid_constant__ FctBatch B)
{
    const BlockTile bt = block_tile<false, TI, TJR>(B);
    const StepArgs& a = B.a[bt.d];
    faces_body<3, ZV, MIX, TJR>(a, 0, a.s.nt, bt.k, bt.bx * TI, bt.by * TJR);
}

// Tiles of the batched class pass: 32 x 32 cells by 256 threads of four cells each.
constexpr int CLASS_ROWS = 32;
__global__ void __launch_bounds__(TI / 4 * CLASS_ROWS) fct_class_batched(const __grid_constant__ FctBatch B)
{
    const BlockTile bt = block_tile<false, TI, CLASS_ROWS>(B);
    class_body(B.a[bt.d], bt.k, bt.bx * TI + 4 * (threadIdx.x % (TI / 4)), bt.by * CLASS_ROWS + threadIdx.x / (TI / 4));
}

// Cell pass of stage STAGE = 1, 2 (sigma_baroclinic.py:452-468 `_fct_stage`); stage 3 has none (its face pass
// writes c_L); STAGE = 4 is the unlimited step's final update from the RK3 flux.
template <int STAGE>
__device__ __forceinline__ void update_body(const StepArgs& a, int t, int k, int i, int j)
{
    const Shape s = a.s;
    if (i >= s.nx || j >= s.ny) return;
    const int pl = s.ny * s.nx, p = t * s.n + k, ij = j * s.nx + i;
    const i64 w = plane_at(p, s.ny * (s.nx + 1)) + (j * (s.nx + 1) + i), so = plane_at(p, (s.ny + 1) * s.nx) + ij;
    const i64 g = plane_at(k, pl) + ij, cc = plane_at(p, pl) + ij;
    const double v0 = __ldg(a.V0 + g), v1 = __ldg(a.V1 + g), c0 = __ldg(a.C + cc);
    const double q0 = v0 * c0;
    if (STAGE == 1) {
        const double d = a.Sx[w + 1] - a.Sx[w] + a.Sy[so + s.nx] - a.Sy[so];
        const double q = 0.0 * q0 + 1.0 * (q0 - a.dt * d);
        const double v = v0 + (v1 - v0);
        a.c1[cc] = v > 0.0 ? q / v : c0;
    } else if (STAGE == 2) {
        const double d0 = a.Sx[w + 1] - a.Sx[w] + a.Sy[so + s.nx] - a.Sy[so];
        const double d = a.Tx[w + 1] - a.Tx[w] + a.Ty[so + s.nx] - a.Ty[so];
        const double q1 = 0.0 * q0 + 1.0 * (q0 - a.dt * d0);
        const double q = 0.75 * q0 + 0.25 * (q1 - a.dt * d);
        const double v = v0 + 0.5 * (v1 - v0);
        a.c2[cc] = v > 0.0 ? q / v : c0;
    } else if (STAGE == 4) {     // the unlimited step (tracers.py:289-291): C_out = safe(q0 - dt div F_H, V1)
        const double d = a.Sx[w + 1] - a.Sx[w] + a.Sy[so + s.nx] - a.Sy[so];
        if (a.fx_face != nullptr && i == (a.face_i == s.nx ? s.nx - 1 : a.face_i))
            a.fx_face[((i64)t * s.n + k) * s.ny + j] = a.face_i == s.nx ? a.Sx[w + 1] : a.Sx[w];
        const double q = q0 - a.dt * d;
        a.out[cc] = v1 > 0 ? q / v1 : c0;
    }
}

template <int STAGE, int TJR>
__global__ void __launch_bounds__(TI * TJR) fct_update_kernel(StepArgs a)
{
    int k, t;
    split_plane(a.k0 * a.s.nt + blockIdx.z, a.s.nt, a.tdiv, k, t);
    update_body<STAGE>(a, t, k, blockIdx.x * TI + threadIdx.x % TI, blockIdx.y * TJR + threadIdx.x / TI);
}

template <int STAGE, int TJR>
__global__ void __launch_bounds__(TI * TJR) fct_update_batched(const __grid_constant__ FctBatch B)
{
    const BlockTile bt = block_tile<true, TI, TJR>(B);
    update_body<STAGE>(B.a[bt.d], bt.t, bt.k, bt.bx * TI + threadIdx.x % TI, bt.by * TJR + threadIdx.x / TI);
}

}  // namespace po
