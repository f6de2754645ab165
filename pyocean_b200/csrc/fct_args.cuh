// Argument blocks of the advection kernels and of the batched (multi-domain) launches.
#pragma once

#include "common.cuh"

namespace po {

struct Flags {
    bool open_w, open_e, open_s, open_n, per_x, per_y, z;
    __host__ __device__ explicit Flags(unsigned f)
        : open_w(f & POCEAN_OPEN_W), open_e(f & POCEAN_OPEN_E), open_s(f & POCEAN_OPEN_S),
          open_n(f & POCEAN_OPEN_N), per_x(f & POCEAN_PERIODIC_X), per_y(f & POCEAN_PERIODIC_Y),
          z(!(f & POCEAN_WENO_JS)) {}
};

// Everything one FCT / RK3 step reads and writes.
struct StepArgs {
    Shape s;
    unsigned flags;
    double dt;
    const double* __restrict__ C;
    const double* __restrict__ V0;
    const double* __restrict__ V1;
    const double* __restrict__ Qx;
    const double* __restrict__ Qy;
    const double* __restrict__ Fz;      // RK3 only (nullable)
    const uint8_t* __restrict__ ok;
    const double* __restrict__ inflow;  // nullable
    // workspace
    double* q1;
    double* c1;
    double* q2;
    double* c2;
    double* Sx;                         // FCT: F0, then the antidiffusive flux A
    double* Sy;
    double* Tx;                         // FCT: F1
    double* Ty;
    double* tef0;                       // RK3 TEF column accumulators (nt, n, ny)
    double* tef1;
    // outputs
    double* out;
    int face_i;
    int k0;                             // first layer of a layer-range launch of the single-domain passes (else 0)
    unsigned tdiv;                      // plane_magic(s.nt): plane index -> layer without an integer division
    int per_plane;                      // single-domain face CTAs take one (tracer, layer) plane each (split_tracers)
    double* fx_face;
};

// One domain of a batch: its FCT arguments (a.C the stack, a.out the advected stack, a.q1.. its workspace) and
// the remap of the advected stack onto its target grid (into rout).
struct BatchDomain {
    StepArgs a;
    const double* h_src;
    const double* h_tgt;
    const uint8_t* wet;
    double* rout;
    int remap_scheme;
};

// Layer k and tracer t of plane p = k nt + t (planes run k-major); tdiv = plane_magic(nt).  The multiply-high
// replaces a per-warp integer division (about twenty instructions): 1.6 % of advect_fct at 512 x 512 x 50.
__device__ __forceinline__ void split_plane(int p, int nt, unsigned tdiv, int& k, int& t)
{
    k = plane_div(p, tdiv);
    t = p - k * nt;
}

// CTA offsets of the batched remap launches: domain d owns CTAs off[d] .. off[d+1]-1 of the launch (ndom + 1 entries
// each), for column groups x field pairs, odd fields, all fields.
enum BatchPass { BP_RPAIR = 0, BP_RREM, BP_RALL, BP_COUNT };

// The domain whose CTA range holds CTA b (binary search of off[0..ndom]).
__device__ __forceinline__ int find_domain(const int* __restrict__ off, int ndom, int b)
{
    int lo = 0, hi = ndom - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// A batched FCT launch: its domains' argument blocks and CTA ranges, passed as the kernel's parameter.  Parameters lie in
// constant memory, so a CTA's search for its domain, its tile and every argument it reads are the same for all its
// threads to the compiler and stay in uniform registers, as in a single-domain launch.  (Read from a device table
// through shared memory they cost a batched step 11 % more than the single-domain calls, and each CTA the latency of the
// search.)  Batches of more domains take several launches.
constexpr int BATCH_CAP = 64;
struct FctBatch {
    int ndom;
    int off[BATCH_CAP + 1];                       // domain d owns CTAs off[d] .. off[d+1]-1
    unsigned long long per_layer[BATCH_CAP];      // tile_magic of the tiles of a layer and of a row of tiles
    unsigned long long per_row[BATCH_CAP];
    StepArgs a[BATCH_CAP];
};
static_assert(sizeof(FctBatch) <= 32000, "kernel parameters hold 32764 bytes");

// The FCT workspace cut into a's buffers (advect.cu).
void carve_fct_workspace(StepArgs& a, void* workspace);

// Host launchers of the batched passes (advect.cu, remap.cu).  doms: the step's argument blocks, on the host and (for
// the remap) on the device.
cudaError_t fct_batched_launch(const BatchDomain* doms_host, int ndom, bool zv, bool mixed, int tile_rows,
                               cudaStream_t st);
int fct_batch_launches(const int* shapes, int ndom);
int remap_batch_launches(const int* shapes, int ndom, int nf_mode);
bool remap_batch_segments(long long columns, int nmax);
int remap_batched_columns(bool segments);
cudaError_t remap_batched_launch(const BatchDomain* doms, const int* off_dev, const int* off_host, int ndom, int nf_mode,
                                 int nmax, bool segments, cudaStream_t st);

}  // namespace po
