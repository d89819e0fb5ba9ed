// pd_tile.cuh -- tiled Verlet structure shared by the integrator (see pd_tile.cu).
#pragma once
#include "pd_internal.cuh"

namespace pd {

static constexpr int TXMAX = 32;   // cells per tile along x, at most
static constexpr int TBLOCK = 128;   // threads per tile CTA of the list build
static constexpr int FBLOCK_T = 256; // threads per tile CTA of the pair kernels

struct TileGeom {
    int gs0, gs1, gs2, pad;
    int TX, ntx, ny, nz;
};

// Steps enqueued ahead of their rebuild decision (pd_md_run): a kernel of a step whose
// slot holds a squared displacement above lim2 does nothing but mark the next slot, so
// that every later step of the batch does nothing either.  slot nullptr: always runs.
struct StepGuard {
    const unsigned long long* slot = nullptr;
    unsigned long long* next = nullptr;
    double lim2 = 0;
};
#ifdef __CUDACC__
__device__ __forceinline__ bool step_skipped(const StepGuard& g) {
    if (!g.slot || !(__longlong_as_double((long long)*g.slot) > g.lim2)) return false;
    if (g.next && blockIdx.x == 0 && threadIdx.x == 0) *g.next = 0x7ff0000000000000ull;  // infinity
    return true;
}
#endif

int tile_plan(pd_cl cl, long n_real, int TX_req, TileGeom& tg, long& ntiles);
// the largest staged neighbourhood, centre count and staged layer of the tiles into the
// control block, and with `read` on to the host (one synchronisation)
int tile_sizes(pd_vd h, const TileGeom& tg, long ntiles, const unsigned int* csR, const unsigned int* csI,
               bool read, cudaStream_t st);
bool tile_fits(pd_vd h, unsigned int tmax);  // FP64/FP32 staging of the pair kernel fits
// bound on |d2_f32 - d2| for pairs near r in the vector's box (FP32 prefilter band of the build)
double fp32_band(pd_vd h, double r);
// the same for coordinates of magnitude up to X
double fp32_band_at(double X, double r);
// Rows of the tiles; `cap` and `pcap`: records of the largest neighbourhood and layer.
// PD_ESTATE with *small set (and nothing else wrong) when a layer was larger than pcap.
int tile_build(pd_vd h, const TileGeom& tg, long ntiles, const unsigned int* csR, const unsigned int* csI,
               unsigned int cap, unsigned int pcap, double r_list, Buf& pos32, Buf& nbr, Buf& nn, long& stride,
               int& max_nn, bool* small, cudaStream_t st);
// The FP64 pair kernel stages (x, y) and z from copies of the positions: those of
// the slots [first, first + n) refreshed from the records (room for the vector's capacity)
int tile_split(pd_vd h, Buf& sxy, Buf& sz, long first, long n, cudaStream_t st);
// The velocity-Verlet update a plain FP64 step makes after its forces, done by the
// pair kernel for each domain particle while the particle's force is in registers:
// the closing half kick of this step (kinetic energy partial), the next step's
// opening half kick and drift (the operations of the separate kick-kick-drift
// kernel, in its order), the drifted position into the vector and into the other
// pair of staging copies (the pair kernel still reads the current ones), and the
// largest |x - x_build|^2 into *maxd2.  The force itself is not stored: the next
// step recomputes it before anything reads it.  With `close` (a run's last step) only the
// closing half kick is made and the force is stored.
struct DriftArgs {
    bool close;
    double4* pos;
    const double4* xb;
    double* v;
    long vcap;
    double half, dt, mass;
    double2* sxy_next;
    double* sz_next;
    unsigned long long* maxd2;
};
// LJ forces from the tiled rows (FP64: from the staging copies sxy / sz, which must be
// current).  Per tile, part receives (pe, vir), or (pe, vir, ke) with `drift`.
int tile_lj(pd_vd h, const TileGeom& tg, long ntiles, const unsigned int* csR, const unsigned int* csI,
            unsigned int cap, const Buf& nbr, const Buf& nn, long stride, const pd_lj_params_t& lj, int force_prop,
            double* part, bool energy, int P, const Buf& sxy, const Buf& sz, cudaStream_t st,
            const DriftArgs* drift = nullptr, const StepGuard& guard = StepGuard());
int tile_translate(pd_vd h, const TileGeom& tg, long ntiles, const unsigned int* csR, const unsigned int* csI,
                   const Buf& nbr, const Buf& nn, long stride, int max_nn, int* out_dev, cudaStream_t st);

}  // namespace pd
