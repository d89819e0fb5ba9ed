// pd_verlet.cu -- full Verlet list on the GPU (getVerlet / updateVerlet).
//
// The reference builds this list on the CPU only (vector_dist.hpp:1514-1620):
// for every domain particle, all particles (domain + ghost, self included) with
// d2 < r_cut^2, found through a cell list of side r_cut over the domain
// enlarged by the ghost magnified 1.013.  Here:
//   1. the cell list is built by the counting sort of pd_celllist.cu;
//   2. FP32 copies of the positions are gathered into cell order with the original
//      index in the record's 4th word;
//   3. one CTA per tile of TX cells along x stages the 9 neighbour rows
//      (x-1 .. x+TX for dy, dz in {-1,0,1}; each a contiguous range of the copies) in
//      shared memory, all at once or one z-layer at a time, and every thread scans the 27-cell
//      neighbourhood of its particles from there, in the reference walk order (dz,
//      dy, dx, in-cell order), writing column-major rows nbr[k*stride + i].
// Rows longer than the capacity set ERR_NN_OVERFLOW and record the longest row;
// the host grows the capacity and rebuilds.
//
// Symmetric (half) list, getVerletSym (vector_dist.hpp:1412-1416): each
// interacting pair once.  A domain partner q is kept by p iff q > p; a periodic
// image is kept iff it lies after p in the lexicographic (x, y, z) order.  The
// mirror of a pair (p, image of r) is (r, image of p), shifted by the opposite
// vector, so exactly one of the two is kept; forces or counts accumulated on an
// image are folded onto its source by ghost_put<add_> (vector_dist.hpp:2304).
// The criterion is geometric, not cell-based, so it does not depend on the box
// being a whole number of cells.
#include <cmath>

#include "pd_device.cuh"
#include "pd_internal.cuh"
#include "pd_tile.cuh"
#include "pd_tile_dev.cuh"

namespace pd {

// largest coordinate of a position inside the cell grid, padding cells included
static double verlet_bound(pd_cl cl) {
    double X = 0;
    for (int d = 0; d < 3; ++d) {
        const double a = cl->box_lo[d] - cl->pad * cl->spacing[d];
        const double b = cl->box_lo[d] + (cl->gs[d] - cl->pad) * cl->spacing[d];
        X = std::max(X, std::max(std::fabs(a), std::fabs(b)));
    }
    return X * (1.0 + 1e-6);
}

// p32[k] = FP32 copy of pos[sorted[k]] with the original index in w: what the row
// kernel stages, half the bytes of an FP64 record.  A coordinate beyond `bound`, the padded
// grid, or a NaN is stored as infinity, which no test accepts: the particle lies in a padding
// cell (clamped), so it has no row itself and is more than a cell side, the cutoff, away from
// every particle that has one.
template <class T>
__global__ void k_gather_cs(const typename V4<T>::type* __restrict__ pos, const int* __restrict__ sorted,
                            const unsigned int* __restrict__ cs_end, float4* __restrict__ out, long n_bound, T bound) {
    long n = (long)*cs_end;
    if (n > n_bound) n = n_bound;
    auto f32 = [&](T c) { return fabs(c) <= bound ? (float)c : INFINITY; };
    for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
        const int i = sorted[k];
        const typename V4<T>::type r = ld4(pos, i);
        out[k] = make_float4(f32(r.x), f32(r.y), f32(r.z), __int_as_float(i));
    }
}

template <class T4> __device__ __forceinline__ bool lex_after(const T4& a, const T4& b) {
    return a.x > b.x || (a.x == b.x && (a.y > b.y || (a.y == b.y && a.z > b.z)));
}

// the 9 cell-row ranges of tile t in the cell-ordered array (no image ranges: real
// particles and ghosts are sorted together)
__device__ __forceinline__ void verlet_layout(const TileGeom& tg, long t, const unsigned int* __restrict__ cs,
                                              TileSh& S) {
    const int tx = (int)(t % tg.ntx);
    const long rest = t / tg.ntx;
    const int y = (int)(rest % tg.ny) + tg.pad, z = (int)(rest / tg.ny) + tg.pad;
    const int x0 = tg.pad + tx * tg.TX, x1 = min(x0 + tg.TX, tg.gs0 - tg.pad);
    const int ncol = x1 - x0 + 3;  // cells x0-1 .. x1 and the end of cell x1
    for (int e = threadIdx.x; e < 9 * ncol; e += blockDim.x) {
        const int r = e / ncol, j = e % ncol;
        const int dz = r / 3 - 1, dy = r % 3 - 1;
        S.cR[r][j] = cs[(long)(x0 - 1 + j) + (long)tg.gs0 * ((y + dy) + (long)tg.gs1 * (z + dz))];
    }
    if (threadIdx.x < 9) S.cI[threadIdx.x][0] = S.cI[threadIdx.x][ncol - 1] = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int o = 0;
        for (int r = 0; r < 9; ++r) {
            S.oR[r] = S.oI[r] = o;
            o += S.cR[r][ncol - 1] - S.cR[r][0];
        }
        S.total = o;
        S.ncol = ncol;
    }
    __syncthreads();
}

// half-list rule: a domain partner q of i iff q > i, an image iff it lies after i
template <class T>
__device__ __forceinline__ bool sym_keep(const typename V4<T>::type* __restrict__ pos, int i, int q, long n_dom) {
    if (q < n_dom) return q > i;
    const typename V4<T>::type a = ld4(pos, (long)q), b = ld4(pos, (long)i);
    return lex_after(a, b);
}

// Entries of particle i from the n candidates c4[0..n) appended to its row in
// candidate order: accept masks of two chunks of 32 first, then one stream
// of the accepted ones (see seg_rows).  Works on staged and on global records.
template <class T, bool SYM>
__device__ __forceinline__ void verlet_seg(const float4* __restrict__ c4, unsigned int n, const float4 x, int i,
                                           const typename V4<T>::type* __restrict__ pos, T r2, float lo_thr,
                                           float hi_thr, long n_dom, int* __restrict__ out, long stride, int max_nn,
                                           int& c) {
#pragma unroll 1
    for (unsigned int q0 = 0; q0 < n; q0 += 64) {
        const unsigned int m = min(64u, n - q0);
        const unsigned int na = min(32u, m), nb = m - na;
        unsigned int ma = chunk_mask<T>(c4 + q0, na, x, (unsigned int)i, pos, r2, lo_thr, hi_thr);
        unsigned int mb = chunk_mask<T>(c4 + q0 + 32, nb, x, (unsigned int)i, pos, r2, lo_thr, hi_thr);
        int rem = __popc(ma) + __popc(mb);
        // the highest bit of each mask for its chunk's first candidate
        ma <<= 32 - na;
        mb = __funnelshift_lc(0u, mb, 32 - nb);
        for (unsigned int qa = q0; rem > 0; --rem) {
            if (ma == 0) { ma = mb; qa += 32; }
            const int z = __clz(ma);
            ma ^= 0x80000000u >> z;
            const int q = __float_as_int(c4[qa + (unsigned int)z].w);
            if (SYM && !sym_keep<T>(pos, i, q, n_dom)) continue;
            if (c < max_nn) out[(long)c * stride] = q;
            ++c;
        }
    }
}

// Rows of the domain particles of one tile (TX cells of a cell row), global original
// indices, column-major nbr[k*stride + i], in the walk order dz, dy, dx, in-cell.
// Bound by the instructions of the candidate tests (27 cells hold about 6.4 times
// the pairs kept), so: FP32 tests on 16-byte staged copies, sign bits shifted into
// accept masks, the rare candidates within the rounding band decided exactly in the
// position type (the scheme of the integrator's row build).  The neighbourhood is staged
// at once where it fits `pcap` records (eight CTAs per SM), so that a CTA's warps wait for
// each other once; else one z-layer of three cell rows at a time; a layer beyond `pcap`
// records is read from global memory instead.
// Measured: 1,000,000 FP64 particles of a lattice (49 entries a row) 1198 -> 421 us, half
// rows of 200,001 348 -> 144 us against FP64 records of all nine rows staged at once.
template <class T, bool SYM>
__global__ void __launch_bounds__(TBLOCK, 8) k_verlet_rows(const typename V4<T>::type* __restrict__ pos,
                                                        const float4* __restrict__ p32, TileGeom tg,
                                                        const unsigned int* __restrict__ cs, long n_dom, T r2,
                                                        float lo_thr, float hi_thr, int* __restrict__ nbr,
                                                        int* __restrict__ nn, long stride, int max_nn,
                                                        unsigned int pcap,
                                                        unsigned int* __restrict__ ctrl_err,
                                                        unsigned int* __restrict__ ctrl_nnmax) {
    extern __shared__ __align__(128) unsigned char tile_raw[];
    float4* sm = reinterpret_cast<float4*>(tile_raw);
    __shared__ TileSh S;
    verlet_layout(tg, blockIdx.x, cs, S);
    const int ncol = S.ncol;
    const unsigned int ib = S.cR[4][1], ie = S.cR[4][ncol - 2];
    if (ib == ie) return;
    if (threadIdx.x == 0) mbar_init(&S.bar, 1);
    unsigned int ph = 0;
    bool held = false;  // the whole neighbourhood is staged
    // up to MAXI particles a thread and sweep; a denser tile takes further sweeps
    constexpr int MAXI = 2;
    const unsigned int sweep = (unsigned int)MAXI * blockDim.x;
    for (unsigned int sb = ib; sb < ie; sb += sweep) {
        float4 xi[MAXI];
        int jcol[MAXI], cnt[MAXI];
        bool dom = false;
#pragma unroll
        for (int m = 0; m < MAXI; ++m) {
            const unsigned int k = sb + threadIdx.x + (unsigned int)m * blockDim.x;
            xi[m] = k < ie ? p32[k] : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
            cnt[m] = 0;
            int j = 1;
            while (j < ncol - 2 && S.cR[4][j + 1] <= k) ++j;
            const int i = __float_as_int(xi[m].w);
            jcol[m] = i >= 0 && i < n_dom ? j : 0;  // 0: no row (past the tile, or a ghost)
            dom = dom || jcol[m] != 0;
        }
        if (!__syncthreads_or(dom ? 1 : 0)) continue;  // ghosts only; also covers the barrier's initialisation
        // the whole neighbourhood in one pass where it fits the staging, else a z-layer a pass
        const int layers = S.total <= pcap ? 9 : 3;  // rows a pass
        for (int r0 = 0; r0 < 9; r0 += layers) {
            const unsigned int base = S.oR[r0];
            const unsigned int tot = (r0 + layers < 9 ? S.oR[r0 + layers] : S.total) - base;
            const bool staged = tot <= pcap;
            if (staged && tot > 0 && (layers < 9 || !held)) {
                if (threadIdx.x < 32)
                    stage_ranges_warp(S, r0, layers, sm, base, p32, p32, tot * (unsigned int)sizeof(float4), &S.bar);
                const bool ok = mbar_wait_bounded(&S.bar, ph & 1u, 1u << 24);
                if (!ok) {
                    atomicOr(ctrl_err, ERR_TIMEOUT);
                    mbar_wait_bounded(&S.bar, ph & 1u, 1u << 24);
                }
                ++ph;
                held = layers == 9;
                if (!__syncthreads_and(ok ? 1 : 0)) return;
            }
#pragma unroll
            for (int m = 0; m < MAXI; ++m) {
                const int j = jcol[m];
                if (j == 0) continue;
                const int i = __float_as_int(xi[m].w);
                int c = cnt[m];
#pragma unroll 1
                for (int r = r0; r < r0 + layers; ++r) {
                    const unsigned int a = S.cR[r][j - 1], n = S.cR[r][j + 2] - a;
                    if (staged)
                        verlet_seg<T, SYM>(sm + (S.oR[r] - base + (a - S.cR[r][0])), n, xi[m], i, pos, r2, lo_thr,
                                           hi_thr, n_dom, nbr + i, stride, max_nn, c);
                    else
                        verlet_seg<T, SYM>(p32 + a, n, xi[m], i, pos, r2, lo_thr, hi_thr, n_dom, nbr + i, stride,
                                           max_nn, c);
                }
                cnt[m] = c;
            }
            if (layers < 9) {
                // every thread is done with this layer before the next one is copied over it
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncthreads();
            }
        }
#pragma unroll
        for (int m = 0; m < MAXI; ++m) {
            if (jcol[m] == 0) continue;
            int c = cnt[m];
            if (c > max_nn) {
                atomicOr(ctrl_err, ERR_NN_OVERFLOW);
                atomicMax(ctrl_nnmax, (unsigned int)c);
                c = max_nn;
            }
            nn[__float_as_int(xi[m].w)] = c;
        }
    }
}

// Tile width: about a CTA's 128 threads of particles on average, at most 16 cells
// (dense tiles of a sparse system otherwise outgrow the staging), narrower where
// that leaves the GPU's 148 SMs with less than four tiles each.
static int choose_tx(pd_cl cl, long n_all) {
    const double cells = (double)cl->div[0] * cl->div[1] * cl->div[2];
    const double occ = std::max(cells > 0 ? (double)n_all / cells : 1.0, 1e-3);
    const long rows = (long)(cl->gs[1] - 2 * cl->pad) * (cl->gs[2] - 2 * cl->pad);
    const int nxi = cl->gs[0] - 2 * cl->pad;
    int tx = (int)std::min(16.0, 124.0 / occ);
    const long want = 4 * 148;
    if (rows * ((nxi + std::max(tx, 1) - 1) / std::max(tx, 1)) < want) tx = std::min(tx, (int)((long)nxi * rows / want));
    return std::max(1, std::min(tx, nxi));
}

template <class T>
static int verlet_rows(pd_vd h, pd_vl vl, const float4* p32, const TileGeom& tg, long ntiles, long n_dom, long stride,
                       cudaStream_t st) {
    typedef typename V4<T>::type T4;
    pd_cl cl = vl->cl;
    // staging: 1536 records (24 KB, eight CTAs per SM)
    const unsigned int pcap = 1536;
    const T rc = (T)vl->r_cut;
    const T r2 = rc * rc;
    // FP32 positions are staged as they are: their band covers the rounding of the sums only
    // (the test adds in another order than the predicate), down to a few subnormal steps
    const double band = fp32_band_at(sizeof(T) == 8 ? verlet_bound(cl) : 0.0, vl->r_cut) + std::ldexp(1.0, -146);
    const float lo_thr = (float)((double)r2 - band), hi_thr = (float)((double)r2 + band);
    auto go = [&](auto k) {
        pd::launch(k, (unsigned)ntiles, TBLOCK, pcap * sizeof(float4), st, (const T4*)h->pos, p32, tg,
                   (const unsigned int*)cl->cell_start.as<unsigned int>(), n_dom, r2, lo_thr, hi_thr, vl->nbr.as<int>(),
                   vl->nn.as<int>(), stride, vl->max_nn, pcap, &h->ctrl->err, &h->ctrl->nn_max);
    };
    if (vl->sym) go(k_verlet_rows<T, true>);
    else go(k_verlet_rows<T, false>);
    PD_LAUNCH_CHECK();
    return PD_OK;
}

// Build the list of domain particles [0, n_dom) over all particles; the
// particle count is h->n_real + *n_img_dev when n_img_dev is given (device
// resident), else h->n_total.
int verlet_build(pd_vd h, pd_vl vl, long n_dom, const unsigned int* n_img_dev, cudaStream_t st, bool check) {
    pd_cl cl = vl->cl;
    long n_all_bound = n_img_dev ? h->cap : h->n_total;
    PD_TRY(cl_build(h, cl, n_all_bound, n_img_dev, st));
    // cell-ordered FP32 copies with original indices
    PD_TRY(h->tmp.ensure((size_t)(n_all_bound > 0 ? n_all_bound : 1) * sizeof(float4)));
    const unsigned int* cs_end = cl->cell_start.as<unsigned int>() + cl->ncells;
    unsigned g = grid_for(n_all_bound, 256);
    if (h->dtype == PD_F64)
        pd::launch(k_gather_cs<double>, g, 256, 0, st, (const double4*)h->pos, cl->sorted.as<int>(), cs_end,
                                               h->tmp.as<float4>(), n_all_bound, verlet_bound(cl));
    else  // staged as they are
        pd::launch(k_gather_cs<float>, g, 256, 0, st, (const float4*)h->pos, cl->sorted.as<int>(), cs_end,
                                              h->tmp.as<float4>(), n_all_bound, INFINITY);
    PD_LAUNCH_CHECK();
    long stride = ((n_dom + 31) / 32) * 32;
    if (stride < 32) stride = 32;
    if (vl->max_nn <= 0) {
        // first build: capacity from the mean density within r (x1.5 + 32), grown on overflow
        double vol = 1.0;
        for (int d = 0; d < 3; ++d) vol *= (h->hi[d] - h->lo[d] + 2 * h->g[d]);
        double dens = (double)(n_img_dev ? h->n_real * 1.3 : h->n_total) / vol;
        double mean = dens * 4.18879 * vl->r_cut * vl->r_cut * vl->r_cut;
        vl->max_nn = (int)(mean * 1.5 + 32);
    }
    for (int attempt = 0; attempt < 3; ++attempt) {
        PD_TRY(vl->nbr.ensure(sizeof(int) * (size_t)stride * vl->max_nn));
        PD_TRY(vl->nn.ensure(sizeof(int) * (n_dom > 0 ? n_dom : 1)));
        vl->stride = stride;
        vl->n_dom = n_dom;
        if (n_dom > 0) {
            // a particle outside the grid (never mapped) lies in no tile: its row is empty
            PD_CUDA(cudaMemsetAsync(vl->nn.p, 0, sizeof(int) * (size_t)n_dom, st));
            TileGeom tg;
            long ntiles = 0;
            PD_TRY(tile_plan(cl, n_dom, choose_tx(cl, h->n_total > 0 ? h->n_total : h->n_real), tg, ntiles));
            if (h->dtype == PD_F64) PD_TRY(verlet_rows<double>(h, vl, h->tmp.as<float4>(), tg, ntiles, n_dom, stride, st));
            else PD_TRY(verlet_rows<float>(h, vl, h->tmp.as<float4>(), tg, ntiles, n_dom, stride, st));
        }
        if (!check) return PD_OK;
        PD_TRY(read_ctrl(h, st));
        PD_TRY(take_timeout(h, "Verlet list", st));
        if (!(h->ctrl_h->err & ERR_NN_OVERFLOW)) break;
        // grow and rebuild
        vl->max_nn = (int)(h->ctrl_h->nn_max * 1.15 + 8);
        h->ctrl_h->err &= ~ERR_NN_OVERFLOW;
        h->ctrl_h->nn_max = 0;
        PD_CUDA(cudaMemcpyAsync(&h->ctrl->err, &h->ctrl_h->err, sizeof(unsigned int) * 3, cudaMemcpyHostToDevice, st));
    }
    vl->epoch = h->epoch;
    return PD_OK;
}

}  // namespace pd

using namespace pd;

extern "C" {

int pd_verlet_create(pd_vd h, double r_cut, pd_vl* out) {
    if (!h || !out || !(r_cut > 0)) return PD_EINVAL;
    pd_vl vl = new pd_vl_s();
    vl->owner = h;
    vl->r_cut = r_cut;
    vl->cl = new pd_cl_s();
    int r = cl_geometry(vl->cl, h, r_cut, 1.013, 1);
    if (r != PD_OK) {
        delete vl->cl;
        delete vl;
        return r;
    }
    *out = vl;
    return PD_OK;
}

int pd_verlet_create_sym(pd_vd h, double r_cut, pd_vl* out) {
    int r = pd_verlet_create(h, r_cut, out);
    if (r == PD_OK) (*out)->sym = true;
    return r;
}

int pd_verlet_destroy(pd_vl vl) {
    if (!vl) return PD_EINVAL;
    if (vl->cl) pd_celllist_destroy(vl->cl);
    vl->nbr.release();
    vl->nn.release();
    delete vl;
    return PD_OK;
}

int pd_verlet_update(pd_vd h, pd_vl vl, void* stream) {
    if (!h || !vl || vl->owner != h) return PD_EINVAL;
    return verlet_build(h, vl, h->n_real, nullptr, S(stream), true);
}

int pd_verlet_get(pd_vl vl, int* counts, int* idx, long idx_cap, void* stream) {
    if (!vl || !counts) return PD_EINVAL;
    cudaStream_t st = S(stream);
    long n = vl->n_dom;
    if (n == 0) return PD_OK;
    PD_CUDA(cudaMemcpyAsync(counts, vl->nn.p, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    PD_CUDA(cudaStreamSynchronize(st));
    if (!idx) return PD_OK;
    long tot = 0;
    int mx = 0;
    for (long i = 0; i < n; ++i) {
        tot += counts[i];
        mx = std::max(mx, counts[i]);
    }
    if (tot > idx_cap) {
        set_error("pd_verlet_get: idx_cap %ld < %ld entries", idx_cap, tot);
        return PD_EINVAL;
    }
    std::vector<int> col((size_t)vl->stride * mx);
    if (mx > 0)
        PD_CUDA(cudaMemcpy(col.data(), vl->nbr.p, sizeof(int) * (size_t)vl->stride * mx, cudaMemcpyDeviceToHost));
    long o = 0;
    for (long i = 0; i < n; ++i)
        for (int k = 0; k < counts[i]; ++k) idx[o++] = col[(size_t)k * vl->stride + i];
    return PD_OK;
}

}  // extern "C"
