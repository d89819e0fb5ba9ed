// pd_cluster.cu -- velocity-Verlet LJ steps of a small system with the cell list
// rebuilt every step, all steps of a run in one launch: k_md_buckets on the whole GPU
// (second half of this file), k_md_cluster on one thread-block cluster where a bucket
// overflows or the buckets do not fit.
//
// The cell-list step (kick-drift, wrap, periodic images, cell list of particles and
// images, 27-cell force walk, kick, energies) is a dozen dependent phases over a
// few thousand particles: as separate kernels (even replayed from a CUDA graph)
// the launch gaps dominate.  Here one cluster of 16 CTAs (16 SMs; 8 where the GPU
// cannot place a cluster of 16) runs every phase of every step, with the cluster barrier (barrier.cluster, a hardware
// barrier that every thread of the cluster reaches the same number of times: the
// control flow around it is uniform) between dependent phases; the scans run on
// the cluster's first CTA.  Data stay in global memory (a few hundred KB, L2
// resident).  The phases restate the separate kernels' operations (k_kick_drift,
// k_wrap, k_ghost_count / k_ghost_write, the counting sort with its stabilising
// rank pass, k_lj_cell, k_kick) in the same arithmetic order per particle; only
// the order of the energy sums differs.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "pd_device.cuh"
#include "pd_ghost_dev.cuh"
#include "pd_internal.cuh"
#include "pd_lj.cuh"
#include "pd_md.cuh"

namespace cg = cooperative_groups;

namespace pd {

static constexpr int CL_CTAS = 16;       // CTAs of the cluster (non-portable size; 8 where 16 cannot be placed)
static constexpr int CL_THREADS = 1024;  // threads per CTA
static constexpr long CL_MAXN = 65536;   // real particles handled by the cluster path
static constexpr unsigned int CL_SORT_CAP = 256;  // shared ints per warp for ordering a crowded cell

template <class T> struct ClArgs {
    typename V4<T>::type* pos;  // real [0, n), images [n, n + img_cap)
    int* gid;
    int* img_src;
    unsigned char* img_shift;
    T* v;
    T* f;
    long cap, n, img_cap;
    T lo[3], hi[3];
    int per[3];
    const BoxSet<T>* boxes;
    const T* shifts;
    Grid<T> G;
    long ncells;
    unsigned int *cnt, *cstart, *cell_of, *slot, *img_cnt, *img_start, *tot;
    int *sorted_tmp, *sorted;
    typename V4<T>::type* pcs;  // cell-ordered copy of positions and images, w = index bits
    int q;                      // lanes per particle in the force walk (a power of two <= 32)
    LJP<T> P;
    T half, dt;
    double mass;
    double* part;  // [CTAs][3]: potential energy, virial, kinetic energy
    double* E;     // [steps][4]
    int steps;
    unsigned int* err;
};

// coherent loads of position records (data written earlier in the same launch by
// other CTAs of the cluster: not through the read-only cache)
__device__ __forceinline__ double4 ldc4(const double4* p, long i) {
    const double2* q = reinterpret_cast<const double2*>(p + i);
    const double2 a = q[0], b = q[1];
    return make_double4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 ldc4(const float4* p, long i) { return p[i]; }

template <class T> __device__ __forceinline__ T idx_bits(int i);
template <> __device__ __forceinline__ double idx_bits<double>(int i) { return __longlong_as_double((long long)i); }
template <> __device__ __forceinline__ float idx_bits<float>(int i) { return __int_as_float(i); }
template <class T> __device__ __forceinline__ int idx_of(T w);
template <> __device__ __forceinline__ int idx_of<double>(double w) { return (int)__double_as_longlong(w); }
template <> __device__ __forceinline__ int idx_of<float>(float w) { return __float_as_int(w); }

// exclusive scan of a[0, n) into out (out may alias a), total to *total; one CTA
__device__ void cta_scan(const unsigned int* a, unsigned int* out, long n, unsigned int* total, unsigned int* wsum) {
    const long C = (n + CL_THREADS - 1) / CL_THREADS;
    const long b = (long)threadIdx.x * C;
    unsigned int loc = 0;
    for (long j = 0; j < C; ++j)
        if (b + j < n) loc += a[b + j];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int inc = loc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const unsigned int y = wsum[lane];
        unsigned int z = y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int t = __shfl_up_sync(0xffffffffu, z, o);
            if (lane >= o) z += t;
        }
        wsum[lane] = z - y;
    }
    __syncthreads();
    unsigned int run = wsum[warp] + inc - loc;
    for (long j = 0; j < C; ++j)
        if (b + j < n) {
            const unsigned int v = a[b + j];
            out[b + j] = run;
            run += v;
        }
    if (threadIdx.x == CL_THREADS - 1) *total = run;
    __syncthreads();
}

template <class T>
__global__ void __launch_bounds__(CL_THREADS, 1) k_md_cluster(ClArgs<T> A) {
    typedef typename V4<T>::type T4;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ BoxSet<T> B;
    __shared__ unsigned int wsum[32];
    __shared__ int cell_sort_buf[32][CL_SORT_CAP];  // per warp: in-cell ordering of crowded cells
    for (int i = threadIdx.x; i < (int)(sizeof(BoxSet<T>) / 4); i += blockDim.x)
        reinterpret_cast<int*>(&B)[i] = reinterpret_cast<const int*>(A.boxes)[i];
    __syncthreads();
    const unsigned int rank = cluster.block_rank();
    const long gt = (long)rank * CL_THREADS + threadIdx.x;
    const int nct = (int)cluster.num_blocks();
    const long GT = (long)nct * CL_THREADS;
    const long n = A.n;
    unsigned int bad = 0, ovf = 0;
    for (int s = 0; s < A.steps; ++s) {
        // 1. v += h f; x += dt v; periodic wrap.  Cell counts cleared.
        for (long i = gt; i < n; i += GT) {
            T4 x = ldc4(A.pos, i);
            const T vx = A.v[i] + A.half * A.f[i];
            const T vy = A.v[A.cap + i] + A.half * A.f[A.cap + i];
            const T vz = A.v[2 * A.cap + i] + A.half * A.f[2 * A.cap + i];
            x.x += A.dt * vx;
            x.y += A.dt * vy;
            x.z += A.dt * vz;
            A.v[i] = vx;
            A.v[A.cap + i] = vy;
            A.v[2 * A.cap + i] = vz;
            if (A.per[0]) x.x = periodic_l(x.x, A.hi[0], A.lo[0]);
            if (A.per[1]) x.y = periodic_l(x.y, A.hi[1], A.lo[1]);
            if (A.per[2]) x.z = periodic_l(x.z, A.hi[2], A.lo[2]);
            st4(A.pos, i, x);
        }
        for (long c = gt; c <= A.ncells; c += GT) A.cnt[c] = 0u;
        cluster.sync();
        // 2. images per particle: distinct shift ids of the ghost boxes holding it
        for (long i = gt; i < n; i += GT) {
            const T4 r = ldc4(A.pos, i);
            unsigned int c = 0;
            int old = -1;
            for (int b = 0; b < B.nb; ++b) {
                const int sv = B.sv[b];
                if (inside_np(B, b, r.x, r.y, r.z) && sv != old) {
                    old = sv;
                    ++c;
                }
            }
            A.img_cnt[i] = c;
        }
        cluster.sync();
        // 3. image offsets (first CTA)
        if (rank == 0) cta_scan(A.img_cnt, A.img_start, n, A.tot, wsum);
        cluster.sync();
        // 4. the images, particle-major, shift ids ascending
        for (long i = gt; i < n; i += GT) {
            const T4 r = ldc4(A.pos, i);
            long m = A.img_start[i];
            int old = -1;
            for (int b = 0; b < B.nb; ++b) {
                const int sv = B.sv[b];
                if (inside_np(B, b, r.x, r.y, r.z) && sv != old) {
                    old = sv;
                    if (m < A.img_cap && n + m < A.cap) {
                        T4 q;
                        q.x = r.x - A.shifts[3 * sv];
                        q.y = r.y - A.shifts[3 * sv + 1];
                        q.z = r.z - A.shifts[3 * sv + 2];
                        q.w = r.w;
                        st4(A.pos, n + m, q);
                        A.gid[n + m] = A.gid[i];
                        A.img_src[m] = (int)i;
                        A.img_shift[m] = (unsigned char)sv;
                    } else {
                        ovf = 1u;
                    }
                    ++m;
                }
            }
        }
        cluster.sync();
        // 5. cell of every particle and image, slot from the cell's counter
        const long m_img = min((long)*A.tot, A.img_cap);
        const long nt = n + m_img;
        for (long k = gt; k < nt; k += GT) {
            const T4 r = ldc4(A.pos, k);
            const unsigned int c = (unsigned int)A.G.cell(r.x, r.y, r.z, bad);
            A.cell_of[k] = c;
            A.slot[k] = atomicAdd(&A.cnt[c], 1u);
        }
        cluster.sync();
        // 6. cell starts (first CTA)
        if (rank == 0) cta_scan(A.cnt, A.cstart, A.ncells + 1, A.tot + 1, wsum);
        cluster.sync();
        // 7. scatter to the unordered slot
        for (long k = gt; k < nt; k += GT) A.sorted_tmp[A.cstart[A.cell_of[k]] + A.slot[k]] = (int)k;
        cluster.sync();
        // 8. in-cell order by index (one warp per cell), then the cell-ordered position copy
        {
            const long warp = gt >> 5, nw = GT >> 5;
            const int lane = threadIdx.x & 31;
            for (long c = warp; c < A.ncells; c += nw) {
                const unsigned int b0 = A.cstart[c], e0 = A.cstart[c + 1], cn = e0 - b0;
                warp_cell_order(A.sorted_tmp + b0, A.sorted + b0, cn, cell_sort_buf[threadIdx.x >> 5], CL_SORT_CAP);
                __syncwarp();
                for (unsigned int a = lane; a < cn; a += 32) {
                    const int v = A.sorted[b0 + a];
                    T4 r = ldc4(A.pos, v);
                    r.w = idx_bits<T>(v);
                    st4(A.pcs, b0 + a, r);
                }
            }
        }
        cluster.sync();
        // 9. forces: q lanes per particle walk the 27 cells through the cell-ordered
        // copy (three cells of a row are one contiguous range), their sums meet by
        // shuffles; then v += h f and the energies
        double pe = 0, vir = 0, ke = 0;
        {
            const int q = A.q;
            const long per = GT / q;
            const long iters = (n + per - 1) / per;  // the same for every thread (whole warps shuffle)
            const int sub = (int)(gt % q);
            for (long it = 0; it < iters; ++it) {
                const long i = gt / q + it * per;
                const bool active = i < n;
                const T4 xi = ldc4(A.pos, active ? i : 0);
                const int c = active ? (int)A.cell_of[i] : 0;
                const int c0 = c % A.G.gs[0], c1 = (c / A.G.gs[0]) % A.G.gs[1], c2 = c / (A.G.gs[0] * A.G.gs[1]);
                T fx = 0, fy = 0, fz = 0, e = 0, w = 0;
                for (int r9 = 0; r9 < 9 && active; ++r9) {
                    const int y = c1 + r9 % 3 - 1, z = c2 + r9 / 3 - 1;
                    if (y < 0 || z < 0 || y >= A.G.gs[1] || z >= A.G.gs[2]) continue;
                    const int xa = max(c0 - 1, 0), xb = min(c0 + 1, A.G.gs[0] - 1);
                    const long rb = (long)A.G.gs[0] * (y + (long)A.G.gs[1] * z);
                    const unsigned int ka = A.cstart[rb + xa], kb = A.cstart[rb + xb + 1];
#pragma unroll 2
                    for (unsigned int k = ka + sub; k < kb; k += q) {
                        const T4 xq = ldc4(A.pcs, k);
                        if (idx_of<T>(xq.w) == (int)i) continue;
                        const T dx = xi.x - xq.x, dy2 = xi.y - xq.y, dz2 = xi.z - xq.z;
                        const T r2 = dist2(dx, dy2, dz2);
                        if (r2 < A.P.rc2) lj_acc(A.P, r2, dx, dy2, dz2, fx, fy, fz, e, w);
                    }
                }
                for (int o = 1; o < q; o <<= 1) {
                    fx += __shfl_xor_sync(0xffffffffu, fx, o);
                    fy += __shfl_xor_sync(0xffffffffu, fy, o);
                    fz += __shfl_xor_sync(0xffffffffu, fz, o);
                    e += __shfl_xor_sync(0xffffffffu, e, o);
                    w += __shfl_xor_sync(0xffffffffu, w, o);
                }
                if (active && sub == 0) {
                    A.f[i] = fx;
                    A.f[A.cap + i] = fy;
                    A.f[2 * A.cap + i] = fz;
                    pe += 0.5 * (double)e;
                    vir += 0.5 * (double)w;
                    const T vx = A.v[i] + A.half * fx;
                    const T vy = A.v[A.cap + i] + A.half * fy;
                    const T vz = A.v[2 * A.cap + i] + A.half * fz;
                    A.v[i] = vx;
                    A.v[A.cap + i] = vy;
                    A.v[2 * A.cap + i] = vz;
                    ke += 0.5 * A.mass * ((double)vx * vx + (double)vy * vy + (double)vz * vz);
                }
            }
        }
        pe = block_sum<double, CL_THREADS>(pe);
        vir = block_sum<double, CL_THREADS>(vir);
        ke = block_sum<double, CL_THREADS>(ke);
        if (threadIdx.x == 0) {
            A.part[3 * rank] = pe;
            A.part[3 * rank + 1] = vir;
            A.part[3 * rank + 2] = ke;
        }
        cluster.sync();
        // 10. the step's energies, CTA partials in a fixed order
        if (rank == 0 && threadIdx.x == 0) {
            double a = 0, b = 0, c = 0;
            for (int r = 0; r < nct; ++r) {
                a += A.part[3 * r + 2];
                b += A.part[3 * r];
                c += A.part[3 * r + 1];
            }
            double* Es = A.E + 4 * (long)s;
            Es[0] = a;
            Es[1] = b;
            Es[2] = c;
            Es[3] = 1.0;
        }
        // the next step rewrites part only after several cluster barriers
    }
    if (bad) atomicOr(A.err, ERR_CELL_RANGE);
    if (ovf) atomicOr(A.err, ERR_IMG_OVERFLOW);
}

template <class T> static int md_run_cluster_t(pd_md md, int steps, cudaStream_t st, double* E) {
    pd_vd h = md->h;
    pd_cl cl = md->cl;
    const long n = h->n_real;
    Prop& V = h->props[md->mp.vel_prop];
    Prop& F = h->props[md->mp.force_prop];
    // image room: the last count with a margin
    const long img_cap = h->n_img + h->n_img / 2 + 1024;
    PD_TRY(ensure_capacity(h, n + img_cap + 1, st));
    const long nt = n + img_cap;
    const long nc = cl->ncells;
    PD_TRY(cl->cell_cnt.ensure(sizeof(unsigned int) * (nc + 1)));
    PD_TRY(cl->cell_start.ensure(sizeof(unsigned int) * (nc + 1)));
    PD_TRY(cl->cell_of.ensure(sizeof(unsigned int) * nt));
    PD_TRY(cl->slot.ensure(sizeof(unsigned int) * nt));
    PD_TRY(cl->sorted.ensure(sizeof(int) * nt));
    PD_TRY(cl->sorted_tmp.ensure(sizeof(int) * nt));
    PD_TRY(h->img_cnt.ensure(sizeof(unsigned int) * (n + 1)));
    PD_TRY(h->img_start.ensure(sizeof(unsigned int) * (n + 1)));
    PD_TRY(h->img_src.ensure(sizeof(int) * img_cap));
    PD_TRY(h->img_shift.ensure(img_cap));
    PD_TRY(md->kpart.ensure(sizeof(double) * 3 * CL_CTAS + sizeof(unsigned int) * 4));
    PD_TRY(md->E.ensure(sizeof(double) * 4 * (steps + 1)));
    PD_TRY(ghost_boxes_upload(h, st));
    ClArgs<T> A;
    memset(&A, 0, sizeof(A));
    A.pos = (typename V4<T>::type*)h->pos;
    A.gid = h->gid;
    A.img_src = h->img_src.as<int>();
    A.img_shift = h->img_shift.as<unsigned char>();
    A.v = (T*)V.d;
    A.f = (T*)F.d;
    A.cap = h->cap;
    A.n = n;
    A.img_cap = img_cap;
    for (int d = 0; d < 3; ++d) {
        A.lo[d] = (T)h->lo[d];
        A.hi[d] = (T)h->hi[d];
        A.per[d] = h->bc[d] == PD_PERIODIC;
        A.G.lo[d] = (T)cl->box_lo[d];
        A.G.sp[d] = (T)cl->spacing[d];
        A.G.gs[d] = cl->gs[d];
    }
    A.G.pad = cl->pad;
    A.boxes = h->boxes.as<BoxSet<T>>();
    A.shifts = h->shifts.as<T>();
    A.ncells = nc;
    A.cnt = cl->cell_cnt.as<unsigned int>();
    A.cstart = cl->cell_start.as<unsigned int>();
    A.cell_of = cl->cell_of.as<unsigned int>();
    A.slot = cl->slot.as<unsigned int>();
    A.img_cnt = h->img_cnt.as<unsigned int>();
    A.img_start = h->img_start.as<unsigned int>();
    A.sorted = cl->sorted.as<int>();
    A.sorted_tmp = cl->sorted_tmp.as<int>();
    PD_TRY(h->tmp.ensure((size_t)nt * h->pos_bytes));
    A.pcs = h->tmp.as<typename V4<T>::type>();

    A.P.eps24 = (T)(24.0 * md->lj.eps);
    A.P.eps4 = (T)(4.0 * md->lj.eps);
    A.P.sig2 = (T)(md->lj.sigma * md->lj.sigma);
    const T rc = (T)md->lj.r_cut;
    A.P.rc2 = rc * rc;
    A.half = (T)(0.5 * md->mp.dt / md->mp.mass);
    A.dt = (T)md->mp.dt;
    A.mass = md->mp.mass;
    A.part = md->kpart.as<double>();
    A.tot = reinterpret_cast<unsigned int*>(A.part + 3 * CL_CTAS);
    A.E = md->E.as<double>();
    A.steps = steps;
    A.err = &h->ctrl->err;
    // one cluster of 16 CTAs (one per SM) where the GPU can place it, else 8
    static int nct = 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1] = {};
    cfg.blockDim = dim3(CL_THREADS, 1, 1);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    if (nct == 0) {
        nct = 8;
        if (cudaFuncSetAttribute(k_md_cluster<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cfg.gridDim = dim3(CL_CTAS, 1, 1);
            attr[0].val.clusterDim.x = CL_CTAS;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            int nclusters = 0;
            if (cudaOccupancyMaxActiveClusters(&nclusters, k_md_cluster<T>, &cfg) == cudaSuccess && nclusters >= 1)
                nct = CL_CTAS;
        }
        cudaGetLastError();
    }
    {
        const long GT = (long)nct * CL_THREADS;
        int q = 1;
        while (q < 32 && (long)(2 * q) * n <= GT) q <<= 1;
        A.q = q;
    }
    cfg.gridDim = dim3(nct, 1, 1);
    attr[0].val.clusterDim.x = nct;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    PD_CUDA(cudaLaunchKernelEx(&cfg, k_md_cluster<T>, A));
    __atomic_fetch_add(&g_launches, 1ull, __ATOMIC_RELAXED);
    md->cluster_ctas = nct;
    unsigned int tot = 0;
    PD_CUDA(cudaMemcpyAsync(&tot, A.tot, sizeof(unsigned int), cudaMemcpyDeviceToHost, st));
    if (E && steps > 0) PD_CUDA(cudaMemcpyAsync(E, md->E.p, sizeof(double) * 4 * steps, cudaMemcpyDeviceToHost, st));
    PD_TRY(read_ctrl(h, st));  // synchronises the stream
    PD_TRY(take_timeout(h, "pd_md_run", st));
    if (h->ctrl_h->err & (ERR_IMG_OVERFLOW | ERR_CELL_RANGE)) {
        set_error("pd_md_run: cluster step overflow or particle outside the cell grid (err=0x%x)", h->ctrl_h->err);
        return PD_EOVERFLOW;
    }
    // the vector holds the last step's images (generation order) with their records;
    // their properties are refreshed from the sources
    h->n_img = tot;
    h->n_total = n + tot;
    h->img_valid = true;
    h->img_gen_order = true;
    PD_TRY(ghost_replay(h, ~0ul, false, nullptr, h->n_img, st));
    md->steps += steps;
    md->builds += steps;
    h->epoch++;
    return PD_OK;
}

// ---------------------------------------------------------------------------
// The same run on the whole GPU: one cooperative launch of clusters of eight CTAs, one
// grid barrier a step.  The cell list is a bucket of `bcap` records per cell, written by
// the drift itself: whoever computes a particle's force also makes its closing kick, the
// next step's kick and drift, and puts the drifted record and its periodic images into the
// buckets of the next step (two sets of buckets and three of counts, so that a step reads
// one set, fills the next and clears the third).  No scan, scatter or separate ordering
// is left: a CTA that works on a cell stages the 27 buckets around it in shared memory and
// orders each by its key there -- the particle's index, or n + 27 source + shift for an
// image, the order in which ghost_get numbers them -- so the sums do not depend on the
// order in which the buckets were filled.
// Bound by latency: bucket counts, records, pair loop and barrier follow one another.
// Against the ten phases on one cluster of 16 SMs, FP64: 80.6 -> 20.4 us a step for 4,096
// particles, 40 -> 17 for 512, 897 -> 163 for 64,000.
// A bucket that overflows (an uneven system) stops the run before that step; positions
// alternate between two arrays, so the state of the step before is whole, and the
// one-cluster kernel goes on from it.
static constexpr int CB_THREADS = 256;
static constexpr int CB_CLUSTER = 8;
static constexpr int CB_MAXCAP = 128;  // records per bucket at most

template <class T> struct CbArgs {
    typename V4<T>::type* x[2];  // positions of the even and of the odd steps
    T* v;
    T* f;
    long cap, n;
    T lo[3], hi[3];
    int per[3];
    const BoxSet<T>* boxes;
    const T* shifts;
    Grid<T> G;
    long ncells;
    int first[3], num[3];  // cells that can hold particles of the domain
    long units;
    unsigned int* cnt;             // [3][ncells]
    typename V4<T>::type* bk[2];   // [ncells][bcap]
    int bcap;
    LJP<T> P;
    T half, dt;
    double mass;
    double* part;  // [2][CTAs][3]: potential energy, virial, kinetic energy
    double* E;     // [steps][4]
    int steps;
    unsigned int* bar;   // arrivals at the grid barrier
    unsigned int* over;  // 0x7fffffff - (first step with an overflowing bucket), 0: none
    unsigned int* done;
    unsigned int* err;
};

// data written earlier in the launch by other CTAs: from L2
__device__ __forceinline__ double4 ldcg4(const double4* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldcg(q), b = __ldcg(q + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 ldcg4(const float4* p) { return __ldcg(p); }

// grid barrier: the clusters meet by their own barrier, one thread of each on the counter.
// Every CTA of the cooperative launch is resident, so the wait ends; it is bounded all the
// same (about a second; the error bit then voids the run).  False, for the whole CTA, once
// a wait has given up.
__device__ __forceinline__ bool grid_barrier(cg::cluster_group& cl, unsigned int* bar, unsigned int target,
                                             unsigned int* err) {
    cl.sync();
    if (cl.block_rank() == 0 && threadIdx.x == 0) {
        // the cluster's writes before cl.sync() are this thread's to release (cumulativity), the
        // other clusters' its to acquire for the cluster
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned int seen = 0, it = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
        } while (seen < target && ++it < (1u << 21));
        if (seen < target) atomicOr(err, ERR_TIMEOUT);
    }
    cl.sync();
    return __syncthreads_or((__ldcg(err) & ERR_TIMEOUT) ? 1 : 0) == 0;
}

template <class T>
__device__ __forceinline__ void cb_insert(const CbArgs<T>& A, typename V4<T>::type r, int key, int step,
                                          unsigned int& bad) {
    const unsigned int c = (unsigned int)A.G.cell(r.x, r.y, r.z, bad);
    const unsigned int k = atomicAdd(A.cnt + (long)(step % 3) * A.ncells + c, 1u);
    if (k < (unsigned int)A.bcap) {
        r.w = idx_bits<T>(key);
        st4(A.bk[step & 1] + (long)c * A.bcap, k, r);
    } else {
        atomicMax(A.over, 0x7fffffffu - (unsigned int)step);
    }
}

// kick and drift of particle i from its state after the step before, into the buckets of
// `step`; L lanes share the particle (the images' boxes are dealt out over them)
template <class T>
__device__ __forceinline__ void cb_advance(const CbArgs<T>& A, const BoxSet<T>& B, int i, typename V4<T>::type x, T vx,
                                           T vy, T vz, T fx, T fy, T fz, int step, int sub, int L, unsigned int& bad) {
    typedef typename V4<T>::type T4;
    vx = vx + A.half * fx;
    vy = vy + A.half * fy;
    vz = vz + A.half * fz;
    x.x += A.dt * vx;
    x.y += A.dt * vy;
    x.z += A.dt * vz;
    if (A.per[0]) x.x = periodic_l(x.x, A.hi[0], A.lo[0]);
    if (A.per[1]) x.y = periodic_l(x.y, A.hi[1], A.lo[1]);
    if (A.per[2]) x.z = periodic_l(x.z, A.hi[2], A.lo[2]);
    if (sub == 0) {
        x.w = T(0);
        st4(A.x[step & 1], i, x);
        cb_insert(A, x, i, step, bad);
    }
    if (in_core(B, x.x, x.y, x.z)) return;
    for (int b = sub; b < B.nb; b += L)  // (the domain's boxes have a shift each)
        if (inside_np(B, b, x.x, x.y, x.z)) {
            const int sv = B.sv[b];
            T4 q;
            q.x = x.x - A.shifts[3 * sv];
            q.y = x.y - A.shifts[3 * sv + 1];
            q.z = x.z - A.shifts[3 * sv + 2];
            q.w = T(0);
            cb_insert(A, q, (int)A.n + 27 * i + sv, step, bad);
        }
}

template <class T>
__global__ void __launch_bounds__(CB_THREADS, 3) k_md_buckets(CbArgs<T> A) {
    typedef typename V4<T>::type T4;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char cb_raw[];
    T4* sp = reinterpret_cast<T4*>(cb_raw);  // [27 * bcap]
    __shared__ BoxSet<T> B;
    __shared__ unsigned int num[27], off[28], cellid[27];
    __shared__ int keys[CB_THREADS / 32][CB_MAXCAP];
    __shared__ double esum[3][CB_THREADS / 32];
    for (int i = threadIdx.x; i < (int)(sizeof(BoxSet<T>) / 4); i += blockDim.x)
        reinterpret_cast<int*>(&B)[i] = reinterpret_cast<const int*>(A.boxes)[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int nclusters = gridDim.x / CB_CLUSTER;
    unsigned int bad = 0, target = 0;
    // the first step's kick and drift, eight lanes a particle
    for (long t = blockIdx.x * (long)CB_THREADS + threadIdx.x; t < 8 * A.n; t += (long)gridDim.x * CB_THREADS) {
        const long i = t >> 3;
        cb_advance(A, B, (int)i, ldcg4(A.x[0] + i), __ldcg(A.v + i), __ldcg(A.v + A.cap + i), __ldcg(A.v + 2 * A.cap + i),
                   __ldcg(A.f + i), __ldcg(A.f + A.cap + i), __ldcg(A.f + 2 * A.cap + i), 1, (int)(t & 7), 8, bad);
    }
    bool alive = grid_barrier(cluster, A.bar, target += nclusters, A.err);
    int s = 1;
    for (; alive && s <= A.steps; ++s) {
        // (an overflow while filling a later step's buckets has a larger step number)
        const unsigned int ov = __ldcg(A.over);
        if (ov != 0u && (int)(0x7fffffffu - ov) <= s) break;
        for (long c = blockIdx.x * (long)CB_THREADS + threadIdx.x; c < A.ncells; c += (long)gridDim.x * CB_THREADS)
            A.cnt[(long)((s + 2) % 3) * A.ncells + c] = 0u;
        const unsigned int* cnt = A.cnt + (long)(s % 3) * A.ncells;
        const T4* bk = A.bk[s & 1];
        double pe = 0, vir = 0, ke = 0;
        for (long u = blockIdx.x; u < A.units; u += gridDim.x) {
            const int cx = A.first[0] + (int)(u % A.num[0]), cy = A.first[1] + (int)(u / A.num[0] % A.num[1]),
                      cz = A.first[2] + (int)(u / ((long)A.num[0] * A.num[1]));
            if (warp == 0) {
                unsigned int m = 0, id = 0;
                if (lane < 27) {
                    const int x = cx + lane % 3 - 1, y = cy + lane / 3 % 3 - 1, z = cz + lane / 9 - 1;
                    if (x >= 0 && y >= 0 && z >= 0 && x < A.G.gs[0] && y < A.G.gs[1] && z < A.G.gs[2]) {
                        id = (unsigned int)(x + A.G.gs[0] * (y + (long)A.G.gs[1] * z));
                        m = min(__ldcg(cnt + id), (unsigned int)A.bcap);
                    }
                }
                unsigned int inc = m;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned int y = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += y;
                }
                if (lane < 27) {
                    num[lane] = m;
                    cellid[lane] = id;
                    off[lane + 1] = inc;
                }
                if (lane == 0) off[0] = 0;
            }
            __syncthreads();
            if (num[13] == 0) {  // the same for every thread
                __syncthreads();
                continue;
            }
            // each warp: buckets into shared memory, ascending key
            for (int c = warp; c < 27; c += CB_THREADS / 32) {
                const unsigned int m = num[c], o = off[c];
                const T4* src = bk + (long)cellid[c] * A.bcap;
                if (m <= 32) {
                    T4 r;
                    int key = 0x7fffffff;
                    if (lane < (int)m) {
                        r = ldcg4(src + lane);
                        key = idx_of<T>(r.w);
                    }
                    unsigned int rank = 0;
                    for (int j = 0; j < (int)m; ++j) rank += (__shfl_sync(0xffffffffu, key, j) < key) ? 1u : 0u;
                    if (lane < (int)m) sp[o + rank] = r;
                } else {
                    int* kb = keys[warp];
                    for (unsigned int e = lane; e < m; e += 32) kb[e] = idx_of<T>(ldcg4(src + e).w);
                    __syncwarp();
                    for (unsigned int e = lane; e < m; e += 32) {
                        const int key = kb[e];
                        unsigned int rank = 0;
                        for (unsigned int j = 0; j < m; ++j) rank += kb[j] < key ? 1u : 0u;
                        sp[o + rank] = ldcg4(src + e);
                    }
                    __syncwarp();
                }
            }
            __syncthreads();
            const unsigned int oc = off[13], nc = num[13], M = off[27];
            // the domain's particles come first (smaller keys)
            const int nreal = __syncthreads_count(threadIdx.x < nc && idx_of<T>(sp[oc + threadIdx.x].w) < (int)A.n);
            int L = 32;
            while (L > 1 && L * nreal > CB_THREADS) L >>= 1;
            const int q = (int)threadIdx.x / L, sub = (int)threadIdx.x % L;
            const bool active = q < nreal;
            const unsigned int me = oc + (active ? (unsigned int)q : 0u);
            const T4 xi = sp[me];
            T fx = 0, fy = 0, fz = 0, e = 0, w = 0;
            // (v, f) of the particle while the pairs are computed
            const int i = idx_of<T>(xi.w);
            T vx = 0, vy = 0, vz = 0;
            if (active) {
                vx = __ldcg(A.v + i) + A.half * __ldcg(A.f + i);
                vy = __ldcg(A.v + A.cap + i) + A.half * __ldcg(A.f + A.cap + i);
                vz = __ldcg(A.v + 2 * A.cap + i) + A.half * __ldcg(A.f + 2 * A.cap + i);
                for (unsigned int k = sub; k < M; k += L) {
                    const T4 xq = sp[k];
                    const T dx = xi.x - xq.x, dy = xi.y - xq.y, dz = xi.z - xq.z;
                    const T r2 = dist2(dx, dy, dz);
                    if (r2 < A.P.rc2 && k != me) lj_acc(A.P, r2, dx, dy, dz, fx, fy, fz, e, w);
                }
            }
            for (int o = 1; o < L; o <<= 1) {
                fx += __shfl_xor_sync(0xffffffffu, fx, o);
                fy += __shfl_xor_sync(0xffffffffu, fy, o);
                fz += __shfl_xor_sync(0xffffffffu, fz, o);
                e += __shfl_xor_sync(0xffffffffu, e, o);
                w += __shfl_xor_sync(0xffffffffu, w, o);
            }
            const unsigned int group = __ballot_sync(0xffffffffu, active);
            if (active) {
                vx = vx + A.half * fx;
                vy = vy + A.half * fy;
                vz = vz + A.half * fz;
                __syncwarp(group);  // every lane has read before the first one writes
                if (sub == 0) {
                    A.v[i] = vx;
                    A.v[A.cap + i] = vy;
                    A.v[2 * A.cap + i] = vz;
                    A.f[i] = fx;
                    A.f[A.cap + i] = fy;
                    A.f[2 * A.cap + i] = fz;
                    pe += 0.5 * (double)e;
                    vir += 0.5 * (double)w;
                    ke += 0.5 * A.mass * ((double)vx * vx + (double)vy * vy + (double)vz * vz);
                }
                if (s < A.steps) cb_advance(A, B, i, xi, vx, vy, vz, fx, fy, fz, s + 1, sub, L, bad);
            }
            __syncthreads();
        }
        pe = warp_sum(pe);
        vir = warp_sum(vir);
        ke = warp_sum(ke);
        if (lane == 0) {
            esum[0][warp] = pe;
            esum[1][warp] = vir;
            esum[2][warp] = ke;
        }
        __syncthreads();
        if (threadIdx.x < 3) {
            double t = 0;
            for (int k = 0; k < CB_THREADS / 32; ++k) t += esum[threadIdx.x][k];
            A.part[3 * ((long)(s & 1) * gridDim.x + blockIdx.x) + threadIdx.x] = t;
        }
        alive = grid_barrier(cluster, A.bar, target += nclusters, A.err);
        // the step's energies while the other CTAs go on, by the last CTA (of the fewest cells)
        if (blockIdx.x == gridDim.x - 1) {
            const double* pt = A.part + 3 * (long)(s & 1) * gridDim.x;
            double a = 0, b = 0, c = 0;
            for (unsigned int r = threadIdx.x; r < gridDim.x; r += CB_THREADS) {
                b += __ldcg(pt + 3 * r);
                c += __ldcg(pt + 3 * r + 1);
                a += __ldcg(pt + 3 * r + 2);
            }
            a = block_sum<double, CB_THREADS>(a);
            b = block_sum<double, CB_THREADS>(b);
            c = block_sum<double, CB_THREADS>(c);
            if (threadIdx.x == 0) {
                double* Es = A.E + 4 * (long)(s - 1);
                Es[0] = a;
                Es[1] = b;
                Es[2] = c;
                Es[3] = 1.0;
            }
        }
    }
    const int made = s - 1;
    if (made & 1)  // the positions back where the vector keeps them
        for (long i = blockIdx.x * (long)CB_THREADS + threadIdx.x; i < A.n; i += (long)gridDim.x * CB_THREADS)
            st4(A.x[0], i, ldcg4(A.x[1] + i));
    if (blockIdx.x == 0 && threadIdx.x == 0) *A.done = (unsigned int)made;
    if (bad) atomicOr(A.err, ERR_CELL_RANGE);
}

// first and number of the cells along axis d that positions of the domain fall into
template <class T> static void cb_cells(pd_vd h, pd_cl cl, int d, int& first, int& num) {
    first = 0;
    num = cl->gs[d];
    if (h->bc[d] != PD_PERIODIC) return;  // a particle may leave the box
    auto at = [&](T x) {
        const long c = (long)std::floor((x - (T)cl->box_lo[d]) / (T)cl->spacing[d]) + cl->pad;
        return (int)std::max(0L, std::min((long)cl->gs[d] - 1, c));
    };
    first = at((T)h->lo[d]);
    num = at((T)h->hi[d]) - first + 1;
}

// records per bucket for the system's mean occupancy, 0 where the buckets do not suit it
static int cb_capacity(pd_md md) {
    pd_vd h = md->h;
    pd_cl cl = md->cl;
    double inner = 1;
    for (int d = 0; d < 3; ++d) inner *= std::max(1.0, (h->hi[d] - h->lo[d]) / cl->spacing[d]);
    const double occ = (double)h->n_real / inner;
    const int cap = occ <= 10 ? 32 : (occ <= 28 ? 64 : (occ <= 64 ? 128 : 0));
    // two sets of buckets within L2
    return cap && 2.0 * (double)cl->ncells * cap * h->pos_bytes <= 96e6 ? cap : 0;
}

// steps made in buckets; *made < steps where a bucket overflowed (*over) or the GPU cannot place the launch
template <class T> static int md_run_buckets_t(pd_md md, int steps, cudaStream_t st, int* made, bool* over) {
    typedef typename V4<T>::type T4;
    pd_vd h = md->h;
    pd_cl cl = md->cl;
    const long n = h->n_real;
    *made = 0;
    const int bcap = cb_capacity(md);
    const int smem = 27 * bcap * (int)sizeof(T4);
    CbArgs<T> A;
    memset(&A, 0, sizeof(A));
    A.units = 1;
    for (int d = 0; d < 3; ++d) {
        cb_cells<T>(h, cl, d, A.first[d], A.num[d]);
        A.units *= A.num[d];
        A.lo[d] = (T)h->lo[d];
        A.hi[d] = (T)h->hi[d];
        A.per[d] = h->bc[d] == PD_PERIODIC;
        A.G.lo[d] = (T)cl->box_lo[d];
        A.G.sp[d] = (T)cl->spacing[d];
        A.G.gs[d] = cl->gs[d];
    }
    A.G.pad = cl->pad;
    PD_CUDA(cudaFuncSetAttribute(k_md_buckets<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2] = {};
    cfg.blockDim = dim3(CB_THREADS, 1, 1);
    cfg.gridDim = dim3(CB_CLUSTER, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CB_CLUSTER;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cfg.numAttrs = 1;
    int most = 0;
    if (cudaOccupancyMaxActiveClusters(&most, k_md_buckets<T>, &cfg) != cudaSuccess || most < 1) {
        cudaGetLastError();
        return PD_OK;
    }
    // a cell a CTA where that many are resident, else several
    const int nclusters = (int)std::min<long>(most, (A.units + CB_CLUSTER - 1) / CB_CLUSTER);
    const int ctas = nclusters * CB_CLUSTER;
    const size_t bk = (size_t)cl->ncells * bcap * sizeof(T4), part = sizeof(double) * 6 * (size_t)ctas;
    const size_t cnt = sizeof(unsigned int) * (3 * (size_t)cl->ncells + 4);
    PD_TRY(md->buckets.ensure(2 * bk + part + cnt));
    PD_TRY(h->tmp.ensure((size_t)n * sizeof(T4)));
    PD_TRY(md->E.ensure(sizeof(double) * 4 * (steps + 1)));
    PD_TRY(ghost_boxes_upload(h, st));
    const Prop& V = h->props[md->mp.vel_prop];
    const Prop& F = h->props[md->mp.force_prop];
    char* base = md->buckets.as<char>();
    A.x[0] = (T4*)h->pos;
    A.x[1] = h->tmp.as<T4>();
    A.v = (T*)V.d;
    A.f = (T*)F.d;
    A.cap = h->cap;
    A.n = n;
    A.boxes = h->boxes.as<BoxSet<T>>();
    A.shifts = h->shifts.as<T>();
    A.ncells = cl->ncells;
    A.bk[0] = (T4*)base;
    A.bk[1] = (T4*)(base + bk);
    A.part = (double*)(base + 2 * bk);
    A.cnt = (unsigned int*)(base + 2 * bk + part);
    A.bar = A.cnt + 3 * cl->ncells;
    A.over = A.bar + 1;
    A.bcap = bcap;
    A.P.eps24 = (T)(24.0 * md->lj.eps);
    A.P.eps4 = (T)(4.0 * md->lj.eps);
    A.P.sig2 = (T)(md->lj.sigma * md->lj.sigma);
    const T rc = (T)md->lj.r_cut;
    A.P.rc2 = rc * rc;
    A.half = (T)(0.5 * md->mp.dt / md->mp.mass);
    A.dt = (T)md->mp.dt;
    A.mass = md->mp.mass;
    A.E = md->E.as<double>();
    A.steps = steps;
    A.done = &h->ctrl->run_done;
    A.err = &h->ctrl->err;
    PD_CUDA(cudaMemsetAsync(A.cnt, 0, cnt, st));
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.numAttrs = 2;
    if (cudaLaunchKernelEx(&cfg, k_md_buckets<T>, A) != cudaSuccess) {
        cudaGetLastError();
        return PD_OK;
    }
    __atomic_fetch_add(&g_launches, 1ull, __ATOMIC_RELAXED);
    md->cluster_ctas = CB_CLUSTER;
    // the last step's images with their properties; its read-back brings the step count too
    h->n_total = n;
    PD_TRY(ghost_generate(h, 0, true, st));
    if (h->nbox == 0) PD_TRY(read_ctrl(h, st));
    PD_TRY(take_timeout(h, "pd_md_run", st));
    if (h->ctrl_h->err & ERR_CELL_RANGE) {
        set_error("pd_md_run: a particle outside the cell grid (err=0x%x)", h->ctrl_h->err);
        return PD_EOVERFLOW;
    }
    *made = (int)h->ctrl_h->run_done;
    *over = *made < steps;
    md->steps += *made;
    md->builds += *made;
    md->bucket_steps += *made;
    h->epoch++;
    return PD_OK;
}

bool md_cluster_eligible(pd_md md) {
    pd_vd h = md->h;
    return md->mp.use_cell_list && md->physics == 0 && !md->mixed && !md->timing && md->cl && h->n_real > 0 &&
           h->n_real <= CL_MAXN && md->cl->pad == 1 && md->cl->ncells <= 4L * CL_MAXN;
}

// Steps in buckets as long as they hold the particles.  After an overflow 32 steps on one
// cluster, then buckets again; twice as many each time that the buckets did not last as long, so that a
// system too uneven for them loses a launch in thousands of steps and one that was crowded for
// a while returns to them.
int md_run_cluster(pd_md md, int steps, cudaStream_t st, double* E) {
    if (!md->ready) {
        PD_TRY(md_rebuild(md, st));
        PD_TRY(md_forces(md, st));
        md->ready = true;
        PD_TRY(read_ctrl(md->h, st));
        md->h->n_img = md->h->ctrl_h->n_img;
    }
    const bool f64 = md->h->dtype == PD_F64;
    bool buckets = cb_capacity(md) != 0;
    for (int s = 0; s < steps;) {
        double* Es = E ? E + 4 * (long)s : nullptr;
        if (buckets && md->bucket_left == 0) {
            int made = 0;
            bool over = false;
            PD_TRY(f64 ? md_run_buckets_t<double>(md, steps - s, st, &made, &over)
                       : md_run_buckets_t<float>(md, steps - s, st, &made, &over));
            if (E && made > 0) {
                PD_CUDA(cudaMemcpyAsync(Es, md->E.p, sizeof(double) * 4 * made, cudaMemcpyDeviceToHost, st));
                PD_CUDA(cudaStreamSynchronize(st));
            }
            s += made;
            buckets = over || s == steps;  // else the GPU cannot place the launch
            if (over) {
                md->bucket_wait = made > md->bucket_wait ? 32 : std::min(2 * std::max(md->bucket_wait, 16L), 4096L);
                md->bucket_left = md->bucket_wait;
            }
            continue;
        }
        const int part = buckets ? (int)std::min<long>(steps - s, md->bucket_left) : steps - s;
        PD_TRY(f64 ? md_run_cluster_t<double>(md, part, st, Es) : md_run_cluster_t<float>(md, part, st, Es));
        s += part;
        if (buckets) md->bucket_left -= part;
    }
    return PD_OK;
}

}  // namespace pd
