// pd_ghost.cu -- ghost_get on one GPU: periodic images of the real particles.
//
// The reference (one process) runs num_shift_ghost_each_part -> scan ->
// shift_ghost_each_part over the local ghost boxes sorted by shift id
// (vector_dist_comm_util_funcs.cuh:247-304, vector_dist_cuda_funcs.cuh:157-233),
// and with SKIP_LABELLING replays the stored (particle, shift) list
// (process_ghost_particles_local, :133-155).  Here the positions are read in one
// pass with the box list resident in device memory, the total stays on the
// device (the control block) so the image build can also run without a host
// round trip, and image records are kept for the replay.
#include <algorithm>

#include "pd_device.cuh"
#include "pd_internal.cuh"
#include "pd_ghost_dev.cuh"

namespace pd {

struct PropCopy {
    char* d[16];
    int esize[16];
    int ncomp[16];
    int n;
    long cap;
};

__device__ __forceinline__ void copy_props(const PropCopy& pc, long from, long to) {
    for (int p = 0; p < pc.n; ++p) {
        char* base = pc.d[p];
        if (pc.esize[p] == 8) {
            for (int c = 0; c < pc.ncomp[p]; ++c) {
                long long* a = reinterpret_cast<long long*>(base) + (long)c * pc.cap;
                a[to] = a[from];
            }
        } else {
            for (int c = 0; c < pc.ncomp[p]; ++c) {
                int* a = reinterpret_cast<int*>(base) + (long)c * pc.cap;
                a[to] = a[from];
            }
        }
    }
}

// num_shift_ghost_each_part
template <class T>
__global__ void k_ghost_count(const typename V4<T>::type* __restrict__ pos, long n, const BoxSet<T>* __restrict__ Bp,
                              unsigned int* __restrict__ cnt) {
    __shared__ BoxSet<T> B;
    for (int i = threadIdx.x; i < (int)(sizeof(BoxSet<T>) / 4); i += blockDim.x)
        reinterpret_cast<int*>(&B)[i] = reinterpret_cast<const int*>(Bp)[i];
    __syncthreads();
    for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < n; p += (long)gridDim.x * blockDim.x) {
        typename V4<T>::type r = ld4(pos, p);
        unsigned int c = 0;
        int old = -1;
        const int nb = in_core(B, r.x, r.y, r.z) ? 0 : B.nb;
        for (int i = 0; i < nb; ++i) {
            int s = B.sv[i];
            if (inside_np(B, i, r.x, r.y, r.z) && s != old) {
                old = s;
                c++;
            }
        }
        cnt[p] = c;
    }
}

// num_shift_ghost_each_part, scan and shift_ghost_each_part as two kernels that read the
// positions once.  k_ghost_find tests every particle (most lie in the core and have no
// image) and leaves each tile's images as a list of (particle within the tile, box),
// particle-major with ascending boxes, in a region of `list` taken with one atomic; the
// regions lie in any order.  k_ghost_write gets the images of the tiles before its own
// from the tile counts (tile_before) and writes one image a thread: consecutive slots, coalesced, the
// images of a particle in flight together.  Image j of particle p comes to slot
// n + start(p) + j.  Measured against count, scan (three kernels) and write, which read
// every record twice and wrote a particle's images one after the other: see
// ghost_generate.
static constexpr int GM_BLOCK = 256;
template <class T, int ITEMS>
__global__ void __launch_bounds__(GM_BLOCK) k_ghost_find(const typename V4<T>::type* __restrict__ pos, long n,
                                                         const BoxSet<T>* __restrict__ Bp, unsigned int cap_list,
                                                         unsigned int* __restrict__ list,
                                                         unsigned int* __restrict__ taken, uint2* __restrict__ tiles,
                                                         unsigned int* __restrict__ cnt_t) {
    constexpr int NW = GM_BLOCK / 32, NC = ITEMS * NW;
    static_assert(NC <= 32, "one count a lane in the tile's scan");
    __shared__ BoxSet<T> B;
    __shared__ unsigned int cnt[32], sh_base;
    for (int i = threadIdx.x; i < (int)(sizeof(BoxSet<T>) / 4); i += blockDim.x)
        reinterpret_cast<int*>(&B)[i] = reinterpret_cast<const int*>(Bp)[i];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long base = (long)blockIdx.x * (GM_BLOCK * ITEMS) + threadIdx.x;
    typename V4<T>::type r[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k)
        if (base + (long)k * GM_BLOCK < n) r[k] = ld4(pos, base + (long)k * GM_BLOCK);
    __syncthreads();
    unsigned long long hit[ITEMS];  // bit i: an image through box i
    unsigned int before[ITEMS];     // images of the lanes before
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        hit[k] = 0;
        if (base + (long)k * GM_BLOCK < n && !in_core(B, r[k].x, r[k].y, r[k].z)) {
            int old = -1;
            for (int i = 0; i < B.nb; ++i)
                if (inside_np(B, i, r[k].x, r[k].y, r[k].z) && B.sv[i] != old) {
                    old = B.sv[i];
                    hit[k] |= 1ull << i;
                }
        }
        const unsigned int c = __popcll(hit[k]);
        unsigned int x = 0;
        if (__any_sync(0xffffffffu, c != 0)) {
            x = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
        }
        before[k] = x - c;
        if (lane == 31) cnt[k * NW + w] = x;
    }
    __syncthreads();
    if (w == 0) {
        const unsigned int v = lane < NC ? cnt[lane] : 0u;
        unsigned int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        cnt[lane] = x - v;
        if (lane == 31) {
            sh_base = x ? atomicAdd(taken, x) : 0u;
            tiles[blockIdx.x] = make_uint2(x, sh_base);
            cnt_t[blockIdx.x] = x;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        unsigned int j = sh_base + cnt[k * NW + w] + before[k];
        for (unsigned long long h = hit[k]; h; h &= h - 1, ++j)
            if (j < cap_list)
                list[j] = ((unsigned int)(k * GM_BLOCK) + threadIdx.x) << 8 | (unsigned int)(__ffsll((long long)h) - 1);
    }
}

template <class T>
__global__ void __launch_bounds__(GM_BLOCK) k_ghost_write(typename V4<T>::type* __restrict__ pos,
                                                          int* __restrict__ gid, long n, int tile_n,
                                                          const BoxSet<T>* __restrict__ B,
                                                          const T* __restrict__ shifts,
                                                          const unsigned int* __restrict__ list, unsigned int cap_list,
                                                          const uint2* __restrict__ tiles,
                                                          const unsigned int* __restrict__ cnt, bool scanned,
                                                          int* __restrict__ src,
                                                          unsigned char* __restrict__ shf, long img_cap, long cap,
                                                          PropCopy pc, unsigned int* __restrict__ n_img,
                                                          unsigned int* __restrict__ err) {
    const unsigned int t = blockIdx.x;
    const long m0 = tile_before<GM_BLOCK>(cnt, t, scanned);
    const uint2 mine = tiles[t];
    if (threadIdx.x == 0 && t == gridDim.x - 1) *n_img = (unsigned int)m0 + mine.x;
    for (unsigned int j = threadIdx.x; j < mine.x; j += GM_BLOCK) {
        const long m = m0 + j;
        if (m >= img_cap || n + m >= cap || mine.y + j >= cap_list) {
            atomicOr(err, ERR_IMG_OVERFLOW);
            continue;
        }
        const unsigned int e = list[mine.y + j];
        const long p = (long)t * tile_n + (e >> 8);
        const int sv = B->sv[e & 255u];
        typename V4<T>::type q = ld4(pos, p);
        q.x -= shifts[3 * sv];
        q.y -= shifts[3 * sv + 1];
        q.z -= shifts[3 * sv + 2];
        st4(pos, n + m, q);
        gid[n + m] = gid[p];
        src[m] = (int)p;
        shf[m] = (unsigned char)sv;
        copy_props(pc, p, n + m);
    }
}

// process_ghost_particles_local: replay the stored image list
template <class T>
__global__ void k_ghost_replay(typename V4<T>::type* __restrict__ pos, long n, const int* __restrict__ src,
                               const unsigned char* __restrict__ shf, const T* __restrict__ shifts,
                               const unsigned int* __restrict__ n_img_dev, long n_img_bound, int with_pos,
                               PropCopy pc) {
    long m_n = n_img_dev ? (long)*n_img_dev : n_img_bound;
    if (m_n > n_img_bound) m_n = n_img_bound;
    for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < m_n; m += (long)gridDim.x * blockDim.x) {
        int p = src[m];
        if (with_pos) {
            int s = shf[m];
            typename V4<T>::type r = ld4(pos, p);
            r.x -= shifts[3 * s];
            r.y -= shifts[3 * s + 1];
            r.z -= shifts[3 * s + 2];
            st4(pos, n + m, r);
        }
        if (pc.n) copy_props(pc, p, n + m);
    }
}

// ghost_put<op, prp...> on one process (vector_dist_comm.hpp:2086-2182, the local
// part merge_prp_v): every image's value is merged onto its source in image
// order -- the images of a source are consecutive (generation order), so the thread
// of a source's first image applies them in that order and the result is deterministic.
template <class E>
__global__ void k_ghost_put(E* __restrict__ a, long cap, int ncomp, long n, const int* __restrict__ src, long n_img,
                            int op) {
    for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < n_img; m += (long)gridDim.x * blockDim.x) {
        const int p = src[m];
        if (m > 0 && src[m - 1] == p) continue;
        for (int c = 0; c < ncomp; ++c) {
            E* col = a + (long)c * cap;
            E acc = col[p];
            for (long j = m; j < n_img && src[j] == p; ++j) {
                const E v = col[n + j];
                acc = op == PD_PUT_ADD ? acc + v : (op == PD_PUT_MAX ? (v > acc ? v : acc) : v);
            }
            col[p] = acc;
        }
    }
}

static PropCopy make_copy(pd_vd h, unsigned long mask) {
    PropCopy pc;
    memset(&pc, 0, sizeof(pc));
    pc.cap = h->cap;
    for (size_t p = 0; p < h->props.size(); ++p) {
        if (!(mask & (1ul << p))) continue;
        pc.d[pc.n] = h->props[p].d;
        pc.esize[pc.n] = h->props[p].esize;
        pc.ncomp[pc.n] = h->props[p].ncomp;
        pc.n++;
    }
    return pc;
}

// Local periodic ghost boxes of one sub-domain equal to the domain, sorted by
// shift id: the replica of the domain shifted by -L*c (applyBC,
// ie_loc_ghost.hpp:145-200) enlarged by the ghost and intersected with the
// domain (create_loc_ghost_ibox, :102-143); shift vectors -L*c indexed by
// c.lin() (shift_vect_converter.hpp:36-66).
template <class T> static int domain_boxes(pd_vd h, BoxSet<T>& B, T* shifts) {
    T lo[3], hi[3], g[3];
    for (int d = 0; d < 3; ++d) {
        lo[d] = (T)h->lo[d];
        hi[d] = (T)h->hi[d];
        g[d] = (T)h->g[d];
    }
    B.nb = 0;
    B.core = 0;
    for (int l = 0; l < 27; ++l) {
        int c[3] = {l % 3 - 1, (l / 3) % 3 - 1, l / 9 - 1};
        for (int d = 0; d < 3; ++d)
            shifts[3 * l + d] = c[d] == 1 ? -(hi[d] - lo[d]) : (c[d] == -1 ? (hi[d] - lo[d]) : T(0));
        if (c[0] == 0 && c[1] == 0 && c[2] == 0) continue;
        bool ok = true;
        for (int d = 0; d < 3; ++d)
            if (c[d] != 0 && h->bc[d] != PD_PERIODIC) ok = false;
        if (!ok) continue;
        bool empty = false;
        T bl[3], bu[3];
        for (int d = 0; d < 3; ++d) {
            T sh = c[d] == 1 ? (-hi[d] + lo[d]) : (c[d] == -1 ? (hi[d] - lo[d]) : T(0));
            T el = (lo[d] + sh) + (-g[d]), eu = (hi[d] + sh) + g[d];
            bl[d] = lo[d] > el ? lo[d] : el;
            bu[d] = hi[d] < eu ? hi[d] : eu;
            if (bl[d] >= bu[d]) empty = true;
        }
        if (empty) continue;
        for (int d = 0; d < 3; ++d) {
            B.lo[B.nb][d] = bl[d];
            B.hi[B.nb][d] = bu[d];
        }
        B.sv[B.nb] = l;
        B.nb++;
    }
    return B.nb;
}

// The core of a box set inside the domain: on each axis, between the highest box
// upper edge at or below the middle and the lowest box lower edge at or above it
// (boxes across the middle leave that axis open).  Kept only if it is not empty and
// every box misses it on some axis, so that no point of it lies in a box.
template <class T> static void box_core(pd_vd h, BoxSet<T>& B) {
    B.core = 0;
    if (B.nb <= 0) return;
    for (int d = 0; d < 3; ++d) {
        const T lo = (T)h->lo[d], hi = (T)h->hi[d], mid = lo + (hi - lo) / T(2);
        T cl = lo, ch = hi;
        for (int i = 0; i < B.nb; ++i) {
            if (B.hi[i][d] <= mid && B.hi[i][d] > cl) cl = B.hi[i][d];
            if (B.lo[i][d] >= mid && B.lo[i][d] < ch) ch = B.lo[i][d];
        }
        if (!(cl < ch)) return;
        B.clo[d] = cl;
        B.chi[d] = ch;
    }
    for (int i = 0; i < B.nb; ++i) {
        bool misses = false;
        for (int d = 0; d < 3; ++d)
            if (B.hi[i][d] <= B.clo[d] || B.lo[i][d] >= B.chi[d]) misses = true;
        if (!misses) return;
    }
    B.core = 1;
}

template <class T> static int upload_boxes_t(pd_vd h, const BoxSet<T>& B_in, const T* shifts, int n_shifts,
                                             cudaStream_t st) {
    BoxSet<T> B = B_in;
    box_core(h, B);
    PD_TRY(h->boxes.ensure(sizeof(BoxSet<T>)));
    PD_TRY(h->shifts.ensure(sizeof(T) * 3 * (n_shifts > 27 ? n_shifts : 27)));
    PD_CUDA(cudaMemcpyAsync(h->boxes.p, &B, sizeof(BoxSet<T>), cudaMemcpyHostToDevice, st));
    PD_CUDA(cudaMemcpyAsync(h->shifts.p, shifts, sizeof(T) * 3 * n_shifts, cudaMemcpyHostToDevice, st));
    PD_CUDA(cudaStreamSynchronize(st));  // host staging buffers are stack locals
    h->nbox = B.nb;
    h->boxes_dom = false;
    return PD_OK;
}

// the domain's ghost boxes in device memory: uploaded once, and again after a call with
// the caller's own boxes (box, ghost and boundary conditions are fixed at creation)
int ghost_boxes_upload(pd_vd h, cudaStream_t st) {
    if (h->boxes_dom) return PD_OK;
    if (h->dtype == PD_F64) {
        BoxSet<double> B;
        double sh[81];
        domain_boxes(h, B, sh);
        PD_TRY(upload_boxes_t(h, B, sh, 27, st));
    } else {
        BoxSet<float> B;
        float sh[81];
        domain_boxes(h, B, sh);
        PD_TRY(upload_boxes_t(h, B, sh, 27, st));
    }
    h->boxes_dom = true;
    return PD_OK;
}

// domain ghost boxes and shift vectors of an FP64 vector into caller-owned host
// memory (no copy); the caller uploads them to h->boxes / h->shifts
int ghost_boxes_host(pd_vd h, BoxSet<double>* B, double* shifts27) {
    if (h->dtype != PD_F64) return PD_EINVAL;
    domain_boxes(h, *B, shifts27);
    return PD_OK;
}

// images into the slots after the real particles, at most m_cap
static int ghost_make(pd_vd h, long m_cap, cudaStream_t st) {
    const long n = h->n_real;
    PD_TRY(h->img_src.ensure(sizeof(int) * (m_cap > 0 ? m_cap : 1)));
    PD_TRY(h->img_shift.ensure(m_cap > 0 ? m_cap : 1));
    if (n <= 0 || h->nbox == 0) {
        PD_CUDA(cudaMemsetAsync(&h->ctrl->n_img, 0, sizeof(unsigned int), st));
        return PD_OK;
    }
    const PropCopy pc = make_copy(h, ~0ul);
    // four particles a thread, one where that would leave SMs without a tile
    const int items = n >= 148L * GM_BLOCK * 4 ? 4 : 1;
    const unsigned nt = (unsigned)((n + GM_BLOCK * items - 1) / (GM_BLOCK * items));
    // tile records behind the word that counts the list entries taken, then the tiles' counts
    PD_TRY(h->tile_cnt.ensure(sizeof(uint2) * ((size_t)nt + 1) + sizeof(unsigned int) * (size_t)nt));
    PD_TRY(h->img_list.ensure(sizeof(unsigned int) * (size_t)(m_cap > 0 ? m_cap : 1)));
    unsigned int* taken = h->tile_cnt.as<unsigned int>();
    uint2* tiles = h->tile_cnt.as<uint2>() + 1;
    unsigned int* cnt = reinterpret_cast<unsigned int*>(tiles + nt);
    int rc = PD_OK;
    PD_CUDA(cudaMemsetAsync(taken, 0, sizeof(unsigned int), st));
    auto go = [&](auto find, auto write, auto* pos, auto* boxes, auto* shifts) {
        pd::launch(find, nt, GM_BLOCK, 0, st, pos, n, boxes, (unsigned int)m_cap, h->img_list.as<unsigned int>(), taken,
                   tiles, cnt);
        bool scanned;
        rc = prefix_tiles(cnt, nt, st, &scanned);
        if (rc != PD_OK) return;
        pd::launch(write, nt, GM_BLOCK, 0, st, pos, h->gid, n, GM_BLOCK * items, boxes, shifts,
                   (const unsigned int*)h->img_list.as<unsigned int>(), (unsigned int)m_cap, (const uint2*)tiles,
                   (const unsigned int*)cnt, scanned, h->img_src.as<int>(), h->img_shift.as<unsigned char>(), m_cap,
                   h->cap, pc, &h->ctrl->n_img, &h->ctrl->err);
    };
    if (h->dtype == PD_F64) {
        const BoxSet<double>* b = h->boxes.as<BoxSet<double>>();
        const double* sh = h->shifts.as<double>();
        go(items == 4 ? k_ghost_find<double, 4> : k_ghost_find<double, 1>, k_ghost_write<double>, (double4*)h->pos, b, sh);
    } else {
        const BoxSet<float>* b = h->boxes.as<BoxSet<float>>();
        const float* sh = h->shifts.as<float>();
        go(items == 4 ? k_ghost_find<float, 4> : k_ghost_find<float, 1>, k_ghost_write<float>, (float4*)h->pos, b, sh);
    }
    PD_TRY(rc);
    PD_LAUNCH_CHECK();
    return PD_OK;
}

// room for the images of the next ghost_get: the previous count with a margin, before
// the first one the domain's ghost shell at the mean density
static long ghost_room(pd_vd h) {
    if (h->n_img > 0) return h->n_img + h->n_img / 8 + 1024;
    double f = 1;
    for (int d = 0; d < 3; ++d)
        if (h->bc[d] == PD_PERIODIC) f *= 1.0 + 2.0 * std::min(h->g[d] / (h->hi[d] - h->lo[d]), 1.0);
    return (long)((f - 1) * 1.1 * (double)h->n_real) + 1024;
}

// The images of the real particles, their count to the control block.  With sync_count
// the count is read back, one synchronisation (the API path, like the reference's D->H
// copy of the scan tail); where the room estimated before did not suffice the storage
// grows and the images are written again.  Without it `img_cap` bounds the images and an
// overflow sets ERR_IMG_OVERFLOW (the captured integrator path).
// Measured, find + write against count + scan + write: 13 us instead of 33 for 4,099 FP64
// particles (25 for count and write), 53 instead of 76 for 1,000,000; the box upload made
// once and the second read-back dropped (it could only repeat the first) leave one host
// round trip of three.
int ghost_generate(pd_vd h, long img_cap, bool sync_count, cudaStream_t st) {
    if (!sync_count) return ghost_make(h, img_cap, st);
    const long n = h->n_real;
    const bool none = n <= 0 || h->nbox == 0;  // no image whatever the positions: nothing to read back
    long room = none ? 0 : ghost_room(h);
    // no memory for the estimate (particles that keep away from the faces may need far less): what
    // there is, which finds the count
    if (!none && ensure_capacity(h, n + room + 1, st) != PD_OK) room = std::max(h->cap - n - 1, 0L);
    PD_TRY(ghost_make(h, room, st));
    if (none) h->ctrl_h->n_img = 0;
    else PD_TRY(read_ctrl(h, st));
    const long m = h->ctrl_h->n_img;
    if (m > room) {
        h->ctrl_h->err &= ~ERR_IMG_OVERFLOW;
        PD_CUDA(cudaMemcpyAsync(&h->ctrl->err, &h->ctrl_h->err, sizeof(unsigned int), cudaMemcpyHostToDevice, st));
        PD_TRY(ensure_capacity(h, n + m + 1, st));
        PD_TRY(ghost_make(h, m, st));
    }
    h->n_img = m;
    h->n_total = n + m;
    h->img_valid = true;
    h->img_gen_order = true;
    return PD_OK;
}

int ghost_replay(pd_vd h, unsigned long prop_mask, bool with_pos, const unsigned int* n_img_dev, long n_img_bound,
                 cudaStream_t st) {
    if (n_img_bound <= 0) return PD_OK;
    PropCopy pc = make_copy(h, prop_mask);
    unsigned g = grid_for(n_img_bound, 256);
    if (h->dtype == PD_F64)
        pd::launch(k_ghost_replay<double>, g, 256, 0, st, (double4*)h->pos, h->n_real, h->img_src.as<int>(),
                                                  h->img_shift.as<unsigned char>(), h->shifts.as<double>(),
                                                  n_img_dev, n_img_bound, with_pos ? 1 : 0, pc);
    else
        pd::launch(k_ghost_replay<float>, g, 256, 0, st, (float4*)h->pos, h->n_real, h->img_src.as<int>(),
                                                 h->img_shift.as<unsigned char>(), h->shifts.as<float>(), n_img_dev,
                                                 n_img_bound, with_pos ? 1 : 0, pc);
    PD_LAUNCH_CHECK();
    return PD_OK;
}

template <class T> static int user_boxes(pd_vd h, const double* boxes, const int* sv, int nb, BoxSet<T>& B) {
    if (nb < 0 || nb > MAXBOX) {
        set_error("at most %d ghost boxes", MAXBOX);
        return PD_EINVAL;
    }
    memset(&B, 0, sizeof(B));
    B.nb = nb;
    for (int i = 0; i < nb; ++i) {
        for (int d = 0; d < 3; ++d) {
            B.lo[i][d] = (T)boxes[6 * i + d];
            B.hi[i][d] = (T)boxes[6 * i + 3 + d];
        }
        if (sv[i] < 0 || sv[i] > 255) {
            set_error("shift id out of range");
            return PD_EINVAL;
        }
        B.sv[i] = sv[i];
    }
    return PD_OK;
}

}  // namespace pd

using namespace pd;

extern "C" {

int pd_ghost_get(pd_vd h, unsigned long prop_mask, int opt, void* stream) {
    if (!h) return PD_EINVAL;
    if (h->ghost_pending) {
        set_error("ghost_get: an Ighost_get is waiting for its ghost_wait");
        return PD_ESTATE;
    }
    cudaStream_t st = S(stream);
    if ((opt & PD_SKIP_LABELLING) && h->img_valid) {
        // ghost_get_ with SKIP_LABELLING: positions unless NO_POSITION, properties in the mask
        PD_TRY(ghost_replay(h, prop_mask, !(opt & PD_NO_POSITION), nullptr, h->n_img, st));
        return PD_OK;
    }
    h->n_total = h->n_real;
    PD_TRY(ghost_boxes_upload(h, st));
    PD_TRY(ghost_generate(h, 0, true, st));
    if (h->ctrl_h->err & ERR_IMG_OVERFLOW) {
        set_error("ghost_get: image overflow");
        return PD_EOVERFLOW;
    }
    h->epoch++;
    return PD_OK;
}

int pd_ighost_get(pd_vd h, unsigned long prop_mask, int opt, void* stream) {
    if (!h) return PD_EINVAL;
    if (h->ghost_pending) {
        set_error("Ighost_get: the previous Ighost_get was not waited for");
        return PD_ESTATE;
    }
    cudaStream_t st = S(stream);
    h->pend_mask = prop_mask;
    h->pend_opt = opt;
    if ((opt & PD_SKIP_LABELLING) && h->img_valid) {
        PD_TRY(ghost_replay(h, prop_mask, !(opt & PD_NO_POSITION), nullptr, h->n_img, st));
        h->ghost_pending = true;
        h->pend_replay = true;
        return PD_OK;
    }
    // images written without a host read of their count: room for the previous count
    // with a margin (growing the storage, if needed, synchronises once here); an
    // overflow is detected by ghost_wait, which then redoes the call synchronously
    h->n_total = h->n_real;
    h->img_valid = false;
    const long want = h->n_img + h->n_img / 4 + 1024;
    PD_TRY(ensure_capacity(h, h->n_real + want + 1, st));
    PD_TRY(ghost_boxes_upload(h, st));
    PD_TRY(ghost_generate(h, h->cap - h->n_real - 1, false, st));
    h->ghost_pending = true;
    h->pend_replay = false;
    return PD_OK;
}

int pd_ghost_wait(pd_vd h, void* stream) {
    if (!h) return PD_EINVAL;
    if (!h->ghost_pending) return PD_OK;
    cudaStream_t st = S(stream);
    h->ghost_pending = false;
    if (h->pend_replay) return cudaStreamSynchronize(st) == cudaSuccess ? PD_OK : PD_ECUDA;
    PD_TRY(read_ctrl(h, st));
    if (h->ctrl_h->err & ERR_IMG_OVERFLOW) {
        h->ctrl_h->err &= ~ERR_IMG_OVERFLOW;
        PD_CUDA(cudaMemcpyAsync(&h->ctrl->err, &h->ctrl_h->err, sizeof(unsigned int), cudaMemcpyHostToDevice, st));
        return pd_ghost_get(h, h->pend_mask, h->pend_opt & ~PD_SKIP_LABELLING, stream);
    }
    h->n_img = h->ctrl_h->n_img;
    h->n_total = h->n_real + h->n_img;
    h->img_valid = true;
    h->img_gen_order = true;
    h->epoch++;
    return PD_OK;
}

int pd_ghost_put(pd_vd h, unsigned long prop_mask, int op, void* stream) {
    if (!h || (op != PD_PUT_ADD && op != PD_PUT_MAX && op != PD_PUT_REPLACE)) return PD_EINVAL;
    if (!h->img_valid || !h->img_gen_order) {
        set_error("ghost_put: no ghost_get images in generation order (call ghost_get first)");
        return PD_ESTATE;
    }
    cudaStream_t st = S(stream);
    const long n = h->n_real;
    if (n == 0 || h->n_img == 0) return PD_OK;
    const unsigned g = grid_for(h->n_img, 256);
    const int* src = h->img_src.as<int>();
    for (size_t p = 0; p < h->props.size(); ++p) {
        if (!(prop_mask & (1ul << p))) continue;
        Prop& P = h->props[p];
        switch (P.type) {
            case PD_F64: pd::launch(k_ghost_put<double>, g, 256, 0, st, (double*)P.d, h->cap, P.ncomp, n, src, h->n_img, op); break;
            case PD_F32: pd::launch(k_ghost_put<float>, g, 256, 0, st, (float*)P.d, h->cap, P.ncomp, n, src, h->n_img, op); break;
            case PD_I32: pd::launch(k_ghost_put<int>, g, 256, 0, st, (int*)P.d, h->cap, P.ncomp, n, src, h->n_img, op); break;
            case PD_U32: pd::launch(k_ghost_put<unsigned int>, g, 256, 0, st, (unsigned int*)P.d, h->cap, P.ncomp, n, src, h->n_img, op); break;
            case PD_I64: pd::launch(k_ghost_put<long long>, g, 256, 0, st, (long long*)P.d, h->cap, P.ncomp, n, src, h->n_img, op); break;
        }
        PD_LAUNCH_CHECK();
    }
    return PD_OK;
}

int pd_ghost_records(pd_vd h, int* src, int* shift_id, long cap, long* n_img) {
    if (!h || !n_img) return PD_EINVAL;
    *n_img = h->img_valid ? h->n_img : 0;
    long m = *n_img < cap ? *n_img : cap;
    if (m > 0) {
        if (src) PD_CUDA(cudaMemcpy(src, h->img_src.p, sizeof(int) * m, cudaMemcpyDeviceToHost));
        if (shift_id) {
            std::vector<unsigned char> t(m);
            PD_CUDA(cudaMemcpy(t.data(), h->img_shift.p, m, cudaMemcpyDeviceToHost));
            for (long i = 0; i < m; ++i) shift_id[i] = t[i];
        }
    }
    return PD_OK;
}

int pd_ghost_count_boxes(pd_vd h, const double* boxes_host, const int* sv_host, int nb, int* counts_host,
                         void* stream) {
    if (!h || !boxes_host || !sv_host || !counts_host) return PD_EINVAL;
    cudaStream_t st = S(stream);
    long n = h->n_real;
    PD_TRY(h->img_cnt.ensure(sizeof(unsigned int) * (n + 1)));
    unsigned g = grid_for(n, 256);
    if (h->dtype == PD_F64) {
        BoxSet<double> B;
        PD_TRY(user_boxes(h, boxes_host, sv_host, nb, B));
        double sh[3] = {0, 0, 0};
        PD_TRY(upload_boxes_t(h, B, sh, 1, st));
        if (n) pd::launch(k_ghost_count<double>, g, 256, 0, st, (const double4*)h->pos, n, h->boxes.as<BoxSet<double>>(),
                                                        h->img_cnt.as<unsigned int>());
    } else {
        BoxSet<float> B;
        PD_TRY(user_boxes(h, boxes_host, sv_host, nb, B));
        float sh[3] = {0, 0, 0};
        PD_TRY(upload_boxes_t(h, B, sh, 1, st));
        if (n) pd::launch(k_ghost_count<float>, g, 256, 0, st, (const float4*)h->pos, n, h->boxes.as<BoxSet<float>>(),
                                                       h->img_cnt.as<unsigned int>());
    }
    PD_LAUNCH_CHECK();
    if (n) PD_CUDA(cudaMemcpyAsync(counts_host, h->img_cnt.p, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    PD_CUDA(cudaStreamSynchronize(st));
    h->img_valid = false;  // the domain boxes were replaced
    return PD_OK;
}

int pd_ghost_get_boxes(pd_vd h, const double* boxes_host, const int* sv_host, int nb, const double* shifts_host,
                       int n_shifts, void* stream) {
    if (!h || !boxes_host || !sv_host || !shifts_host || n_shifts < 1 || n_shifts > 256) return PD_EINVAL;
    for (int i = 0; i < nb; ++i)
        if (sv_host[i] >= n_shifts) {
            set_error("shift id %d has no shift vector", sv_host[i]);
            return PD_EINVAL;
        }
    cudaStream_t st = S(stream);
    h->n_total = h->n_real;
    if (h->dtype == PD_F64) {
        BoxSet<double> B;
        PD_TRY(user_boxes(h, boxes_host, sv_host, nb, B));
        PD_TRY(upload_boxes_t(h, B, shifts_host, n_shifts, st));
    } else {
        BoxSet<float> B;
        PD_TRY(user_boxes(h, boxes_host, sv_host, nb, B));
        std::vector<float> sh(3 * n_shifts);
        for (int i = 0; i < 3 * n_shifts; ++i) sh[i] = (float)shifts_host[i];
        PD_TRY(upload_boxes_t(h, B, sh.data(), n_shifts, st));
    }
    PD_TRY(ghost_generate(h, 0, true, st));  // (the next domain ghost_get uploads the domain boxes again)
    h->epoch++;
    return (h->ctrl_h->err & ERR_IMG_OVERFLOW) ? PD_EOVERFLOW : PD_OK;
}

}  // extern "C"
