// rb_step.cu -- the prox_rigid_bodies semi-implicit time step on sm_100a.
//
// One rb_step call advances every scene of an rb_bodies batch by one step.  The pipeline (one kernel per
// stage, all on the caller's stream, no host synchronisation, so a sequence of steps can be captured in a
// CUDA graph) follows steppers.py:47 SemiImplicitStepper.step:
//
//   k_bodies          forces, gyroscopic torque, world inverse inertia, W f_ext      state_storage.py:43-185
//   k_world_vertices  rotate_array(q, V) + r for every body vertex                   collision_detection.py:32
//   k_clusters        32-leaf cluster boxes (unions of k-DOP K=3 leaf boxes + envelope) kdop_bvh.py:52, kdop.py:53
//   k_roots           body boxes (the BVH root)                                         kdop_bvh.py:215
//   k_pairs           body pairs in combinations() order whose roots overlap           collision_detection.py:70
//   k_mid             per pair, the triangles of each side whose leaf overlaps a leaf   kdop_bvh.py:127, :234
//                     of the other side (ascending, = np.unique of the traversal)      collision_detection.py:234
//   k_narrow          Frank-Wolfe deepest point on each candidate triangle in the       collision_detection.py:87
//                     other body's SDF, contact emission
//   k_dedup           first-occurrence duplicate removal and compaction                 collision_detection.py:255
//   k_contacts        contact frame, Jacobian, W J^T, b, Delassus diagonal, r, mu        contacts.py:31-55
//   k_solve           proximal solver (one block per scene)                             gauss_seidel_solver.py:14
//   k_integrate       u += dt W f + W J^T sol; r, q update                               state_storage.py:239-302
//   k_post_*          post-stabilisation                                                steppers.py:15
//
// Counts that are only known on the device (pairs, candidates, contacts) are read by the consumers from
// device counters; kernels that depend on them run grid-stride loops over those counters.
#include <cuda_runtime.h>

#include <climits>
#include <cstdio>
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>

#include "rainbow_b200.h"
#include "rb_device.cuh"
#include "rb_internal.h"
#include "rb_layout.h"

namespace rb {

// kernels launched by this library in this process (rb_launch_count)
std::atomic<int64_t> g_launches{0};
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

constexpr int kWarpsPerBlock = 4;
constexpr int kBlock = 32 * kWarpsPerBlock;
constexpr int kAbort = 15;   // counters[kAbort]: nonzero once a capacity was exceeded
constexpr int kNWide = 13, kWideNext = 14;   // counters: pairs of k_mid_wide, and the next of them
constexpr int kSolveSmemBodies = 4608;   // 216 KB of body accumulators per solver block

// ---------------------------------------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ int scene_of(const int32_t* scene_start, int n_scenes, int body) {
    int lo = 0, hi = n_scenes;   // find s with scene_start[s] <= body < scene_start[s+1]
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (__ldg(scene_start + mid) <= body) lo = mid; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---------------------------------------------------------------------------------------------------------
// device-wide exclusive scan of int32 counts (three phases; the element count may live on the device)
// data[0..n) -> exclusive prefix sums, data[n] = total, which ScanTotal may also put into a counter
// ---------------------------------------------------------------------------------------------------------
// with a device count, n_host is the capacity the count is clamped to
__device__ __forceinline__ int scan_n(const int32_t* n_dev, int n_host) { return n_dev ? min(*n_dev, n_host) : n_host; }

__global__ void k_scan_reduce(const int32_t* __restrict__ data, const int32_t* n_dev, int n_host,
                              int32_t* __restrict__ partial) {
    const int n = scan_n(n_dev, n_host);
    const int chunk = (n + gridDim.x - 1) / gridDim.x;
    const int start = blockIdx.x * chunk, end = min(n, start + chunk);
    int s = 0;
    for (int i = start + threadIdx.x; i < end; i += blockDim.x) s += data[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ int ws[32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
        partial[blockIdx.x] = t;
    }
}
// what becomes of a scan's total: written to counters[which], and, above the capacity, the status bit that aborts the
// rest of the step (unless an earlier stage overflowed: the total is not meaningful then)
struct ScanTotal {
    int32_t* counters = nullptr;
    int which = 0, capacity = 0, bit = 0;
    int32_t* status = nullptr;
    __device__ __forceinline__ void put(int32_t total) const {
        if (!counters) return;
        counters[which] = total;
        if (!counters[kAbort] && total > capacity) {
            atomicOr(counters + kAbort, bit);
            atomicOr(status, bit);
        }
    }
};
__global__ void k_scan_top(int32_t* __restrict__ partial, int nblocks, const ScanTotal total) {
    // single block of 1024 threads, nblocks <= 1024
    __shared__ int s[1024];
    const int t = threadIdx.x;
    int v = t < nblocks ? partial[t] : 0;
    s[t] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        int a = t >= o ? s[t - o] : 0;
        __syncthreads();
        s[t] += a;
        __syncthreads();
    }
    if (t < nblocks) partial[t] = s[t] - v;
    if (t == 1023) { partial[nblocks] = s[t]; total.put(s[t]); }
}
// the whole scan by one block: with few elements the launches of the three phases cost more than the elements
// (11 us against 4 for 4097 bodies)
constexpr int kScanOne = 16384;
__global__ void __launch_bounds__(1024) k_scan_one(int32_t* __restrict__ data, const int32_t* n_dev, int n_host,
                                                   const ScanTotal total) {
    __shared__ int ws[33];
    const int n = scan_n(n_dev, n_host);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += 4096) {   // four elements a thread
        const int i = base + 4 * threadIdx.x;
        int v[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) { v[k] = i + k < n ? data[i + k] : 0; sum += v[k]; }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += a;
        }
        if (lane == 31) ws[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            const int w = ws[lane];
            int wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int a = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += a;
            }
            ws[lane] = wi - w;
            if (lane == 31) ws[32] = wi;
        }
        __syncthreads();
        int at = carry + ws[wid] + incl - sum;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i + k < n) data[i + k] = at;
            at += v[k];
        }
        carry += ws[32];
        __syncthreads();
    }
    if (threadIdx.x == 0) { data[n] = carry; total.put(carry); }
}
__global__ void k_scan_down(int32_t* __restrict__ data, const int32_t* n_dev, int n_host,
                            const int32_t* __restrict__ partial) {
    const int n = scan_n(n_dev, n_host);
    const int chunk = (n + gridDim.x - 1) / gridDim.x;
    const int start = blockIdx.x * chunk, end = min(n, start + chunk);
    __shared__ int ws[32];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = partial[blockIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int base = start; base < end; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int v = i < end ? data[i] : 0;
        int incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            int a = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += a;
        }
        if (lane == 31) ws[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            int wv = lane < nw ? ws[lane] : 0;
            int wi = wv;
            for (int o = 1; o < 32; o <<= 1) {
                int a = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += a;
            }
            if (lane < nw) ws[lane] = wi - wv;
        }
        __syncthreads();
        const int c = carry;
        if (i < end) data[i] = c + ws[wid] + incl - v;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = c + ws[wid] + incl;
        __syncthreads();
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) data[n] = partial[gridDim.x];
}
static void scan_total(int32_t* data, const int32_t* n_dev, int n_host, int32_t* partial, const ScanTotal total,
                       cudaStream_t st) {
    if (n_host <= kScanOne) {
        k_scan_one<<<1, 1024, 0, st>>>(data, n_dev, n_host, total); note_launch();
        return;
    }
    const int G = kScanGrid;
    k_scan_reduce<<<G, 256, 0, st>>>(data, n_dev, n_host, partial); note_launch();
    k_scan_top<<<1, 1024, 0, st>>>(partial, G, total); note_launch();
    k_scan_down<<<G, 256, 0, st>>>(data, n_dev, n_host, partial); note_launch();
}
void scan(int32_t* data, const int32_t* n_dev, int n_host, int32_t* partial, cudaStream_t st) {
    scan_total(data, n_dev, n_host, partial, ScanTotal{}, st);
}

// ---------------------------------------------------------------------------------------------------------
// bodies: state_storage.py:108 _compute_total_external_forces, :158 _compute_inverse_mass_matrix, :53
// ---------------------------------------------------------------------------------------------------------
struct StepArgs {
    rb_shapes sh;
    rb_bodies bd;
    rb_caps caps;
    rb_params pr;
    rb_outputs out;
    Workspace ws;
};

// also starts the step: counters, contact counts and the scenes' statistics at zero, and, with no FP32 phase to do it
// (it reads the last step's), the scenes' FP32 bookkeeping
__global__ void k_bodies(const StepArgs a) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < 16) a.ws.counters[b] = 0;
    if (b <= a.bd.n_bodies) a.ws.bc_ptr[b] = 0;
    if (b < a.bd.n_scenes) {
        rb_scene_stats* st = a.out.stats + b;
        st->n_grid_lookups = 0; st->n_leaf_overlaps = 0;
        st->n_grid_lookups32 = 0; st->n_search_flips = 0; st->n_accept_flips = 0;
        if (a.pr.precision == RB_PRECISION_FP64) { a.ws.sweeps32[b] = -1; a.ws.fin32[b] = 0; }
    }
    if (b >= a.bd.n_bodies) return;
    a.ws.bc_fill[b] = 0;
    double* d = a.ws.dux + 6 * b;
    double* du = a.ws.du + 6 * b;
    double* Wi = a.ws.Winv + 9 * b;
    if (a.bd.fixed[b]) {
        for (int i = 0; i < 6; ++i) { d[i] = 0.0; du[i] = 0.0; }
        for (int i = 0; i < 9; ++i) Wi[i] = 0.0;
        return;
    }
    const double* q = a.bd.x + 7 * b + 3;
    const d3 v = ld3(a.bd.u + 6 * b), w = ld3(a.bd.u + 6 * b + 3);
    double R[9], Iw[9], Ib[3], Binv[3];
    quat_to_matrix(q, R);
    for (int i = 0; i < 3; ++i) Ib[i] = a.bd.inertia[3 * b + i];
    update_inertia_tensor(R, Ib, Iw);
    const d3 c = cross_np(w, gemv3_np(Iw, w));
    double T[3] = {-c.x, -c.y, -c.z}, F[3] = {0.0, 0.0, 0.0};
    const double mass = a.bd.mass[b];
    for (int e = a.bd.force_ptr[b]; e < a.bd.force_ptr[b + 1]; ++e) {
        const int f = a.bd.force_list[e];
        const double* fp = a.bd.force_params + 4 * f;
        double Fi[3], Ti[3];
        if (a.bd.force_kind[f] == 0) {          // types.py:204 Gravity.compute: F = -m g up
            const double s = -mass * fp[0];
            Fi[0] = s * fp[1]; Fi[1] = s * fp[2]; Fi[2] = s * fp[3];
            Ti[0] = 0.0; Ti[1] = 0.0; Ti[2] = 0.0;
        } else {                                 // types.py:239 Damping.compute: F = -v alpha, T = -w beta
            Fi[0] = -v.x * fp[0]; Fi[1] = -v.y * fp[0]; Fi[2] = -v.z * fp[0];
            Ti[0] = -w.x * fp[1]; Ti[1] = -w.y * fp[1]; Ti[2] = -w.z * fp[1];
        }
        for (int i = 0; i < 3; ++i) { F[i] = F[i] + Fi[i]; T[i] = T[i] + Ti[i]; }
    }
    const double m = 1.0 / mass;
    for (int i = 0; i < 3; ++i) Binv[i] = 1.0 / Ib[i];
    update_inertia_tensor(R, Binv, Wi);
    const double dt = a.pr.dt;
    for (int i = 0; i < 3; ++i) {   // bsr_matvec over the 3x3 blocks of W
        double s = 0.0;
        s += (i == 0 ? m : 0.0) * F[0];
        s += (i == 1 ? m : 0.0) * F[1];
        s += (i == 2 ? m : 0.0) * F[2];
        double t = 0.0;
        t += Wi[3 * i] * T[0];
        t += Wi[3 * i + 1] * T[1];
        t += Wi[3 * i + 2] * T[2];
        d[i] = s; d[3 + i] = t;
        du[i] = dt * s; du[3 + i] = dt * t;   // steppers.py:64 delta_u = dt * delta_u_ext
    }
}

// collision_detection.py:32 V_world = rotate_array(q, V) + r
__global__ void k_world_vertices(const StepArgs a, int n_verts) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n_verts) return;
    const int b = a.bd.vert_body[g];
    const int local = g - a.bd.body_v0[b];
    const int s = a.bd.shape[b];
    const d3 V = ld3(a.sh.V + 3 * (size_t)(a.sh.v_off[s] + local));
    const double* xb = a.bd.x + 7 * b;
    const d3 p = quat_rotate_row(xb + 3, V);
    st3(a.ws.Vw + 3 * (size_t)g, d3{p.x + xb[0], p.y + xb[1], p.z + xb[2]});
}

// leaf box of triangle t of a body (kdop.py:53 make with K=3: min/max of the triangle's world coordinates
// -/+ envelope), from the body's world vertices Vw and its shape's triangles T; L = (lo[3], hi[3])
__device__ __forceinline__ void leaf_box(const int32_t* T, const double* Vw, int t, double env, double* L) {
    const int32_t* tri = T + 3 * (size_t)t;
    const int v[3] = {tri[0], tri[1], tri[2]};
    for (int axis = 0; axis < 3; ++axis) {
        double l = INFINITY, h = -INFINITY;
        for (int k = 0; k < 3; ++k) {
            const double pr = Vw[3 * v[k] + axis];
            if (pr < l) l = pr;
            if (pr > h) h = pr;
        }
        L[axis] = l - env;
        L[3 + axis] = h + env;
    }
}

// the box of every run of 32 consecutive triangles of a body (the union of their leaf boxes); one warp per
// cluster.  Leaf boxes are not stored: the mid phase recomputes the few it tests from the world vertices.
__global__ void k_clusters(const StepArgs a, int n_clusters) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= n_clusters) return;
    const int b = a.bd.clu_body[warp];
    const int c = warp - a.bd.body_c0[b];
    const int s = a.bd.shape[b];
    const int nt = a.sh.t_off[s + 1] - a.sh.t_off[s];
    const int t = 32 * c + lane;
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    if (t < nt) {
        double L[6];
        leaf_box(a.sh.T + 3 * (size_t)a.sh.t_off[s], a.ws.Vw + 3 * (size_t)a.bd.body_v0[b], t, a.pr.envelope, L);
        for (int axis = 0; axis < 3; ++axis) { lo[axis] = L[axis]; hi[axis] = L[3 + axis]; }
    }
    for (int axis = 0; axis < 3; ++axis) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[axis] = fmin(lo[axis], __shfl_xor_sync(0xffffffffu, lo[axis], o));
            hi[axis] = fmax(hi[axis], __shfl_xor_sync(0xffffffffu, hi[axis], o));
        }
    }
    if (lane == 0) {
        double* C = a.ws.clu + 6 * (size_t)warp;
        C[0] = lo[0]; C[1] = lo[1]; C[2] = lo[2]; C[3] = hi[0]; C[4] = hi[1]; C[5] = hi[2];
    }
}

// body box = union of its cluster boxes (kdop_bvh.py:229-231); one warp per body
__global__ void k_roots(const StepArgs a) {
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (b >= a.bd.n_bodies) return;
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int c = a.bd.body_c0[b] + lane; c < a.bd.body_c0[b + 1]; c += 32) {
        const double* C = a.ws.clu + 6 * (size_t)c;
        for (int axis = 0; axis < 3; ++axis) { lo[axis] = fmin(lo[axis], C[axis]); hi[axis] = fmax(hi[axis], C[3 + axis]); }
    }
    for (int axis = 0; axis < 3; ++axis)
        for (int o = 16; o > 0; o >>= 1) {
            lo[axis] = fmin(lo[axis], __shfl_xor_sync(0xffffffffu, lo[axis], o));
            hi[axis] = fmax(hi[axis], __shfl_xor_sync(0xffffffffu, hi[axis], o));
        }
    if (lane == 0) {
        double* R = a.ws.root + 6 * b;
        R[0] = lo[0]; R[1] = lo[1]; R[2] = lo[2]; R[3] = hi[0]; R[4] = hi[1]; R[5] = hi[2];
    }
}

// ---------------------------------------------------------------------------------------------------------
// broad phase: body pairs (i < j, same scene) in combinations() order whose boxes overlap; warp per body
// ---------------------------------------------------------------------------------------------------------
template <bool WRITE>
__global__ void k_pairs(const StepArgs a) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= a.bd.n_bodies) return;
    if (WRITE && a.ws.counters[kAbort]) return;
    const int s = scene_of(a.bd.scene_start, a.bd.n_scenes, i);
    const int end = a.bd.scene_start[s + 1];
    double Ri[6];
    for (int k = 0; k < 6; ++k) Ri[k] = a.ws.root[6 * i + k];
    int count = 0;
    const int base = WRITE ? a.ws.pair_cnt[i] : 0;
    for (int j0 = i + 1; j0 < end; j0 += 32) {
        const int j = j0 + lane;
        const bool ov = j < end && overlap(Ri, a.ws.root + 6 * j);
        const unsigned bal = __ballot_sync(0xffffffffu, ov);
        if (WRITE && ov) {
            const int pos = base + count + __popc(bal & lanemask_lt());
            a.ws.pairs[2 * pos] = i;
            a.ws.pairs[2 * pos + 1] = j;
        }
        count += __popc(bal);
    }
    if (!WRITE && lane == 0) a.ws.pair_cnt[i] = count;
}

// ---------------------------------------------------------------------------------------------------------
// mid phase: for body pair (A, B) the A-triangles whose leaf box overlaps some B leaf box and vice versa.
// The reference's tandem traversal (kdop_bvh.py:127-178) reports exactly the overlapping leaf pairs because
// each inner volume is the exact union of its children; np.unique of each column (collision_detection.py:234)
// makes both sets ascending.  Clusters of 32 triangles with exact union boxes prune the same way.
// ---------------------------------------------------------------------------------------------------------
// per-warp shared arrays of k_mid, sized at launch by the largest shape: lists of the clusters of A (of B)
// whose box overlaps B's (A's) body box, and the hit masks of their 32 triangles
__device__ __forceinline__ void mid_arrays(int max_clusters, int warp, int16_t*& listA, int16_t*& listB,
                                           uint32_t*& maskA, uint32_t*& maskB) {
    extern __shared__ uint32_t mid_smem[];
    const int words = 3 * max_clusters;   // 2 lists of int16 + 2 masks of uint32 = 3 words per cluster
    uint32_t* base = mid_smem + (size_t)warp * words;
    maskA = base;
    maskB = base + max_clusters;
    listA = reinterpret_cast<int16_t*>(base + 2 * max_clusters);
    listB = listA + max_clusters;
}

// writes a pair's candidates, the set bits of both sides' masks, in ascending (side, triangle) order, in room reserved
// with one atomic: pair_items[p] = first candidate of the pair, pair_n_items[p] = their number (one warp)
__device__ __forceinline__ void mid_emit(const StepArgs& a, int p, int nA, int nB, const int16_t* listA, const int16_t* listB,
                                         const uint32_t* maskA, const uint32_t* maskB, int n_ovl) {
    const int lane = threadIdx.x & 31;
    int cnt = 0;
    for (int k = lane; k < nA; k += 32) cnt += __popc(maskA[k]);
    for (int k = lane; k < nB; k += 32) cnt += __popc(maskB[k]);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    int pos = 0;
    if (lane == 0) pos = atomicAdd(a.ws.counters + kNItems, cnt);
    pos = __shfl_sync(0xffffffffu, pos, 0);
    if (lane == 0) { a.ws.pair_items[p] = pos; a.ws.pair_n_items[p] = cnt; a.ws.pair_ovl[p] = n_ovl; }
    if (pos + cnt > a.caps.item_capacity) return;   // k_narrow aborts the step
    for (int side = 0; side < 2; ++side) {
        const int n = side ? nB : nA;
        const int16_t* list = side ? listB : listA;
        const uint32_t* mask = side ? maskB : maskA;
        for (int k = 0; k < n; ++k) {
            const uint32_t bits = mask[k];
            if (bits & (1u << lane)) {
                const int at = pos + __popc(bits & lanemask_lt());
                a.ws.item_pair[at] = p;
                a.ws.item_tri[at] = (side << 31) | (32 * list[k] + lane);
            }
            pos += __popc(bits);
        }
    }
}

// Single pass: warps take pairs from a shared counter and find the pair's candidate triangles.  A pair of more than
// kMidLight cluster pairs (4: 944 us, 16: 540, 64: 595 for both kernels on 55,960 pairs) goes to k_mid_wide's list (in pair_cont, which is written later): one warp took up to a
// millisecond over two deeply overlapping 448-triangle spheres, whatever the other pairs.
constexpr int kMidLight = 16;
__global__ void __launch_bounds__(kBlock) k_mid(const StepArgs a, int max_clusters) {
    int16_t *listA, *listB;
    uint32_t *maskA, *maskB;
    mid_arrays(max_clusters, threadIdx.x >> 5, listA, listB, maskA, maskB);
    const int lane = threadIdx.x & 31;
    if (a.ws.counters[kAbort]) return;
    const int n_pairs = a.ws.counters[kNPairs];
    for (;;) {
        int p = 0;
        if (lane == 0) p = atomicAdd(a.ws.counters + kMidNext, 1);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= n_pairs) break;
        const int A = a.ws.pairs[2 * p], B = a.ws.pairs[2 * p + 1];
        const int cA0 = a.bd.body_c0[A], ncA = a.bd.body_c0[A + 1] - cA0;
        const int cB0 = a.bd.body_c0[B], ncB = a.bd.body_c0[B + 1] - cB0;
        const int ntA = a.bd.body_t0[A + 1] - a.bd.body_t0[A];
        const int ntB = a.bd.body_t0[B + 1] - a.bd.body_t0[B];
        const int32_t* TA = a.sh.T + 3 * (size_t)a.sh.t_off[a.bd.shape[A]];
        const int32_t* TB = a.sh.T + 3 * (size_t)a.sh.t_off[a.bd.shape[B]];
        const double* VwA = a.ws.Vw + 3 * (size_t)a.bd.body_v0[A];
        const double* VwB = a.ws.Vw + 3 * (size_t)a.bd.body_v0[B];
        const double env = a.pr.envelope;
        const double* rootA = a.ws.root + 6 * A;
        const double* rootB = a.ws.root + 6 * B;
        if (ncA > max_clusters || ncB > max_clusters) {
            if (lane == 0) {
                atomicOr(a.out.status, RB_STATUS_MESH_TOO_LARGE);
                atomicOr(a.ws.counters + kAbort, RB_STATUS_MESH_TOO_LARGE);
                a.ws.pair_items[p] = 0; a.ws.pair_n_items[p] = 0; a.ws.pair_ovl[p] = 0;
            }
            continue;
        }
        int nA = 0, nB = 0;
        for (int c0 = 0; c0 < ncA; c0 += 32) {
            const int c = c0 + lane;
            const bool ok = c < ncA && overlap(a.ws.clu + 6 * (size_t)(cA0 + c), rootB);
            const unsigned bal = __ballot_sync(0xffffffffu, ok);
            if (ok) listA[nA + __popc(bal & lanemask_lt())] = (int16_t)c;
            nA += __popc(bal);
        }
        for (int c0 = 0; c0 < ncB; c0 += 32) {
            const int c = c0 + lane;
            const bool ok = c < ncB && overlap(a.ws.clu + 6 * (size_t)(cB0 + c), rootA);
            const unsigned bal = __ballot_sync(0xffffffffu, ok);
            if (ok) listB[nB + __popc(bal & lanemask_lt())] = (int16_t)c;
            nB += __popc(bal);
        }
        if (nA * nB > kMidLight) {
            if (lane == 0) a.ws.pair_cont[atomicAdd(a.ws.counters + kNWide, 1)] = p;
            __syncwarp();
            continue;
        }
        for (int k = lane; k < nA; k += 32) maskA[k] = 0u;
        for (int k = lane; k < nB; k += 32) maskB[k] = 0u;
        __syncwarp();
        int n_ovl = 0;
        for (int ia = 0; ia < nA; ++ia) {
            const int ca = listA[ia];
            double CA[6];
            for (int k = 0; k < 6; ++k) CA[k] = a.ws.clu[6 * (size_t)(cA0 + ca) + k];
            const int ta = 32 * ca + lane;
            const bool validA = ta < ntA;
            double LA[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            if (validA) leaf_box(TA, VwA, ta, env, LA);
            bool hitA = false;
            for (int ib = 0; ib < nB; ++ib) {
                const int cb = listB[ib];
                const double* CB = a.ws.clu + 6 * (size_t)(cB0 + cb);
                if (!overlap(CA, CB)) continue;
                // a leaf pair can only overlap if each leaf overlaps the other leaf's cluster box
                const unsigned amask = __ballot_sync(0xffffffffu, validA && overlap(LA, CB));
                if (!amask) continue;
                const int tb = 32 * cb + lane;
                const bool validB = tb < ntB;
                double LB[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                if (validB) leaf_box(TB, VwB, tb, env, LB);
                unsigned bmask = __ballot_sync(0xffffffffu, validB && overlap(LB, CA));
                unsigned hitB = 0u;
                // every candidate leaf pair is tested once, broadcasting the leaves of the side with fewer
                if (__popc(bmask) <= __popc(amask)) {   // B leaves to the A lanes
                    const bool mine = (amask >> lane) & 1u;
                    while (bmask) {
                        const int jb = __ffs(bmask) - 1;
                        bmask &= bmask - 1;
                        double Lj[6];
                        for (int k = 0; k < 6; ++k) Lj[k] = __shfl_sync(0xffffffffu, LB[k], jb);
                        if (mine && overlap(LA, Lj)) { hitA = true; hitB |= 1u << jb; }
                    }
                    n_ovl += __popc(hitB);
                    hitB = __reduce_or_sync(0xffffffffu, hitB);
                } else {                                 // A leaves to the B lanes
                    const bool mineB = (bmask >> lane) & 1u;
                    unsigned am = amask, hitAbits = 0u;
                    bool bhit = false;
                    while (am) {
                        const int ja = __ffs(am) - 1;
                        am &= am - 1;
                        double Li[6];
                        for (int k = 0; k < 6; ++k) Li[k] = __shfl_sync(0xffffffffu, LA[k], ja);
                        if (mineB && overlap(Li, LB)) { bhit = true; hitAbits |= 1u << ja; ++n_ovl; }
                    }
                    hitB = __ballot_sync(0xffffffffu, bhit);
                    hitAbits = __reduce_or_sync(0xffffffffu, hitAbits);
                    if ((hitAbits >> lane) & 1u) hitA = true;
                }
                if (lane == 0) maskB[ib] |= hitB;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, hitA);
            if (lane == 0) maskA[ia] = bal;
        }
        __syncwarp();
        mid_emit(a, p, nA, nB, listA, listB, maskA, maskB, __reduce_add_sync(0xffffffffu, n_ovl));
        __syncwarp();
    }
}

// The pairs of many cluster pairs, a block each: the leaf boxes of up to kMidCache of B's clusters are computed once into
// shared memory, and every warp takes clusters of A, finds B's clusters that overlap one a lane each, and tests its 32
// leaves against the leaves that overlap it, read by all lanes at once.  (All of k_mid with a warp to every pair: 869 us
// for 55,960 pairs of boxes and 448-triangle spheres, 397 for the 2231 of one pile and 321 for 39,664 lattice pairs; both
// kernels 540, 120 and 211.)
constexpr int kMidCache = 16;
constexpr int kMidWideWarps = 8;
__host__ __device__ inline size_t mid_wide_bytes(int max_clusters) {
    return (size_t)kMidCache * 32 * 6 * sizeof(double) + (size_t)3 * sizeof(uint32_t) * max_clusters;
}
__global__ void __launch_bounds__(32 * kMidWideWarps) k_mid_wide(const StepArgs a, int max_clusters) {
    extern __shared__ __align__(16) char wide_smem[];
    double* leaves = reinterpret_cast<double*>(wide_smem);   // six per leaf of the cached clusters
    uint32_t* maskA = reinterpret_cast<uint32_t*>(wide_smem + (size_t)kMidCache * 32 * 6 * sizeof(double));
    uint32_t* maskB = maskA + max_clusters;
    int16_t* listA = reinterpret_cast<int16_t*>(maskB + max_clusters);
    int16_t* listB = listA + max_clusters;
    __shared__ int next, count[2], overlaps;
    if (a.ws.counters[kAbort]) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n_wide = a.ws.counters[kNWide];
    const double env = a.pr.envelope;
    for (;;) {
        if (threadIdx.x == 0) { next = atomicAdd(a.ws.counters + kWideNext, 1); overlaps = 0; }
        __syncthreads();
        if (next >= n_wide) break;
        const int p = a.ws.pair_cont[next];
        const int A = a.ws.pairs[2 * p], B = a.ws.pairs[2 * p + 1];
        const int cA0 = a.bd.body_c0[A], cB0 = a.bd.body_c0[B];
        const int ntA = a.bd.body_t0[A + 1] - a.bd.body_t0[A], ntB = a.bd.body_t0[B + 1] - a.bd.body_t0[B];
        const int32_t* TA = a.sh.T + 3 * (size_t)a.sh.t_off[a.bd.shape[A]];
        const int32_t* TB = a.sh.T + 3 * (size_t)a.sh.t_off[a.bd.shape[B]];
        const double* VwA = a.ws.Vw + 3 * (size_t)a.bd.body_v0[A];
        const double* VwB = a.ws.Vw + 3 * (size_t)a.bd.body_v0[B];
        if (wid < 2) {   // the clusters of either body that overlap the other's box
            const int me = wid ? B : A, c1 = wid ? cB0 : cA0, nc = a.bd.body_c0[me + 1] - c1;
            const double* other = a.ws.root + 6 * (wid ? A : B);
            int16_t* list = wid ? listB : listA;
            uint32_t* mask = wid ? maskB : maskA;
            int n = 0;
            for (int c0 = 0; c0 < nc; c0 += 32) {
                const int c = c0 + lane;
                const bool ok = c < nc && overlap(a.ws.clu + 6 * (size_t)(c1 + c), other);
                const unsigned bal = __ballot_sync(0xffffffffu, ok);
                if (ok) { const int at = n + __popc(bal & lanemask_lt()); list[at] = (int16_t)c; mask[at] = 0u; }
                n += __popc(bal);
            }
            if (lane == 0) count[wid] = n;
        }
        __syncthreads();
        const int nA = count[0], nB = count[1];
        int n_ovl = 0;
        for (int b0 = 0; b0 < nB; b0 += kMidCache) {
            const int nb = min(kMidCache, nB - b0);
            for (int ib = wid; ib < nb; ib += kMidWideWarps) {
                const int t = 32 * listB[b0 + ib] + lane;
                double L[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};   // overlaps nothing
                if (t < ntB) leaf_box(TB, VwB, t, env, L);
                double2* o = reinterpret_cast<double2*>(leaves + 6 * (32 * ib + lane));
                o[0] = make_double2(L[0], L[1]); o[1] = make_double2(L[2], L[3]); o[2] = make_double2(L[4], L[5]);
            }
            __syncthreads();
            for (int ia = wid; ia < nA; ia += kMidWideWarps) {
                const int ca = listA[ia];
                double CA[6], LA[6];
                for (int k = 0; k < 6; ++k) CA[k] = a.ws.clu[6 * (size_t)(cA0 + ca) + k];
                const int ta = 32 * ca + lane;
                const bool validA = ta < ntA;
                if (validA) leaf_box(TA, VwA, ta, env, LA);
                unsigned todo = __ballot_sync(0xffffffffu, lane < nb && overlap(CA, a.ws.clu + 6 * (size_t)(cB0 + listB[b0 + min(lane, nb - 1)])));
                bool hitA = false;
                for (; todo; todo &= todo - 1) {
                    const int ib = __ffs(todo) - 1;
                    const double* CB = a.ws.clu + 6 * (size_t)(cB0 + listB[b0 + ib]);
                    // a leaf pair can only overlap if each leaf overlaps the other leaf's cluster box
                    const bool mine = validA && overlap(LA, CB);
                    if (!__any_sync(0xffffffffu, mine)) continue;
                    const int tb = 32 * listB[b0 + ib] + lane;
                    unsigned bmask = __ballot_sync(0xffffffffu, tb < ntB && overlap(leaves + 6 * (32 * ib + lane), CA));
                    unsigned hitB = 0u;
                    for (; bmask; bmask &= bmask - 1) {
                        const int jb = __ffs(bmask) - 1;
                        const double2* q = reinterpret_cast<const double2*>(leaves + 6 * (32 * ib + jb));
                        const double2 q0 = q[0], q1 = q[1], q2 = q[2];
                        // the six comparisons of overlap(), without branches
                        const bool ov = mine & !((LA[3] < q0.x) | (q1.y < LA[0]) | (LA[4] < q0.y) | (q2.x < LA[1]) |
                                                 (LA[5] < q1.x) | (q2.y < LA[2]));
                        const unsigned bal = __ballot_sync(0xffffffffu, ov);
                        hitA |= ov;
                        if (bal) hitB |= 1u << jb;
                        n_ovl += __popc(bal);
                    }
                    if (lane == 0 && hitB) atomicOr(maskB + b0 + ib, hitB);
                }
                const unsigned bal = __ballot_sync(0xffffffffu, hitA);
                if (lane == 0) maskA[ia] |= bal;   // the warp's own cluster
            }
            __syncthreads();
        }
        if (lane == 0) atomicAdd(&overlaps, n_ovl);
        __syncthreads();
        if (wid == 0) mid_emit(a, p, nA, nB, listA, listB, maskA, maskB, overlaps);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------------------
// narrow phase (collision_detection.py:87 _compute_contacts): one thread per candidate triangle
// ---------------------------------------------------------------------------------------------------------
constexpr int kAlphas = 32;   // step lengths 2 / (i + 2) of the search, kept in shared memory
// seed and Frank-Wolfe search on one triangle (ps: its corners in the SDF owner's frame) in FP64
// (collision_detection.py:134-165).  Returns the point; n_fw = iterations, trace = the seed (bits 0-1) and
// each iteration's vertex (2 bits each from bit 2)
__device__ __forceinline__ d3 fw_search64(const GridView& g, const double* alphas, const d3* ps, int max_it,
                                          double tol, int& n_fw, uint32_t& trace) {
    // seed: corner with the smallest gradient norm (:136-140); norm(list, axis=1) sums squares unfused
    double gn[3];
    for (int c = 0; c < 3; ++c) {
        const d3 gr = grid_gradient(g, ps[c]);
        gn[c] = sqrt((gr.x * gr.x + gr.y * gr.y) + gr.z * gr.z);
    }
    int best = 0;
    if (gn[1] < gn[best]) best = 1;
    if (gn[2] < gn[best]) best = 2;
    trace = (uint32_t)best;
    d3 x = best == 0 ? ps[0] : (best == 1 ? ps[1] : ps[2]);   // selects keep ps in registers
    n_fw = 0;
    for (int i = 0; i < max_it; ++i) {   // Frank-Wolfe (:144-165)
        ++n_fw;
        // the reference evaluates the same gradient once per corner; one evaluation gives identical values
        const d3 gr = grid_gradient(g, x);
        const double o0 = dot3_np(ps[0], gr), o1 = dot3_np(ps[1], gr), o2 = dot3_np(ps[2], gr);
        int v = 0;
        double ov = o0;
        if (o1 < ov) { v = 1; ov = o1; }
        if (o2 < ov) { v = 2; ov = o2; }
        if (i < 15) trace |= (uint32_t)v << (2 + 2 * i);
        const double alpha = i < kAlphas ? alphas[i] : 2.0 / (double)(i + 2);
        const d3 s = v == 0 ? ps[0] : (v == 1 ? ps[1] : ps[2]);
        x = d3{x.x + alpha * (s.x - x.x), x.y + alpha * (s.y - x.y), x.z + alpha * (s.z - x.z)};
        if (ov > tol) break;
    }
    return x;
}

// the same search with its lookups on the FP32 copy of the grid (profiling bit 2 of the FP32 modes).  The point x and
// the objectives stay FP64; a decision whose margin lies within the FP32 lookups' error bound (an exact tie of
// coplanar corners, a near-tie, an objective next to the tolerance) is taken again on FP64 lookups, so every
// decision, and x, equal fw_search64's.  l64 / l32 count the FP64 and FP32 lookups made.
__device__ __forceinline__ d3 fw_search_f32(const GridView& g, const float* values32, const double* alphas,
                                            const d3* ps, int max_it, double tol, int& n_fw, uint32_t& trace, int& l64, int& l32) {
    double scale = 0.0;   // max over corners of |p|_1: an objective's error is at most err x scale
    for (int c = 0; c < 3; ++c) scale = fmax(scale, fabs(ps[c].x) + fabs(ps[c].y) + fabs(ps[c].z));
    double gn[3], err = 0.0;
    for (int c = 0; c < 3; ++c) {
        double e;
        const d3 gr = grid_gradient_f32(g, values32, ps[c], e);
        gn[c] = sqrt((gr.x * gr.x + gr.y * gr.y) + gr.z * gr.z);
        err = fmax(err, e);
    }
    l32 += 3;
    {   // a seed whose gradient norms lie within 2 sqrt(3) err of another's is chosen on FP64 lookups
        const double lo = fmin(gn[0], fmin(gn[1], gn[2]));
        int close = 0;
        for (int c = 0; c < 3; ++c) close += gn[c] - lo <= 4.0 * 1.7320508075688772 * err;
        if (close > 1) {
            for (int c = 0; c < 3; ++c) {
                const d3 gr = grid_gradient(g, ps[c]);
                gn[c] = sqrt((gr.x * gr.x + gr.y * gr.y) + gr.z * gr.z);
            }
            l64 += 3;
        }
    }
    int best = 0;
    if (gn[1] < gn[best]) best = 1;
    if (gn[2] < gn[best]) best = 2;
    trace = (uint32_t)best;
    d3 x = best == 0 ? ps[0] : (best == 1 ? ps[1] : ps[2]);
    n_fw = 0;
    for (int i = 0; i < max_it; ++i) {
        ++n_fw;
        double e;
        d3 gr = grid_gradient_f32(g, values32, x, e);
        ++l32;
        double o0 = dot3_np(ps[0], gr), o1 = dot3_np(ps[1], gr), o2 = dot3_np(ps[2], gr);
        const double margin = 4.0 * e * scale;
        const double lo = fmin(o0, fmin(o1, o2));
        const int close = (o0 - lo <= margin) + (o1 - lo <= margin) + (o2 - lo <= margin);
        if (close > 1 || fabs(lo - tol) <= margin) {   // decide on the FP64 gradient
            gr = grid_gradient(g, x);
            ++l64;
            o0 = dot3_np(ps[0], gr); o1 = dot3_np(ps[1], gr); o2 = dot3_np(ps[2], gr);
        }
        int v = 0;
        double ov = o0;
        if (o1 < ov) { v = 1; ov = o1; }
        if (o2 < ov) { v = 2; ov = o2; }
        if (i < 15) trace |= (uint32_t)v << (2 + 2 * i);
        const double alpha = i < kAlphas ? alphas[i] : 2.0 / (double)(i + 2);
        const d3 s = v == 0 ? ps[0] : (v == 1 ? ps[1] : ps[2]);
        x = d3{x.x + alpha * (s.x - x.x), x.y + alpha * (s.y - x.y), x.z + alpha * (s.z - x.z)};
        if (ov > tol) break;
    }
    return x;
}

// the plain FP64 search's trace and acceptance for the check of the FP32 search (a call of its
// own, so that it does not raise the registers of the search itself)
__device__ __noinline__ void fw_check64(const GridView& g, const double* alphas, const d3* ps, const double* qB, int max_it, double tol,
                                        double envelope, int& n64, uint32_t& trace64, int& accept64) {
    const d3 x64 = fw_search64(g, alphas, ps, max_it, tol, n64, trace64);
    accept64 = 0;
    if (grid_is_inside(g, x64, 0.5) && grid_value(g, x64) <= envelope)
        accept64 = norm3_np(quat_rotate(qB, grid_gradient(g, x64))) > 0.0;
}

// kF32 (profiling bit 2): the seed and Frank-Wolfe lookups on the FP32 grid copy (near-ties decided on FP64 lookups);
// the acceptance tests (is_inside, phi <= envelope) and the contact's point, normal and gap in FP64 at the point
// found.  It also runs the plain FP64 search and counts, per scene, the candidates whose search decisions or
// acceptance differ (a check of the error bound: zero when it holds).
template <bool kF32>
__global__ void __launch_bounds__(256, 2) k_narrow(const StepArgs a) {
    __shared__ double alphas[kAlphas];
    if (threadIdx.x < kAlphas) alphas[threadIdx.x] = 2.0 / (double)((int)threadIdx.x + 2);
    __syncthreads();
    if (a.ws.counters[kAbort]) return;
    const int n_items = a.ws.counters[kNItems];
    if (n_items > a.caps.item_capacity) {   // the mid phase left the candidates out: the rest of the step is off
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            atomicOr(a.ws.counters + kAbort, RB_STATUS_ITEM_OVERFLOW);
            atomicOr(a.out.status, RB_STATUS_ITEM_OVERFLOW);
        }
        return;
    }
    const int max_it = a.pr.contact_optimization_max_iterations;
    const double tol = a.pr.contact_optimization_tolerance;
    const double envelope = a.pr.envelope;
    for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < n_items; it += gridDim.x * blockDim.x) {
        const int p = a.ws.item_pair[it];
        const unsigned st = (unsigned)a.ws.item_tri[it];
        const int side = st >> 31, tri = st & 0x7fffffff;
        const int A = a.ws.pairs[2 * p], B = a.ws.pairs[2 * p + 1];
        const int mesh = side ? B : A, sdf = side ? A : B;
        const int sm = a.bd.shape[mesh], ss = a.bd.shape[sdf];
        const int32_t* T = a.sh.T + 3 * (size_t)(a.sh.t_off[sm] + tri);
        const double* Vw = a.ws.Vw + 3 * (size_t)a.bd.body_v0[mesh];
        const double* xB = a.bd.x + 7 * sdf;
        const double qB[4] = {xB[3], xB[4], xB[5], xB[6]};
        const double cqB[4] = {qB[0], -qB[1], -qB[2], -qB[3]};
        const d3 rB = d3{xB[0], xB[1], xB[2]};
        d3 ps[3];
        for (int c = 0; c < 3; ++c) {
            const d3 pw = ld3(Vw + 3 * T[c]);
            ps[c] = quat_rotate_row(cqB, sub(pw, rB));   // :120-121
        }
        const GridView g = load_grid(a.sh.grid_meta + 12 * ss, a.sh.grid + a.sh.g_off[ss]);
        int n_fw = 0, lookups = 0, lookups32 = 0;
        uint32_t trace = 0u;
        d3 x;
        if (kF32) {
            x = fw_search_f32(g, a.sh.grid32 + a.sh.g_off[ss], alphas, ps, max_it, tol, n_fw, trace, lookups, lookups32);
        } else {
            x = fw_search64(g, alphas, ps, max_it, tol, n_fw, trace);
            lookups = 3 + n_fw;   // seed gradients + one gradient per Frank-Wolfe iteration
        }
        int flag = 0;
        if (grid_is_inside(g, x, 0.5)) {   // :172 (is_inside default boundary 0.5)
            lookups += 1;
            const double phi = grid_value(g, x);
            if (phi <= envelope) {
                lookups += 1;
                const d3 nb = grid_gradient(g, x);
                const d3 nw = quat_rotate(qB, nb);
                const double ln = norm3_np(nw);
                if (ln > 0.0) {
                    const d3 xr = quat_rotate(qB, x);
                    st3(a.ws.item_p + 3 * (size_t)it, d3{xr.x + rB.x, xr.y + rB.y, xr.z + rB.z});
                    st3(a.ws.item_n + 3 * (size_t)it, d3{nw.x / ln, nw.y / ln, nw.z / ln});
                    a.ws.item_g[it] = phi;
                    flag = 1;
                    if (fabs(1.0 - norm3_np(d3{nw.x / ln, nw.y / ln, nw.z / ln})) > 0.1)   // types.py:293
                        atomicOr(a.out.status, RB_STATUS_NONUNIT_NORMAL);
                }
            }
        }
        a.ws.item_flag[it] = flag;
        if (a.pr.profiling) {   // statistics for the bandwidth accounting (lookups per scene) and decision flips
            const int s = scene_of(a.bd.scene_start, a.bd.n_scenes, A);
            atomicAdd(&a.out.stats[s].n_grid_lookups, lookups);
            if (kF32) {   // the check against the plain FP64 search
                atomicAdd(&a.out.stats[s].n_grid_lookups32, lookups32);
                int n64 = 0, accept64 = 0;
                uint32_t trace64 = 0u;
                fw_check64(g, alphas, ps, qB, max_it, tol, envelope, n64, trace64, accept64);
                if (n64 != n_fw || trace64 != trace) atomicAdd(&a.out.stats[s].n_search_flips, 1);
                if (accept64 != flag) atomicAdd(&a.out.stats[s].n_accept_flips, 1);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// contact reduction (collision_detection.py:255): a contact is dropped when an earlier contact of the same
// unordered body pair has the identical position.  Contacts of one body pair are contiguous (one pair list
// entry), so the test runs per pair.
// ---------------------------------------------------------------------------------------------------------
// Few candidates of a pair are accepted (of 4.3 million in 55,960 pairs 94,817 are kept), so a warp collects the
// accepted ones' positions first, in order, and compares each with the kept ones before it; the kept candidates'
// indices go to the pair's room in item_pair, which is not read any more, for the write pass to go over alone.
// (Comparing every chunk of candidates with every earlier chunk, and scanning all of them again in the write pass,
// took 316 and 119 us; this 72 and 42.)
constexpr int kDedupRoom = 64;   // accepted candidates a warp holds at a time
__global__ void __launch_bounds__(kBlock) k_dedup(const StepArgs a) {
    __shared__ double pos[kWarpsPerBlock][kDedupRoom][3];
    __shared__ int index[kWarpsPerBlock][kDedupRoom];
    if (a.ws.counters[kAbort]) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n_pairs = a.ws.counters[kNPairs];
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < n_pairs; p += (gridDim.x * blockDim.x) >> 5) {
        const int i0 = a.ws.pair_items[p], i1 = i0 + a.ws.pair_n_items[p];
        int kept = 0;
        for (int c0 = i0; c0 < i1;) {
            // the next accepted candidates, as many whole chunks of 32 as there is room for
            int n = 0;
            for (; c0 < i1 && n <= kDedupRoom - 32; c0 += 32) {
                const int i = c0 + lane;
                const bool mine = i < i1 && a.ws.item_flag[i] != 0;
                const unsigned bal = __ballot_sync(0xffffffffu, mine);
                if (mine) {
                    const int at = n + __popc(bal & lanemask_lt());
                    const double* q = a.ws.item_p + 3 * (size_t)i;
                    pos[wid][at][0] = q[0]; pos[wid][at][1] = q[1]; pos[wid][at][2] = q[2];
                    index[wid][at] = i;
                }
                n += __popc(bal);
            }
            __syncwarp();
            for (int j0 = 0; j0 < n; j0 += 32) {
                const int j = j0 + lane;
                bool keep = j < n;
                const double px = pos[wid][keep ? j : 0][0], py = pos[wid][keep ? j : 0][1], pz = pos[wid][keep ? j : 0][2];
                for (int e = 0; e < kept; ++e) {   // those kept in earlier chunks
                    const double* q = a.ws.item_p + 3 * (size_t)a.ws.item_pair[i0 + e];
                    if (q[0] == px && q[1] == py && q[2] == pz) keep = false;
                }
                const int own = min(32, n - j0);
                for (int e = 0; e < own; ++e)      // and the earlier ones of this chunk (a dropped one equals a kept one)
                    if (e < lane && pos[wid][j0 + e][0] == px && pos[wid][j0 + e][1] == py && pos[wid][j0 + e][2] == pz)
                        keep = false;
                const unsigned bal = __ballot_sync(0xffffffffu, keep);
                if (keep) a.ws.item_pair[i0 + kept + __popc(bal & lanemask_lt())] = index[wid][j];
                kept += __popc(bal);
                __syncwarp();
            }
        }
        if (lane == 0) a.ws.pair_cont[p] = kept;
    }
}

// the kept candidates become contacts, in order: eight lanes a pair (most have fewer than eight contacts)
__global__ void k_emit(const StepArgs a) {
    if (a.ws.counters[kAbort]) return;
    const int n_pairs = a.ws.counters[kNPairs];
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; p < n_pairs; p += (gridDim.x * blockDim.x) >> 3) {
        const int base = a.ws.pair_cont[p], end = min(a.ws.pair_cont[p + 1], a.caps.contact_capacity);
        if (base >= end) continue;
        const int i0 = a.ws.pair_items[p];
        const int A = a.ws.pairs[2 * p], B = a.ws.pairs[2 * p + 1];
        for (int k = base + (threadIdx.x & 7); k < end; k += 8) {
            const int i = a.ws.item_pair[i0 + k - base];
            const int tri = a.ws.item_tri[i];
            const int side = (unsigned)tri >> 31;
            a.out.contact_ids[2 * k] = side ? A : B;     // ContactPoint(bodyB_sdf_owner, bodyA_mesh_owner, ...)
            a.out.contact_ids[2 * k + 1] = side ? B : A;
            for (int c = 0; c < 3; ++c) {
                a.out.contact_p[3 * (size_t)k + c] = a.ws.item_p[3 * (size_t)i + c];
                a.out.contact_n[3 * (size_t)k + c] = a.ws.item_n[3 * (size_t)i + c];
            }
            a.out.contact_g[k] = a.ws.item_g[i];
            // key of the contact for warm starting: contacts come out in ascending key order
            a.ws.ckey[2 * (size_t)k] = ((int64_t)A << 31) | (int64_t)B;
            a.ws.ckey[2 * (size_t)k + 1] = (int64_t)(side << 30) | (int64_t)(tri & 0x7fffffff);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// contact problem (contacts.py:31 initialize): thread per contact
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ double jrow_dot(const double* Jr, const double* wlo, const double* whi) {
    double s = 0.0;
    for (int c = 0; c < 6; ++c) s += Jr[c] * wlo[c];
    for (int c = 0; c < 6; ++c) s += Jr[6 + c] * whi[c];
    return s;
}

// Layout of a contact's 4 x 12 blocks of J and of W J^T (48 doubles, columns: six of the lo body, six of the hi
// body).  The solver reads them by quads: lane q takes row q of J, and of W J^T the columns 2q, 2q + 1 and 8 + q in
// all four rows, 12 doubles each as six 16-byte pieces.  Piece j of the four lanes is contiguous (64 bytes), so a
// warp's load of one piece touches one line per contact; with rows stored whole the 32 lanes fell on up to 28 lines
// (4096-body lattice, eight warps sweeping: 4948 against 4193 cycles a level; one warp on the 32-box tower is the
// same either way).
__device__ __forceinline__ int j_at(int row, int col) { return 8 * (col >> 1) + 2 * row + (col & 1); }
__device__ __forceinline__ int w_at(int row, int col) {
    const int q = col < 8 ? col >> 1 : col - 8, p = col < 8 ? col & 1 : 2;
    return 16 * p + 8 * (row >> 1) + 2 * q + (row & 1);
}
// column col of W J^T (rows 0..3) as two 16-byte pieces
__device__ __forceinline__ void w_column(const double* WJT, int k, int col, double* o) {
    const double2* W = reinterpret_cast<const double2*>(WJT + 48 * (size_t)k + w_at(0, col));
    const double2 t = W[0], u = W[4];
    o[0] = t.x; o[1] = t.y; o[2] = u.x; o[3] = u.y;
}

__global__ void k_contacts(const StepArgs a) {
    // one thread per (contact, row): row q's J and W J^T blocks, b, Delassus diagonal, r and start impulse;
    // the row-0 thread also writes the contact's body pair and mu
    if (a.ws.counters[kAbort]) return;
    const int K = a.ws.counters[kNContacts];
    const double dt = a.pr.dt;
    double r_scale = a.pr.scheme == RB_SCHEME_RIGID_GS ? 1.0 : 0.1;   // solver_interface.py:48
    if (a.pr.termination == RB_TERMINATE_RESIDUAL_FIXED_R && a.pr.relaxation > 0.0) r_scale *= a.pr.relaxation;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 4 * K; t += gridDim.x * blockDim.x) {
        const int k = t >> 2, row = t & 3;
        const int A = a.out.contact_ids[2 * k], B = a.out.contact_ids[2 * k + 1];
        const d3 p = ld3(a.out.contact_p + 3 * k);
        const d3 rA = sub(p, ld3(a.bd.x + 7 * A)), rB = sub(p, ld3(a.bd.x + 7 * B));
        d3 vs, vt, vn;
        make_orthonormal_vectors(ld3(a.out.contact_n + 3 * k), vs, vt, vn);   // (t, b, n)
        const int lo = min(A, B), hi = max(A, B);
        double JA[6], JB[6], J[12], W[12];
        if (row < 3) {   // contacts.py:140-147
            const d3 d = row == 0 ? vn : (row == 1 ? vs : vt);
            const d3 ca = cross_np(rA, d), cb = cross_np(rB, d);
            JA[0] = -d.x; JA[1] = -d.y; JA[2] = -d.z; JA[3] = -ca.x; JA[4] = -ca.y; JA[5] = -ca.z;
            JB[0] = d.x; JB[1] = d.y; JB[2] = d.z; JB[3] = cb.x; JB[4] = cb.y; JB[5] = cb.z;
        } else {
            JA[0] = -0.0; JA[1] = -0.0; JA[2] = -0.0; JA[3] = -vn.x; JA[4] = -vn.y; JA[5] = -vn.z;
            JB[0] = 0.0; JB[1] = 0.0; JB[2] = 0.0; JB[3] = vn.x; JB[4] = vn.y; JB[5] = vn.z;
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) { J[i] = A == lo ? JA[i] : JB[i]; J[6 + i] = A == lo ? JB[i] : JA[i]; }
        bool hasw[2];
#pragma unroll
        for (int side = 0; side < 2; ++side) {   // WJT = W J^T (bsr_matmat order)
            const int bb = side ? hi : lo;
            hasw[side] = !a.bd.fixed[bb];
            const double m = hasw[side] ? 1.0 / a.bd.mass[bb] : 0.0;
            const double* Wi = a.ws.Winv + 9 * bb;
            const double* Jr = J + 6 * side;
            double* Wr = W + 6 * side;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                double s = 0.0;
                s += (i == 0 ? m : 0.0) * Jr[0];
                s += (i == 1 ? m : 0.0) * Jr[1];
                s += (i == 2 ? m : 0.0) * Jr[2];
                double tt = 0.0;
                tt += Wi[3 * i + 0] * Jr[3];
                tt += Wi[3 * i + 1] * Jr[4];
                tt += Wi[3 * i + 2] * Jr[5];
                Wr[i] = hasw[side] ? s : 0.0;
                Wr[3 + i] = hasw[side] ? tt : 0.0;
            }
        }
        {
            double2* Jk = reinterpret_cast<double2*>(a.ws.J + 48 * (size_t)k + j_at(row, 0));
#pragma unroll
            for (int j = 0; j < 6; ++j) Jk[4 * j] = make_double2(J[2 * j], J[2 * j + 1]);
            double* Wk = a.ws.WJT + 48 * (size_t)k;
#pragma unroll
            for (int c = 0; c < 12; ++c) Wk[w_at(row, c)] = W[c];
        }
        // b = (1 + e) v + J (dt W f_ext) + g   (contacts.py:46)
        const int sc = scene_of(a.bd.scene_start, a.bd.n_scenes, A);
        const int M = a.bd.scene_material_count[sc];
        const int entry = a.bd.scene_material_offset[sc] + a.bd.material[A] * M + a.bd.material[B];
        const double eps = a.pr.use_bounce ? a.bd.material_eps[entry] : 0.0;
        const double* ulo = a.bd.u + 6 * lo;
        const double* uhi = a.bd.u + 6 * hi;
        const double* dlo = a.ws.du + 6 * lo;
        const double* dhi = a.ws.du + 6 * hi;
        const double vrow = jrow_dot(J, ulo, uhi);
        double gk0 = 0.0;
        if (row == 0 && a.pr.use_pre_stabilization) {   // contacts.py:188 _compute_error_vector
            const double gap = a.out.contact_g[k];
            const double rate = a.pr.gap_reduction / dt;
            const double upper = -a.pr.max_gap_value / dt;
            const double lower = -a.pr.min_gap_value;
            if (gap < lower && vrow <= 0.0) {
                const double tg = rate * gap;
                gk0 = upper > tg ? upper : tg;
            }
        }
        const double jd = jrow_dot(J, dlo, dhi);
        const double e = row == 0 ? eps : 0.0;
        a.ws.b[4 * k + row] = ((1.0 + e) * vrow + jd) + gk0;
        // Delassus diagonal: reduceat over the nonzero products J .* WJT^T in column order (contacts.py:49)
        double prods[12];
        int m = 0;
#pragma unroll
        for (int c = 0; c < 12; ++c) {
            if (!hasw[c / 6]) continue;
            const double pr = J[c] * W[c];
            if (pr != 0.0) prods[m++] = pr;
        }
        double dg = np_reduce_sum(prods, m);
        if (dg == 0.0) dg = 1.0;
        a.ws.diag[4 * k + row] = dg;
        a.ws.r[4 * k + row] = r_scale / dg;
        double x0 = 0.0;
        if (a.pr.warm_start && a.out.cache_count) {   // previous impulse of the same contact (binary search)
            const int64_t k1 = a.ws.ckey[2 * k], k2 = a.ws.ckey[2 * k + 1];
            int lo_i = 0, hi_i = min(*a.out.cache_count, a.caps.contact_capacity);
            while (lo_i < hi_i) {
                const int mid = (lo_i + hi_i) >> 1;
                const int64_t m1 = a.out.cache_key[2 * mid], m2 = a.out.cache_key[2 * mid + 1];
                if (m1 < k1 || (m1 == k1 && m2 < k2)) lo_i = mid + 1; else hi_i = mid;
            }
            if (lo_i < *a.out.cache_count && a.out.cache_key[2 * lo_i] == k1 && a.out.cache_key[2 * lo_i + 1] == k2)
                x0 = a.out.cache_sol[4 * lo_i + row];
        }
        a.ws.x[4 * k + row] = x0;
        a.out.contact_sol[4 * k + row] = x0;
        if (row == 0) {
            a.ws.lohi[2 * k] = lo;
            a.ws.lohi[2 * k + 1] = hi;
            if (hasw[0]) atomicAdd(a.ws.bc_ptr + lo, 1);
            if (hasw[1]) atomicAdd(a.ws.bc_ptr + hi, 1);
            a.ws.mu[k] = a.bd.material_mu[3 * entry];
        }
    }
}

// per-body contact lists, ascending contact index (the column order of the SciPy products): counted by k_contacts,
// filled in any order, then sorted.  A fixed body has no list, and its contacts no predecessor on it.
__global__ void k_body_contacts_fill(const StepArgs a) {
    if (a.ws.counters[kAbort]) return;
    const int K = a.ws.counters[kNContacts];
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < 2 * K; c += gridDim.x * blockDim.x) {   // k << 1 | side
        const int b = a.ws.lohi[c];
        if (a.bd.fixed[b]) { a.ws.cpred[c] = -1; continue; }
        a.ws.blist32[a.ws.bc_ptr[b] + atomicAdd(a.ws.bc_fill + b, 1)] = (uint32_t)c;
    }
}
// a warp per body: an entry's place is the number of smaller ones (one thread's insertion sort took 357 us where the
// busiest of 37,148 bodies has ~100 contacts, this 16); then the predecessor of each contact along this body, the
// chain the Gauss-Seidel levels follow
__global__ void k_body_contacts_sort(const StepArgs a) {
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (b >= a.bd.n_bodies || a.ws.counters[kAbort]) return;
    const int e0 = a.ws.bc_ptr[b], n = a.ws.bc_ptr[b + 1] - e0;
    const uint32_t* in = a.ws.blist32 + e0;
    int32_t* out = a.ws.bc_list + e0;
    for (int c0 = 0; c0 < n; c0 += 32) {
        const uint32_t v = c0 + lane < n ? in[c0 + lane] : 0xffffffffu;
        int rank = 0;
        for (int d0 = 0; d0 < n; d0 += 32) {
            const uint32_t u = d0 + lane < n ? in[d0 + lane] : 0xffffffffu;
            const int m = min(32, n - d0);
            for (int e = 0; e < m; ++e) rank += __shfl_sync(0xffffffffu, u, e) < v;
        }
        if (c0 + lane < n) out[rank] = (int32_t)v;
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) a.ws.cpred[out[i]] = i > 0 ? out[i - 1] >> 1 : -1;
}

// component d of (WJT x) of a body, over its contacts bc_list[e0 .. e1): sequential over the contacts (ascending)
// and their four rows.  The loads of four contacts are issued before their products are accumulated in order.
__device__ __forceinline__ double body_wjt_dot(const Workspace& ws, int e0, int e1, int d, const double* x) {
    double s = 0.0;
    int e = e0;
    for (; e + 4 <= e1; e += 4) {
        int code[4];
        double W[4][4], xv[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) code[j] = ws.bc_list[e + j];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = code[j] >> 1;
            w_column(ws.WJT, k, 6 * (code[j] & 1) + d, W[j]);
#pragma unroll
            for (int q = 0; q < 4; ++q) xv[j][q] = x[4 * (size_t)k + q];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) s += W[j][q] * xv[j][q];
    }
    for (; e < e1; ++e) {
        const int code = ws.bc_list[e], k = code >> 1;
        double W[4];
        w_column(ws.WJT, k, 6 * (code & 1) + d, W);
#pragma unroll
        for (int q = 0; q < 4; ++q) s += W[q] * x[4 * (size_t)k + q];
    }
    return s;
}
// six lanes of a warp per body, one velocity component each: this lane's body (-1: none) and component
__device__ __forceinline__ int body_of_six(int n_bodies, int& d) {
    const int lane = threadIdx.x & 31, slot = lane / 6;
    d = lane - 6 * slot;
    const int b = 5 * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) + slot;
    return slot < 5 && b < n_bodies ? b : -1;
}
// the six components held by the lanes of this lane's body
__device__ __forceinline__ void gather_six(double v, double* o) {
    const int lane = threadIdx.x & 31, base = min(lane / 6, 4) * 6;
#pragma unroll
    for (int i = 0; i < 6; ++i) o[i] = __shfl_sync(0xffffffffu, v, base + i);
}

// ---------------------------------------------------------------------------------------------------------
// solver: one thread group per scene -- a warp for small scenes (warp-synchronous, many scenes per SM), a
// block for large ones.  Every member of the group evaluates the solver's control logic redundantly from the
// same reduced values, so no broadcast through shared memory is needed.
// ---------------------------------------------------------------------------------------------------------
struct SceneRange { int b0, b1, c0, c1; };
__device__ __forceinline__ SceneRange scene_range(const StepArgs& a, int s) {
    SceneRange R;
    R.b0 = a.bd.scene_start[s];
    R.b1 = a.bd.scene_start[s + 1];
    // contacts follow the pair order, pairs follow the body order
    const int p0 = a.ws.pair_cnt[R.b0], p1 = a.ws.pair_cnt[R.b1];
    R.c0 = a.ws.pair_cont[p0];
    R.c1 = a.ws.pair_cont[p1];
    return R;
}

// the larger one, or NaN once either is (v: the largest so far)
__device__ __forceinline__ double nanmax(double v, double t) { return (t > v || t != t) ? t : v; }
__device__ __forceinline__ float nanmax(float v, float t) { return (t > v || t != t) ? t : v; }

struct WarpGroup {
    __device__ __forceinline__ int rank() const { return threadIdx.x & 31; }
    __device__ __forceinline__ int size() const { return 32; }
    __device__ __forceinline__ void sync() const { __syncwarp(); }
    __device__ __forceinline__ bool any(bool p) const { __syncwarp(); return __any_sync(0xffffffffu, p); }
    __device__ __forceinline__ double max(double v) const {
        for (int o = 16; o > 0; o >>= 1) v = nanmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
    __device__ __forceinline__ int imax(int v) const {
        for (int o = 16; o > 0; o >>= 1) v = ::max(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
    __device__ __forceinline__ void max2(double& u, double& v) const { u = max(u); v = max(v); }
    // exclusive prefix sum of the members' values and their total
    __device__ __forceinline__ int scan(int v, int& total) const {
        const int lane = threadIdx.x & 31;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        total = __shfl_sync(0xffffffffu, incl, 31);
        return incl - v;
    }
};

struct BlockGroup {
    double* red;   // 32 doubles of shared memory
    int* ired;     // 33 ints of shared memory
    __device__ __forceinline__ int rank() const { return threadIdx.x; }
    __device__ __forceinline__ int size() const { return blockDim.x; }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    __device__ __forceinline__ bool any(bool p) const { return __syncthreads_or(p); }
    __device__ double max(double v) const {
        double w = 0.0;
        max2(v, w);
        return v;
    }
    // two maxima with one pair of barriers (up to sixteen warps)
    __device__ void max2(double& u, double& v) const {
        for (int o = 16; o > 0; o >>= 1) {
            u = nanmax(u, __shfl_xor_sync(0xffffffffu, u, o));
            v = nanmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        }
        const int wid = threadIdx.x >> 5;
        if ((threadIdx.x & 31) == 0) { red[2 * wid] = u; red[2 * wid + 1] = v; }
        __syncthreads();
        u = red[0]; v = red[1];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) { u = nanmax(u, red[2 * k]); v = nanmax(v, red[2 * k + 1]); }
        __syncthreads();
    }
    __device__ int imax(int v) const {
        for (int o = 16; o > 0; o >>= 1) v = ::max(v, __shfl_xor_sync(0xffffffffu, v, o));
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        __syncthreads();
        if (lane == 0) ired[wid] = v;
        __syncthreads();
        int m = ired[0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) m = ::max(m, ired[k]);
        __syncthreads();
        return m;
    }
    __device__ int scan(int v, int& total) const {
        int warp_total;
        int at = WarpGroup{}.scan(v, warp_total);
        const int wid = threadIdx.x >> 5;
        if ((threadIdx.x & 31) == 0) ired[wid] = warp_total;
        __syncthreads();
        total = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            if (k < wid) at += ired[k];
            total += ired[k];
        }
        __syncthreads();
        return at;
    }
};

// the first `threads` threads of a block (a multiple of 32), with a barrier of their own
struct SubGroup {
    int threads;
    __device__ __forceinline__ int rank() const { return threadIdx.x; }
    __device__ __forceinline__ int size() const { return threads; }
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }
};

// two groups of threads by turns: group 0 ends its turn at barrier 1 and waits for the other's end at barrier 2, group 1
// the other way round (written with their numbers, so that a block keeps three barriers and not all sixteen)
__device__ __forceinline__ void turn_wait(int group, int threads) {
    if (group) asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
    else asm volatile("bar.sync 2, %0;" ::"r"(threads) : "memory");
}
__device__ __forceinline__ void turn_done(int group, int threads) {
    if (group) asm volatile("bar.arrive 2, %0;" ::"r"(threads) : "memory");
    else asm volatile("bar.arrive 1, %0;" ::"r"(threads) : "memory");
}

// The working set of one scene's FP64 solve.  Only the free bodies with contacts have accumulators w = WJT x that
// change; they are numbered ("slots", in any order) and their accumulators lie together, in shared memory when they
// fit, else in global memory, followed by one zero slot that stands for every fixed body (a scene whose contacts
// touch a fixed body has at most nb - 1 free ones, so nb slots hold them all).  In a lattice of 4096 bodies 547
// contacts touch 302 of them.
//   span  per slot the body's range in bc_list (at the scene's place of the w2 array)
//   meta  per contact, in level order: contact, 6 x the slots of its lo and hi bodies, flags (bit 0 / 1: lo / hi is
//         free; bit 2: an idle quad's stand-in), in the compact FP32 rows' room (c32), which no FP64 solve reads
//   steps the sweep's sequence of steps, after the metas there (a meta and a step take 24 of a row's 208 bytes)
struct Solve64 {
    double* w;
    const int2* span;
    const int4* meta;
    const int2* steps;
    const int32_t* bc_list;
    const double *J, *WJT, *mu;
    int K, n_touched, n_steps;
    int warps;       // warps that sweep a step (a block's; 1 for a warp)
    bool turns;      // two groups of them by turns
    bool w_shared;   // w lies in shared memory
};
constexpr int kMetaIdle = 4;
constexpr int kStepEnds = 1 << 16;
// accumulators i and i + 1 (i even), and single ones, by their own space's loads and stores
template <bool kShared>
struct W64 {
    double* w;
    uint32_t s;
    __device__ __forceinline__ explicit W64(double* p) : w(p), s(kShared ? (uint32_t)__cvta_generic_to_shared(p) : 0u) {}
    __device__ __forceinline__ double2 pair(int i) const {
        double2 v;
        if (kShared) asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(s + 8 * i) : "memory");
        else v = *reinterpret_cast<const double2*>(w + i);
        return v;
    }
    __device__ __forceinline__ double one(int i) const {
        double v;
        if (kShared) asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(s + 8 * i) : "memory");
        else v = w[i];
        return v;
    }
    __device__ __forceinline__ void set(int i, double v) const {
        if (kShared) asm volatile("st.shared.f64 [%0], %1;" ::"r"(s + 8 * i), "d"(v) : "memory");
        else w[i] = v;
    }
    __device__ __forceinline__ void set(int i, double2 v) const {
        if (kShared) asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(s + 8 * i), "d"(v.x), "d"(v.y) : "memory");
        else *reinterpret_cast<double2*>(w + i) = v;
    }
};

// numbers the scene's touched bodies in body order: body -> slot in bc_fill (free once bc_list is filled), and
// put(slot, body, e0, e1) for each.  A member takes a run of bodies, counts and then puts.  Returns their number.
template <class G, class Put>
__device__ __forceinline__ int scene_touched(const StepArgs& a, const G& g, const SceneRange& R, Put put) {
    const int run = (R.b1 - R.b0 + g.size() - 1) / g.size();
    const int b0 = min(R.b0 + g.rank() * run, R.b1), b1 = min(b0 + run, R.b1);
    int n = 0, total;
#pragma unroll 4
    for (int b = b0; b < b1; ++b) n += a.ws.bc_ptr[b + 1] > a.ws.bc_ptr[b];   // fixed bodies have no list entries
    int at = g.scan(n, total);
    if (n > 0)
        for (int b = b0; b < b1; ++b) {
            const int e0 = a.ws.bc_ptr[b], e1 = a.ws.bc_ptr[b + 1];
            if (e1 > e0) { a.ws.bc_fill[b] = at; put(at++, b, e0, e1); }
        }
    return total;
}

// Warps that sweep a scene, eight contacts each, and whether two groups of them do so by turns: the choice with the least
// cost over the scene's levels (ptr).  A step (a run of a level's contacts that the warps take at once) costs 1150 cycles
// with one warp, or 750 by turns, and 100 more for every further warp: their FP64 and load instructions hold one another
// up even where they have no contact (64-box lattice: 1420 with three; 4096-body lattice: 1870 with eight).  Every warp
// of the block counts for itself.
__device__ __forceinline__ int sweep_warps(const int* ptr, int L, int max_warps, bool& turns) {
    int steps[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int l = threadIdx.x & 31; l < L; l += 32) {
        const int n = ptr[l + 1] - ptr[l];
#pragma unroll
        for (int w = 0; w < 8; ++w) steps[w] += (n + 8 * w + 7) / (8 * w + 8);
    }
    int best = 1, cost = INT_MAX;
    turns = false;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        const int n = __reduce_add_sync(0xffffffffu, steps[w]);
        const int together = n * (23 + 2 * w), by_turns = n * (15 + 2 * w);
        if (w < max_warps && together < cost) { cost = together; best = w + 1; turns = false; }
        if (2 * w + 1 < max_warps && by_turns < cost) { cost = by_turns; best = w + 1; turns = true; }
    }
    return best;
}

// The steps of a sweep: a level of up to `narrow` contacts is one step, a wider one is cut into runs of `run`;
// put(j, first position, contacts, whether the level ends, whether it is a wide one).  Every warp of the group counts,
// its first one puts.  Returns their number.
template <class G, class Put>
__device__ __forceinline__ int sweep_steps(const G& g, const int* ptr, int L, int narrow, int run, Put put) {
    int n_steps = 0;
    for (int l0 = 0; l0 < L; l0 += 32) {
        const int lane = threadIdx.x & 31, l = l0 + lane;
        const int st = l < L ? ptr[l] : 0, n = l < L ? ptr[l + 1] - st : 0;
        const int parts = n <= narrow ? min(n, 1) : (n + run - 1) / run;
        int at = parts;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += t;
        }
        const int total = __shfl_sync(0xffffffffu, at, 31);
        if (g.rank() < 32)
            for (int p = 0; p < parts; ++p)
                put(n_steps + at - parts + p, st + p * run, min(run, n - p * run), p + 1 == parts, n > narrow);
        n_steps += total;
    }
    return n_steps;
}

// the scene's working set once its contact order is known (L levels; 0: ascending order, no sweeps); w_smem holds
// smem_bodies accumulators
template <class G>
__device__ __forceinline__ Solve64 scene_setup64(const StepArgs& a, const G& g, const SceneRange& R, int s, int L,
                                                 double* w_smem, int smem_bodies) {
    const int* order = L > 0 ? a.ws.lev_order + R.c0 : nullptr;
    Solve64 v;
    v.K = R.c1 - R.c0;
    int2* span = reinterpret_cast<int2*>(a.ws.w2 + 6 * (size_t)R.b0);
    v.n_touched = scene_touched(a, g, R, [&](int at, int, int e0, int e1) { span[at] = make_int2(e0, e1); });
    g.sync();
    const int zero = v.n_touched < R.b1 - R.b0 ? v.n_touched : 0;
    v.w_shared = w_smem != nullptr && v.n_touched + 1 <= smem_bodies;
    v.w = v.w_shared ? w_smem : a.ws.w + 6 * (size_t)R.b0;
    v.span = span;
    int4* meta = reinterpret_cast<int4*>(a.ws.c32 + kS32Floats * (size_t)R.c0);
    v.meta = meta;
    v.bc_list = a.ws.bc_list;
    v.J = a.ws.J; v.WJT = a.ws.WJT; v.mu = a.ws.mu;
    for (int i = g.rank(); i < v.K; i += g.size()) {
        const int k = order ? order[i] : R.c0 + i;
        const int lo = a.ws.lohi[2 * k], hi = a.ws.lohi[2 * k + 1];
        const bool fl = !a.bd.fixed[lo], fh = !a.bd.fixed[hi];
        meta[i] = make_int4(k, 6 * (fl ? a.ws.bc_fill[lo] : zero), 6 * (fh ? a.ws.bc_fill[hi] : zero),
                            (fl ? 1 : 0) | (fh ? 2 : 0));
    }
    if (zero == v.n_touched && g.rank() < 6) v.w[6 * zero + g.rank()] = 0.0;
    int2* steps = reinterpret_cast<int2*>(meta + v.K);
    v.steps = steps;
    const int* ptr = a.ws.lev_ptr + R.c0 + s;
    v.warps = 1;
    v.turns = false;
    if (g.size() > 32) v.warps = sweep_warps(ptr, L, g.size() >> 5, v.turns);
    v.n_steps = sweep_steps(g, ptr, L, 8 * v.warps, 8 * v.warps, [&](int at, int start, int count, bool ends, bool) {
        steps[at] = make_int2(start, count | (ends && !v.turns ? kStepEnds : 0));
    });
    g.sync();
    return v;
}

// w = WJT x, sequential over each body's contacts (the order of WJT.dot(x)).  A component's chain is 4 additions a
// contact, so six lanes take a body, one component each; the next contacts' list codes are loaded while the current ones' products are accumulated in order.
constexpr int kWjtAhead = 4;
template <class G>
__device__ __noinline__ void scene_wjt(const G g, const Solve64 v, const double* x) {
    const int lane = g.rank() & 31, slot = lane / 6, d = lane - 6 * slot;
    const int stride = 5 * (g.size() >> 5);
    if (slot < 5) {
        int i = 5 * (g.rank() >> 5) + slot;
        int2 span = i < v.n_touched ? v.span[i] : make_int2(0, 0);
        int code[kWjtAhead];
#pragma unroll
        for (int j = 0; j < kWjtAhead; ++j) code[j] = span.x + j < span.y ? v.bc_list[span.x + j] : -1;
        while (i < v.n_touched) {
            const int2 ahead = i + stride < v.n_touched ? v.span[i + stride] : make_int2(0, 0);
            double t = 0.0;
            for (int e = span.x; e < span.y; e += kWjtAhead) {
                double Wv[kWjtAhead][4], xv[kWjtAhead][4];
                bool on[kWjtAhead];
#pragma unroll
                for (int j = 0; j < kWjtAhead; ++j) {
                    on[j] = code[j] >= 0;
                    if (!on[j]) continue;
                    const int k = code[j] >> 1;
                    w_column(v.WJT, k, 6 * (code[j] & 1) + d, Wv[j]);
                    const double2* xk = reinterpret_cast<const double2*>(x + 4 * (size_t)k);
                    const double2 t0 = xk[0], t1 = xk[1];
                    xv[j][0] = t0.x; xv[j][1] = t0.y; xv[j][2] = t1.x; xv[j][3] = t1.y;
                }
                const bool same = e + kWjtAhead < span.y;   // this body's next contacts, else the next body's first
                const int e2 = same ? e + kWjtAhead : ahead.x, end2 = same ? span.y : ahead.y;
#pragma unroll
                for (int j = 0; j < kWjtAhead; ++j) code[j] = e2 + j < end2 ? v.bc_list[e2 + j] : -1;
#pragma unroll
                for (int j = 0; j < kWjtAhead; ++j)
                    if (on[j])
#pragma unroll
                        for (int q = 0; q < 4; ++q) t += Wv[j][q] * xv[j][q];
            }
            v.w[6 * i + d] = t;
            span = ahead;
            i += stride;
        }
    }
    g.sync();
}

// what lane q of a quad (four neighbouring lanes, one contact) reads of its contact ahead of time: row q of J with
// its b and r (or, for the residual, the diagonal), the four impulses and mu
struct Contact64 {
    double J[12], x[4], xq, b, r, mu;
    int4 me;
};
__device__ __forceinline__ void contact64_load(const Solve64& v, int4 me, int q, const double* b, const double* r,
                                               const double* x, Contact64& c) {
    const size_t k = (size_t)me.x;
    c.me = me;
    const double2* J = reinterpret_cast<const double2*>(v.J + 48 * k + 2 * q);
#pragma unroll
    for (int i = 0; i < 6; ++i) { const double2 t = J[4 * i]; c.J[2 * i] = t.x; c.J[2 * i + 1] = t.y; }
    c.b = b[4 * k + q];
    c.r = r[4 * k + q];
    const double2* xk = reinterpret_cast<const double2*>(x + 4 * k);
    const double2 x0 = xk[0], x1 = xk[1];
    c.x[0] = x0.x; c.x[1] = x0.y; c.x[2] = x1.x; c.x[3] = x1.y;
    c.xq = x[4 * k + q];
    c.mu = v.mu[k];
}
// the meta of position i of the level order, or an idle quad's stand-in (any contact, nothing written) past end
__device__ __forceinline__ int4 contact64_meta(const Solve64& v, int i, int end) {
    int4 me = v.meta[min(i, v.K - 1)];
    if (i >= end) me.w = kMetaIdle;
    return me;
}
// J_q . [w_lo; w_hi] of the quad's contact (jrow_dot's order), the accumulators read as 16-byte pairs
template <bool kShared>
__device__ __forceinline__ double contact64_jw(const Contact64& c, const W64<kShared> w) {
    double u[12];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double2 l = w.pair(c.me.y + 2 * i), h = w.pair(c.me.z + 2 * i);
        u[2 * i] = l.x; u[2 * i + 1] = l.y; u[6 + 2 * i] = h.x; u[7 + 2 * i] = h.y;
    }
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 12; ++i) s += c.J[i] * u[i];
    return s;
}
// the quad's four values of z
__device__ __forceinline__ void quad_gather(double z, double* o) {
    const int base = (threadIdx.x & 31) & ~3;
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = __shfl_sync(0xffffffffu, z, base | i);
}
// prox_sphere (prox_operators.py:14) of the tangential values z[1..3] as one factor kind: 0 takes none of z, 1 takes
// z, 2 takes z * scale.
__device__ __forceinline__ int prox_factor(const double* z, double mu, double xn, double& scale) {
    const double radius = mu * xn;
    const double sqr = z[1] * z[1] + z[2] * z[2] + z[3] * z[3];
    const int kind = xn <= 0.0 ? 0 : (sqr <= radius * radius ? 1 : 2);
    scale = ratio_sqrt(kind == 2 ? radius : 1.0, kind == 2 ? sqr : 1.0);   // zeros would leave its range
    return kind;
}
__device__ __forceinline__ double prox_apply(int kind, double scale, double z) {
    const double t = z * scale;
    return kind == 0 ? 0.0 : (kind == 1 ? z : t);
}

// One projected Gauss-Seidel sweep (contacts.py:66-107) over the scene's levels, a quad per contact: lane q
// computes z_q from the current w, the four z meet by shuffles, every lane applies the prox (normal impulse
// clamped at zero, friction projected on the ball of radius mu x_n, or zeroed for post-stabilisation) and adds
// three of the twelve components of WJT[:, block] delta to w -- 2q, 2q + 1 and 8 + q, six per body -- with the
// reference's term order.  Reads the impulses x, writes the swept ones to y (which may be x).  Returns this
// thread's largest |y - x|.
//
// Bound by one contact's chain (12 dependent additions of 8 cycles, two shuffles, the prox's root and quotient, 5
// more additions: ~450 cycles) and by the ~290 instructions of a step, which one warp issues every ~4 cycles: what
// does not depend on w is kept off the chain.  A level of the 32-box tower takes 1210 cycles and one of 150-250
// boxes and spheres ~1500; with one thread per contact, its 96 matrix elements loaded after the level's barrier,
// they took 2700 and 6300.  The sweep is one sequence of steps (a level, or as many of its contacts as there are
// quads; steps[j] = first position, contacts, whether a level ends); each value of the next step's contact is
// loaded into the register of the current one's as soon as that is used up, its meta a step before that, so one
// copy of the loop body holds one contact and no register is moved.
template <class G, bool kShared>
__device__ __noinline__ double gs_sweep_quads(const G g, const Solve64 v, int n_steps, const double* b, const double* r,
                                              const double* x, double* y, bool normal_only) {
    const W64<kShared> w(v.w);
    const int q = g.rank() & 3, slot = g.rank() >> 2;
    const double* J = v.J + 2 * q;
    const double* WJT = v.WJT + 2 * q;
    b += q; r += q; y += q;
    const double* xs = x + q;
    double m = 0.0;
    auto meta = [&](int2 st) {
        int4 me = v.meta[min(st.x + slot, v.K - 1)];
        if (slot >= (st.y & 0xffff)) me.w = kMetaIdle;
        return me;
    };
    Contact64 c;
    double W[12];   // columns 2q, 2q + 1, 8 + q, four rows each
    auto load_w = [&](int k) {
        const double2* p = reinterpret_cast<const double2*>(WJT + 48 * (size_t)k);
#pragma unroll
        for (int i = 0; i < 6; ++i) { const double2 t = p[4 * i]; W[2 * i] = t.x; W[2 * i + 1] = t.y; }
    };
    auto load_j = [&](int k) {
        const double2* p = reinterpret_cast<const double2*>(J + 48 * (size_t)k);
#pragma unroll
        for (int i = 0; i < 6; ++i) { const double2 t = p[4 * i]; c.J[2 * i] = t.x; c.J[2 * i + 1] = t.y; }
    };
    auto load_x = [&](int k) {
        const double2* p = reinterpret_cast<const double2*>(x + 4 * (size_t)k);
        const double2 t = p[0], u = p[1];
        c.x[0] = t.x; c.x[1] = t.y; c.x[2] = u.x; c.x[3] = u.y;
    };
    int2 st0 = v.steps[0], st1 = v.steps[min(1, n_steps - 1)];
    c.me = meta(st0);
    load_j(c.me.x);
    load_x(c.me.x);
    load_w(c.me.x);
    c.xq = xs[4 * (size_t)c.me.x]; c.b = b[4 * (size_t)c.me.x]; c.r = r[4 * (size_t)c.me.x]; c.mu = v.mu[c.me.x];
    int4 next = meta(st1);
#pragma unroll 1
    for (int j = 0; j < n_steps; ++j) {
        const int2 st2 = v.steps[min(j + 2, n_steps - 1)];
        const double jw = contact64_jw(c, w);
        load_j(next.x);
        const double xq = c.xq, zq = xq - c.r * (jw + c.b);
        c.xq = xs[4 * (size_t)next.x]; c.b = b[4 * (size_t)next.x]; c.r = r[4 * (size_t)next.x];
        double z[4];
        quad_gather(zq, z);
        const double xn = z[0] > 0.0 ? z[0] : 0.0;
        double scale = 1.0;
        const int kind = normal_only ? 0 : prox_factor(z, c.mu, xn, scale);
        c.mu = v.mu[next.x];
        const double d0 = xn - c.x[0], d1 = prox_apply(kind, scale, z[1]) - c.x[1];
        const double d2 = prox_apply(kind, scale, z[2]) - c.x[2], d3v = prox_apply(kind, scale, z[3]) - c.x[3];
        load_x(next.x);
        const double yq = q == 0 ? xn : prox_apply(kind, scale, zq);
        double ta = 0.0, tb = 0.0, tc = 0.0;
        ta += W[0] * d0; tb += W[4] * d0; tc += W[8] * d0;
        ta += W[1] * d1; tb += W[5] * d1; tc += W[9] * d1;
        ta += W[2] * d2; tb += W[6] * d2; tc += W[10] * d2;
        ta += W[3] * d3v; tb += W[7] * d3v; tc += W[11] * d3v;
        load_w(next.x);
        const int ia = q < 3 ? c.me.y + 2 * q : c.me.z, ic = c.me.z + 2 + q;
        const double2 wa = w.pair(ia);
        const double wc = w.one(ic);
        if (c.me.w & (q < 3 ? 1 : 2)) w.set(ia, make_double2(wa.x + ta, wa.y + tb));
        if (c.me.w & 2) w.set(ic, wc + tc);
        if (!(c.me.w & kMetaIdle)) {
            y[4 * (size_t)c.me.x] = yq;
            m = nanmax(m, fabs(yq - xq));
        }
        if (st0.y & kStepEnds) g.sync();   // the last step of its level
        st0 = st1; st1 = st2;
        c.me = next;
        next = meta(st2);
    }
    return m;
}

// The same sweep by two groups of `warps` warps that take the steps by turns: while one computes a step, the other loads all
// that its next step's contact does not have from w, so only the chain itself lies between the barriers: the accumulators'
// loads, the row products, the prox, the update and its stores.  A group that has stored its step's w arrives at that
// step's barrier and goes on to its loads; the other waits there.  (32-box tower 883 -> 631 us a solve of 100 sweeps,
// 64-box lattice 1150 -> 719, 64 piles 8616 -> 5297; the 4096-body lattice, of which eight warps took a step at once,
// 2306 -> 2053 with two groups of four.)
template <bool kShared>
__device__ __noinline__ double gs_sweep_turns(const Solve64 v, int n_steps, const double* b, const double* r,
                                              const double* x, double* y, bool normal_only) {
    const W64<kShared> w(v.w);
    const int half = 32 * v.warps, group = (int)threadIdx.x >= half, rank = threadIdx.x - group * half;
    const int q = rank & 3, slot = rank >> 2;
    const double* J = v.J + 2 * q;
    const double* WJT = v.WJT + 2 * q;
    b += q; r += q; y += q;
    const double* xs = x + q;
    double m = 0.0;
    auto meta = [&](int j) {
        const int2 st = v.steps[min(j, n_steps - 1)];
        int4 me = v.meta[min(st.x + slot, v.K - 1)];
        if (slot >= st.y) me.w = kMetaIdle;
        return me;
    };
    int4 next = meta(group);
#pragma unroll 1
    for (int j = group; j < n_steps; j += 2) {
        const int4 me = next;
        const size_t k = (size_t)me.x;
        Contact64 c;
        c.me = me;
        double W[12];   // columns 2q, 2q + 1, 8 + q, four rows each
        const double2* pj = reinterpret_cast<const double2*>(J + 48 * k);
        const double2* pw = reinterpret_cast<const double2*>(WJT + 48 * k);
        const double2* px = reinterpret_cast<const double2*>(x + 4 * k);
#pragma unroll
        for (int i = 0; i < 6; ++i) { const double2 t = pj[4 * i]; c.J[2 * i] = t.x; c.J[2 * i + 1] = t.y; }
#pragma unroll
        for (int i = 0; i < 6; ++i) { const double2 t = pw[4 * i]; W[2 * i] = t.x; W[2 * i + 1] = t.y; }
        const double2 x01 = px[0], x23 = px[1];
        const double xq = xs[4 * k], bq = b[4 * k], rq = r[4 * k], mu = v.mu[k];
        next = meta(j + 2);
        const int ia = q < 3 ? me.y + 2 * q : me.z, ic = me.z + 2 + q;
        const bool put_a = (me.w & (q < 3 ? 1 : 2)) != 0, put_c = (me.w & 2) != 0;
        if (j > 0) turn_wait(group, 2 * half);
        const double zq = xq - rq * (contact64_jw(c, w) + bq);
        double z[4];
        quad_gather(zq, z);
        const double2 wa = w.pair(ia);
        const double wc = w.one(ic);
        const double xn = z[0] > 0.0 ? z[0] : 0.0;
        double scale = 1.0;
        const int kind = normal_only ? 0 : prox_factor(z, mu, xn, scale);
        const double d0 = xn - x01.x, d1 = prox_apply(kind, scale, z[1]) - x01.y;
        const double d2 = prox_apply(kind, scale, z[2]) - x23.x, d3v = prox_apply(kind, scale, z[3]) - x23.y;
        double ta = 0.0, tb = 0.0, tc = 0.0;
        ta += W[0] * d0; tb += W[4] * d0; tc += W[8] * d0;
        ta += W[1] * d1; tb += W[5] * d1; tc += W[9] * d1;
        ta += W[2] * d2; tb += W[6] * d2; tc += W[10] * d2;
        ta += W[3] * d3v; tb += W[7] * d3v; tc += W[11] * d3v;
        if (put_a) w.set(ia, make_double2(wa.x + ta, wa.y + tb));
        if (put_c) w.set(ic, wc + tc);
        if (j + 1 < n_steps) turn_done(group, 2 * half);
        const double yq = q == 0 ? xn : prox_apply(kind, scale, zq);
        if (!(me.w & kMetaIdle)) {
            y[4 * k] = yq;
            m = nanmax(m, fabs(yq - xq));
        }
    }
    return m;
}

// A block sweeps a scene with the number of its warps that scene_setup64 chose.  One warp has warp barriers between the
// levels, several a barrier of their own, and the block meets at the end of the sweep.
template <class G>
__device__ __forceinline__ double gs_sweep_levels(const G& g, const Solve64& v, const double* b, const double* r,
                                                  const double* x, double* y, bool normal_only) {
    if constexpr (std::is_same_v<G, BlockGroup>) {
        double m = 0.0;
        if (v.turns) {
            if ((int)threadIdx.x < 64 * v.warps)
                m = v.w_shared ? gs_sweep_turns<true>(v, v.n_steps, b, r, x, y, normal_only)
                               : gs_sweep_turns<false>(v, v.n_steps, b, r, x, y, normal_only);
        } else if (v.warps == 1) {
            if (threadIdx.x < 32) m = gs_sweep_levels(WarpGroup{}, v, b, r, x, y, normal_only);
        } else if ((int)threadIdx.x < 32 * v.warps) {
            const SubGroup sub = {32 * v.warps};
            m = v.w_shared ? gs_sweep_quads<SubGroup, true>(sub, v, v.n_steps, b, r, x, y, normal_only)
                           : gs_sweep_quads<SubGroup, false>(sub, v, v.n_steps, b, r, x, y, normal_only);
        }
        g.sync();
        return m;
    } else {
        return v.w_shared ? gs_sweep_quads<G, true>(g, v, v.n_steps, b, r, x, y, normal_only)
                          : gs_sweep_quads<G, false>(g, v, v.n_steps, b, r, x, y, normal_only);
    }
}

// Wavefront levels of the serial Gauss-Seidel order: level(k) = 1 + max level of the earlier contacts on
// k's non-fixed bodies.  Contacts of one level share no non-fixed body and every body sees its contacts in
// ascending order, so sweeping level by level (each level in parallel, any order inside a level) reproduces
// the serial sweep exactly.  The levels are the longest-path depths along the per-body predecessor chains,
// found by parallel relaxation; contacts are then bucketed by level.  Returns the number of levels.
template <class G>
__device__ int bucket_classes(const StepArgs& a, const G& g, const SceneRange& R, int s);

template <class G>
__device__ int scene_levels(const StepArgs& a, const G& g, const SceneRange& R, int s) {
    for (int k = R.c0 + g.rank(); k < R.c1; k += g.size()) a.ws.lev_of[k] = 1;
    g.sync();
    for (;;) {
        bool changed = false;
        for (int k = R.c0 + g.rank(); k < R.c1; k += g.size()) {
            const int p0 = a.ws.cpred[2 * k], p1 = a.ws.cpred[2 * k + 1];
            const int l0 = p0 >= 0 ? *(volatile int*)(a.ws.lev_of + p0) : 0;
            const int l1 = p1 >= 0 ? *(volatile int*)(a.ws.lev_of + p1) : 0;
            const int l = 1 + max(l0, l1);
            if (l != a.ws.lev_of[k]) { a.ws.lev_of[k] = l; changed = true; }
        }
        if (!g.any(changed)) break;
    }
    return bucket_classes(a, g, R, s);
}

// The same levels with the relaxation and the bucketing in shared memory: scratch (s32_level_scratch bytes)
// holds the two predecessors of each contact (scene-local int16), its level (int16) and one counter per level;
// the levels then go to lev_of and the buckets to lev_ptr / lev_order.  Same fixed point, same order within a
// level up to the order of atomics, which no result depends on.
__host__ __device__ inline size_t s32_level_scratch(int K) { return 6 * (size_t)K + 4 * (size_t)(K + 2) + 16; }
template <class G>
__device__ int scene_levels_smem(const StepArgs& a, const G& g, const SceneRange& R, int s, int16_t* scratch) {
    const int K = R.c1 - R.c0;
    int16_t* pred = scratch;
    volatile int16_t* lev = scratch + 2 * K;
    int* cnt = reinterpret_cast<int*>(reinterpret_cast<char*>(scratch) + ((6 * (size_t)K + 15) & ~size_t(15)));
    for (int k = g.rank(); k < K; k += g.size()) {
        const int p0 = a.ws.cpred[2 * (R.c0 + k)], p1 = a.ws.cpred[2 * (R.c0 + k) + 1];
        pred[2 * k] = (int16_t)(p0 >= 0 ? p0 - R.c0 : -1);
        pred[2 * k + 1] = (int16_t)(p1 >= 0 ? p1 - R.c0 : -1);
    }
    g.sync();
    // predecessors come earlier: one warp goes through the contacts 32 at a time, those of the earlier runs final, and
    // relaxes within the run until nothing changes (relaxing all of them in rounds of the whole team took 60 to 100
    // thousand cycles for 600 contacts on 50 to 90 levels)
    if (g.rank() < 32)
        for (int k0 = 0; k0 < K; k0 += 32) {
            const int k = k0 + g.rank();
            const bool mine = k < K;
            const int p0 = mine ? pred[2 * k] : -1, p1 = mine ? pred[2 * k + 1] : -1;
            int l = 1;
            if (mine) lev[k] = 1;
            __syncwarp();
            for (;;) {
                const int l0 = p0 >= 0 ? lev[p0] : 0, l1 = p1 >= 0 ? lev[p1] : 0;
                const int next = 1 + max(l0, l1);
                const bool changed = mine && next != l;
                if (!__any_sync(0xffffffffu, changed)) break;   // (every lane has read before any writes)
                if (changed) { l = next; lev[k] = (int16_t)l; }
                __syncwarp();
            }
        }
    g.sync();
    int L = 0;
    for (int k = g.rank(); k < K; k += g.size()) {
        const int l = lev[k];
        a.ws.lev_of[R.c0 + k] = l;
        L = max(L, l);
    }
    L = g.imax(L);
    for (int l = g.rank(); l <= L; l += g.size()) cnt[l] = 0;
    g.sync();
    for (int k = g.rank(); k < K; k += g.size()) atomicAdd(cnt + lev[k] - 1, 1);
    g.sync();
    int* ptr = a.ws.lev_ptr + R.c0 + s;   // ptr[l-1] .. ptr[l]: contacts of level l (1-based), ptr[L] = K
    if (g.rank() == 0) {
        int acc = 0;
        for (int l = 0; l < L; ++l) { const int c = cnt[l]; ptr[l] = acc; cnt[l] = acc; acc += c; }
        ptr[L] = acc;
    }
    g.sync();
    // the order within a level does not change any result (its contacts share no body that is written)
    for (int k = g.rank(); k < K; k += g.size()) a.ws.lev_order[R.c0 + atomicAdd(cnt + lev[k] - 1, 1)] = R.c0 + k;
    g.sync();
    return L;
}

// the levels with the accumulators' shared memory as scratch where it suffices (it is not in use yet)
template <class G>
__device__ __forceinline__ int scene_levels_any(const StepArgs& a, const G& g, const SceneRange& R, int s, double* w_smem,
                                                int smem_bodies) {
    const int K = R.c1 - R.c0;
    if (w_smem != nullptr && K <= 32767 && s32_level_scratch(K) <= 6 * sizeof(double) * (size_t)smem_bodies)
        return scene_levels_smem(a, g, R, s, reinterpret_cast<int16_t*>(w_smem));
    return scene_levels(a, g, R, s);
}

// Groups the scene's contacts by their class lev_of[k] (1-based level or colour): lev_ptr[c-1] .. lev_ptr[c]
// index lev_order, which lists the contacts of class c.  Returns the number of classes.
template <class G>
__device__ int bucket_classes(const StepArgs& a, const G& g, const SceneRange& R, int s) {
    int L = 0;
    for (int k = R.c0 + g.rank(); k < R.c1; k += g.size()) L = max(L, a.ws.lev_of[k]);
    L = g.imax(L);
    int* ptr = a.ws.lev_ptr + R.c0 + s;   // ptr[l-1] .. ptr[l]: contacts of level l (1-based), ptr[L] = K
    int* cur = a.ws.lev_cur + R.c0 + s;
    for (int l = g.rank(); l <= L; l += g.size()) cur[l] = 0;
    g.sync();
    for (int k = R.c0 + g.rank(); k < R.c1; k += g.size()) atomicAdd(cur + a.ws.lev_of[k] - 1, 1);
    g.sync();
    if (g.rank() == 0) {
        int acc = 0;
        for (int l = 0; l < L; ++l) { const int c = cur[l]; ptr[l] = acc; cur[l] = acc; acc += c; }
        ptr[L] = acc;
    }
    g.sync();
    for (int k = R.c0 + g.rank(); k < R.c1; k += g.size())
        a.ws.lev_order[R.c0 + atomicAdd(cur + a.ws.lev_of[k] - 1, 1)] = k;
    g.sync();
    return L;
}

// Graph colouring of the scene's contacts for RB_ORDER_COLOURED: two contacts are neighbours when they share a
// non-fixed body.  Jones-Plassmann rounds with hashed priorities (higher hash first, then lower scene-local
// index): in each round every uncoloured contact whose uncoloured neighbours all come later in priority takes
// the smallest colour none of its coloured neighbours has.  Deterministic, so every launch shape gives the
// same colours; the oracle's rbo_colour_contacts is the same procedure.
__device__ __forceinline__ uint32_t jp_hash(uint32_t k) {
    k ^= k >> 16; k *= 0x7feb352dU; k ^= k >> 15; k *= 0x846ca68bU; k ^= k >> 16;
    return k;
}
__device__ __forceinline__ bool jp_before(int p, int q) {
    const uint32_t hp = jp_hash((uint32_t)p), hq = jp_hash((uint32_t)q);
    return hp > hq || (hp == hq && p < q);
}
// colour (0-based) contact k takes this round, or -1 while a neighbour of higher priority is uncoloured
__device__ int colour_pick(const StepArgs& a, const SceneRange& R, int k) {
    const int* col = a.ws.lev_of;   // colour + 1; 0 = uncoloured
    uint64_t used = 0;
    for (int side = 0; side < 2; ++side) {
        const int b = a.ws.lohi[2 * k + side];
        if (a.bd.fixed[b]) continue;
        for (int e = a.ws.bc_ptr[b]; e < a.ws.bc_ptr[b + 1]; ++e) {
            const int m = a.ws.bc_list[e] >> 1;
            if (m == k) continue;
            const int c = col[m];
            if (c == 0) {
                if (jp_before(m - R.c0, k - R.c0)) return -1;
            } else if (c <= 64) {
                used |= 1ull << (c - 1);
            }
        }
    }
    for (int c = 0;; ++c) {
        bool taken = false;
        if (c < 64) {
            taken = (used >> c) & 1ull;
        } else {
            for (int side = 0; side < 2 && !taken; ++side) {
                const int b = a.ws.lohi[2 * k + side];
                if (a.bd.fixed[b]) continue;
                for (int e = a.ws.bc_ptr[b]; e < a.ws.bc_ptr[b + 1] && !taken; ++e) {
                    const int m = a.ws.bc_list[e] >> 1;
                    taken = m != k && col[m] == c + 1;
                }
            }
        }
        if (!taken) return c;
    }
}
template <class G>
__device__ int scene_colours(const StepArgs& a, const G& g, const SceneRange& R, int s) {
    int* col = a.ws.lev_of;
    int* pick = a.ws.lev_cur + R.c0 + s;   // this round's choices (the class counters are built afterwards)
    for (int k = R.c0 + g.rank(); k < R.c1; k += g.size()) col[k] = 0;
    g.sync();
    const int K = R.c1 - R.c0;
    for (int round = 0; round <= K; ++round) {   // every round colours at least the top-priority contact
        bool left = false;
        for (int k = R.c0 + g.rank(); k < R.c1; k += g.size()) {
            int c = -1;
            if (col[k] == 0) { c = colour_pick(a, R, k); left = true; }
            pick[k - R.c0] = c;
        }
        g.sync();
        if (!g.any(left)) break;
        for (int k = R.c0 + g.rank(); k < R.c1; k += g.size())
            if (pick[k - R.c0] >= 0) col[k] = pick[k - R.c0] + 1;
        g.sync();
    }
    return bucket_classes(a, g, R, s);
}

// complementarity residual ||x - prox(x - D^-1 (A x + b))||_inf / max(1, ||x||_inf), D = diag(A): the
// tolerance the solver modes are compared at.  Every scheme scales the prox argument by a positive multiple of
// D^-1, so they all share this map's zeros as fixed points.  A x = J W J^T x through w = WJT x (the
// accumulators are rebuilt from x at the start of every sweep, so they are free to hold this product here).
template <class G>
__device__ double scene_residual(const StepArgs& a, const G& g, const Solve64& v, const double* x) {
    scene_wjt(g, v, x);
    const int q = g.rank() & 3, slot = g.rank() >> 2, nslot = g.size() >> 2;
    double m = 0.0, xm = 0.0;
    Contact64 c;
    contact64_load(v, contact64_meta(v, slot, v.K), q, a.ws.b, a.ws.diag, x, c);
    for (int i = 0; i < v.K; i += nslot) {   // a quad per contact, the next one's values loaded meanwhile
        const double jw = contact64_jw(c, W64<false>(v.w));
        const double xq = c.xq;
        const double bq = c.b, dq = c.r, mu = c.mu;
        const bool mine = !(c.me.w & kMetaIdle);
        contact64_load(v, contact64_meta(v, i + nslot + slot, v.K), q, a.ws.b, a.ws.diag, x, c);
        double z[4];
        const double zq = xq - (1.0 / dq) * (jw + bq);
        quad_gather(zq, z);
        const double pn = z[0] > 0.0 ? z[0] : 0.0;
        double scale;
        const int kind = prox_factor(z, mu, pn, scale);
        if (mine) {
            m = nanmax(m, fabs(xq - (q == 0 ? pn : prox_apply(kind, scale, zq))));
            xm = fmax(xm, fabs(xq));
        }
    }
    g.max2(m, xm);
    return m / (xm > 1.0 ? xm : 1.0);
}

// ---------------------------------------------------------------------------------------------------------
// hinge joints (constraints/hinges.py): 5 rows per hinge between a parent and a child body
// ---------------------------------------------------------------------------------------------------------
// per-body hinge lists of each scene (thread per scene): entries (hinge << 1 | side), hinges ascending; every
// hinge gives both of its bodies an entry, so scene s's entries fill [2 h0, 2 h1) exactly
__global__ void k_hinge_lists(const StepArgs a) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= a.bd.n_scenes || a.ws.counters[kAbort]) return;
    const int b0 = a.bd.scene_start[s], b1 = a.bd.scene_start[s + 1];
    const int h0 = a.bd.scene_hinge_start[s], h1 = a.bd.scene_hinge_start[s + 1];
    int32_t* cnt = a.ws.hlast;
    for (int b = b0; b < b1; ++b) cnt[b] = 0;
    for (int k = h0; k < h1; ++k) { cnt[a.bd.hinge_bodies[2 * k]]++; cnt[a.bd.hinge_bodies[2 * k + 1]]++; }
    int pos = 2 * h0;
    for (int b = b0; b < b1; ++b) { a.ws.hbody_ptr[b] = pos; pos += cnt[b]; cnt[b] = 0; }
    if (s == a.bd.n_scenes - 1) a.ws.hbody_ptr[a.bd.n_bodies] = pos;
    for (int k = h0; k < h1; ++k)
        for (int side = 0; side < 2; ++side) {
            const int P = a.bd.hinge_bodies[2 * k], C = a.bd.hinge_bodies[2 * k + 1];
            const int b = side ? max(P, C) : min(P, C);
            a.ws.hbody_list[a.ws.hbody_ptr[b] + cnt[b]++] = (k << 1) | side;
        }
}

// hinges.py:28-50 Hinges.initialize with _compute_jacobian_matrix (:95-180) and _compute_error_vector
// (:188-218): J, W J^T (bsr_matmat order), b = (J u + J dt du_ext) + g, diag = sum(J .* WJT^T) (zeros -> 1),
// r = 1/diag, x = sol = 0.  Thread per hinge.
__global__ void k_hinges(const StepArgs a) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.bd.n_hinges || a.ws.counters[kAbort]) return;
    const int A = a.bd.hinge_bodies[2 * k], B = a.bd.hinge_bodies[2 * k + 1];
    const double* f = a.bd.hinge_frames + 12 * (size_t)k;
    const double* qA = a.bd.x + 7 * A + 3;
    const double* qB = a.bd.x + 7 * B + 3;
    const d3 ap = quat_rotate(qA, ld3(f)), ac = quat_rotate(qB, ld3(f + 3)), np_ = quat_rotate(qA, ld3(f + 6));
    d3 t, bb, nn;
    make_orthonormal_vectors(np_, t, bb, nn);
    // JA_v[0:3] = I, JA_w[0:3] = -star(arm_p), JA_w[3] = t, JA_w[4] = b; JB_v[0:3] = -I, JB_w[0:3] = star(arm_c),
    // JB_w[3] = -t, JB_w[4] = -b; star(v) = [[0, -v2, v1], [v2, 0, -v0], [-v1, v0, 0]]
    const double sp[3][3] = {{0.0, -ap.z, ap.y}, {ap.z, 0.0, -ap.x}, {-ap.y, ap.x, 0.0}};
    const double sc[3][3] = {{0.0, -ac.z, ac.y}, {ac.z, 0.0, -ac.x}, {-ac.y, ac.x, 0.0}};
    double JA[5][6], JB[5][6];
    for (int i = 0; i < 5; ++i)
        for (int j = 0; j < 6; ++j) { JA[i][j] = 0.0; JB[i][j] = 0.0; }
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            JA[i][j] = i == j ? 1.0 : 0.0;
            JA[i][3 + j] = -sp[i][j];
            JB[i][j] = -(i == j ? 1.0 : 0.0);
            JB[i][3 + j] = sc[i][j];
        }
    const double tv[3] = {t.x, t.y, t.z}, bv[3] = {bb.x, bb.y, bb.z};
    for (int j = 0; j < 3; ++j) {
        JA[3][3 + j] = tv[j]; JA[4][3 + j] = bv[j];
        JB[3][3 + j] = -tv[j]; JB[4][3 + j] = -bv[j];
    }
    const int lo = min(A, B), hi = max(A, B);
    a.ws.hlohi[2 * k] = lo;
    a.ws.hlohi[2 * k + 1] = hi;
    double* J = a.ws.hJ + 60 * (size_t)k;
    double* W = a.ws.hWJT + 60 * (size_t)k;
    for (int row = 0; row < 5; ++row)
        for (int j = 0; j < 6; ++j) {
            J[12 * row + (A == lo ? 0 : 6) + j] = JA[row][j];
            J[12 * row + (B == lo ? 0 : 6) + j] = JB[row][j];
        }
    bool hasw[2];
    for (int side = 0; side < 2; ++side) {
        const int bd = side ? hi : lo;
        hasw[side] = !a.bd.fixed[bd];
        const double m = hasw[side] ? 1.0 / a.bd.mass[bd] : 0.0;
        const double* Wi = a.ws.Winv + 9 * (size_t)bd;
        for (int row = 0; row < 5; ++row) {
            const double* Jr = J + 12 * row + 6 * side;
            double* Wr = W + 12 * row + 6 * side;
            for (int i = 0; i < 3; ++i) {
                double s = 0.0;
                s += (i == 0 ? m : 0.0) * Jr[0];
                s += (i == 1 ? m : 0.0) * Jr[1];
                s += (i == 2 ? m : 0.0) * Jr[2];
                double u = 0.0;
                u += Wi[3 * i + 0] * Jr[3];
                u += Wi[3 * i + 1] * Jr[4];
                u += Wi[3 * i + 2] * Jr[5];
                Wr[i] = hasw[side] ? s : 0.0;
                Wr[3 + i] = hasw[side] ? u : 0.0;
            }
        }
    }
    double g[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (a.pr.use_pre_stabilization) {
        const d3 rp = add(ap, ld3(a.bd.x + 7 * A)), rc = add(ac, ld3(a.bd.x + 7 * B));
        const d3 ncv = quat_rotate(qB, ld3(f + 9));
        const d3 u = cross_np(nn, ncv);
        const double rate = a.pr.gap_reduction / a.pr.dt;
        g[0] = (rc.x - rp.x) * rate;
        g[1] = (rc.y - rp.y) * rate;
        g[2] = (rc.z - rp.z) * rate;
        g[3] = dot3_np(t, u) * rate;
        g[4] = dot3_np(bb, u) * rate;
    }
    const double* ulo = a.bd.u + 6 * lo;
    const double* uhi = a.bd.u + 6 * hi;
    const double* dlo = a.ws.du + 6 * lo;
    const double* dhi = a.ws.du + 6 * hi;
    for (int row = 0; row < 5; ++row) {
        const double* Jr = J + 12 * row;
        const double* Wr = W + 12 * row;
        a.ws.hb[5 * (size_t)k + row] = (jrow_dot(Jr, ulo, uhi) + jrow_dot(Jr, dlo, dhi)) + g[row];
        double prods[12];
        int m = 0;
        for (int c = 0; c < 12; ++c) {
            if (!hasw[c / 6]) continue;
            const double prod = Jr[c] * Wr[c];
            if (prod != 0.0) prods[m++] = prod;
        }
        const double d = np_reduce_sum(prods, m);
        const double diag = d == 0.0 ? 1.0 : d;
        a.ws.hdiag[5 * (size_t)k + row] = diag;
        a.ws.hr[5 * (size_t)k + row] = 1.0 / diag;
        a.ws.hx[5 * (size_t)k + row] = 0.0;
        a.ws.hsol[5 * (size_t)k + row] = 0.0;
    }
}

// w = W J^T x of the hinge problem for every body of the scene (hinges ascending, 5 rows each)
template <class G>
__device__ void hinge_wjt(const StepArgs& a, const G& g, const SceneRange& R) {
    for (int b = R.b0 + g.rank(); b < R.b1; b += g.size()) {
        double s6[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (!a.bd.fixed[b])
            for (int e = a.ws.hbody_ptr[b]; e < a.ws.hbody_ptr[b + 1]; ++e) {
                const int code = a.ws.hbody_list[e];
                const int k = code >> 1, side = code & 1;
                const double* Wk = a.ws.hWJT + 60 * (size_t)k + 6 * side;
                for (int d = 0; d < 6; ++d) {
                    double t = s6[d];
                    for (int row = 0; row < 5; ++row) t += Wk[12 * row + d] * a.ws.hx[5 * (size_t)k + row];
                    s6[d] = t;
                }
            }
        for (int d = 0; d < 6; ++d) a.ws.hw[6 * (size_t)b + d] = s6[d];
    }
    g.sync();
}

// hinges.py:62-90: x_b -= r_b (J w + b)_b from the w before this hinge, then w += WJT[:, b] dx
__device__ __forceinline__ void hinge_update(const StepArgs& a, int k) {
    const int lo = a.ws.hlohi[2 * k], hi = a.ws.hlohi[2 * k + 1];
    const double* J = a.ws.hJ + 60 * (size_t)k;
    double* wlo = a.ws.hw + 6 * (size_t)lo;
    double* whi = a.ws.hw + 6 * (size_t)hi;
    double jw[5], delta[5];
    for (int row = 0; row < 5; ++row) jw[row] = jrow_dot(J + 12 * row, wlo, whi);
    for (int row = 0; row < 5; ++row) {
        const size_t i = 5 * (size_t)k + row;
        const double xo = a.ws.hx[i];
        const double xn = xo - a.ws.hr[i] * (jw[row] + a.ws.hb[i]);
        a.ws.hx[i] = xn;
        delta[row] = xn - xo;
    }
    for (int side = 0; side < 2; ++side) {
        const int bd = side ? hi : lo;
        if (a.bd.fixed[bd]) continue;
        double* wb = side ? whi : wlo;
        const double* Ws = a.ws.hWJT + 60 * (size_t)k + 6 * side;
        for (int d = 0; d < 6; ++d) {
            double t = 0.0;
            for (int row = 0; row < 5; ++row) t += Ws[12 * row + d] * delta[row];
            wb[d] = wb[d] + t;
        }
    }
}

// levels of the scene's hinges in their serial order (a hinge follows the earlier hinges on its non-fixed
// bodies), by one thread: hlev_order[h0 ..] lists the hinges level by level, ascending inside a level, and
// hlev_ptr[h0 + s + l - 1] .. hlev_ptr[h0 + s + l] index the hinges of level l.  Returns the number of levels.
template <class G>
__device__ int hinge_levels(const StepArgs& a, const G& g, const SceneRange& R, int s, int h0, int h1) {
    int L = 0;
    if (g.rank() == 0) {
        int32_t* last = a.ws.hlast;
        for (int b = R.b0; b < R.b1; ++b) last[b] = 0;
        int32_t* lev = a.ws.hlev;
        for (int k = h0; k < h1; ++k) {
            const int lo = a.ws.hlohi[2 * k], hi = a.ws.hlohi[2 * k + 1];
            const int l0 = a.bd.fixed[lo] ? 0 : last[lo], l1 = a.bd.fixed[hi] ? 0 : last[hi];
            const int l = 1 + max(l0, l1);
            if (!a.bd.fixed[lo]) last[lo] = l;
            if (!a.bd.fixed[hi]) last[hi] = l;
            lev[k] = l;
            L = max(L, l);
        }
        int32_t* ptr = a.ws.hlev_ptr + h0 + s;
        for (int l = 0; l <= L; ++l) ptr[l] = 0;
        for (int k = h0; k < h1; ++k) ptr[lev[k]]++;
        for (int l = 1; l <= L; ++l) ptr[l] += ptr[l - 1];          // ptr[l] = end of level l
        for (int l = L; l >= 1; --l) ptr[l] = ptr[l - 1];          // ptr[l] = start of level l, used as
        ptr[0] = 0;                                                  // the level's cursor: after the fill
        for (int k = h0; k < h1; ++k) a.ws.hlev_order[h0 + ptr[lev[k]]++] = k;   // it is the level's end
    }
    g.sync();
    return g.imax(L);
}

// The reference stepper's Gauss-Seidel loop over [contacts (when any), hinges] (gauss_seidel_solver.py:14-101):
// every iteration sweeps each problem in turn (each with its own accumulators w, built from its own x at the
// start of its sweep), accepts or rolls back its iterate against that problem's own last merit and adapts its
// r-factors; the convergence tests use the largest merit of the iteration.  FP64, serial order, merit rule.
template <class G>
__device__ void solve_scene_hinges(const StepArgs& a, const G& g, int s, double* w_smem, int smem_bodies) {
    const int max_it = a.pr.max_iterations;
    double* x = a.ws.x;
    double* sol = a.out.contact_sol;
    const double* b = a.ws.b;
    double* r = a.ws.r;
    const SceneRange R = scene_range(a, s);
    const int K = R.c1 - R.c0;
    const int h0 = a.bd.scene_hinge_start[s], h1 = a.bd.scene_hinge_start[s + 1];
    rb_scene_stats* st = a.out.stats + s;
    double* hist = (a.out.residuals && a.pr.profiling) ? a.out.residuals + (size_t)s * a.caps.max_iterations : nullptr;
    if (g.rank() == 0) {
        st->n_contacts = K; st->contact_start = R.c0; st->iterations = -1; st->exitcode = -1;
        st->merit = 0.0; st->residual = 0.0; st->post_iterations = -1; st->post_exitcode = -1;
        st->n_levels = 0; st->fp32_sweeps = 0;
    }
    if (hist) for (int i = g.rank(); i < max_it; i += g.size()) hist[i] = INFINITY;
    const int L = K > 0 ? scene_levels_any(a, g, R, s, w_smem, smem_bodies) : 0;
    Solve64 v = {};
    if (K > 0) v = scene_setup64(a, g, R, s, L, w_smem, smem_bodies);
    const int HL = hinge_levels(a, g, R, s, h0, h1);
    if (g.rank() == 0) st->n_levels = L;
    const int* hptr = a.ws.hlev_ptr + h0 + s;
    double last_c = INFINITY, last_h = INFINITY, global_last = INFINITY, shown = 0.0;
    int iterations = max_it, exitcode = 0;
    for (int it = 0; it < max_it; ++it) {
        double gm = 0.0;
        if (K > 0) {   // Contacts.sweep, then the accept / roll-back rule
            scene_wjt(g, v, x);
            // x = sol at the start of every sweep, so the sweep's largest change is the merit ||x - sol||_inf
            const double merit = g.max(gs_sweep_levels(g, v, b, r, x, x, false));
            const bool reject = merit > last_c;
            const bool inc = !reject && last_c - merit < a.pr.too_small_merit_change;
            for (int i = 4 * R.c0 + g.rank(); i < 4 * R.c1; i += g.size()) {
                if (reject) { r[i] = a.pr.nu_reduce * r[i]; x[i] = sol[i]; }
                else { sol[i] = x[i]; if (inc) r[i] = a.pr.nu_increase * r[i]; }
            }
            if (reject) gm = gm > last_c ? gm : last_c;
            else { last_c = merit; gm = gm > merit ? gm : merit; }
            g.sync();
        }
        {              // Hinges.sweep, then the same rule with the hinge problem's own merit and r-factors
            hinge_wjt(a, g, R);
            for (int l = 1; l <= HL; ++l) {
                for (int i = hptr[l - 1] + g.rank(); i < hptr[l]; i += g.size()) hinge_update(a, a.ws.hlev_order[h0 + i]);
                g.sync();
            }
            double m = 0.0;
            for (int i = 5 * h0 + g.rank(); i < 5 * h1; i += g.size()) m = nanmax(m, fabs(a.ws.hx[i] - a.ws.hsol[i]));
            const double merit = g.max(m);
            const bool reject = merit > last_h;
            const bool inc = !reject && last_h - merit < a.pr.too_small_merit_change;
            for (int i = 5 * h0 + g.rank(); i < 5 * h1; i += g.size()) {
                if (reject) { a.ws.hr[i] = a.pr.nu_reduce * a.ws.hr[i]; a.ws.hx[i] = a.ws.hsol[i]; }
                else { a.ws.hsol[i] = a.ws.hx[i]; if (inc) a.ws.hr[i] = a.pr.nu_increase * a.ws.hr[i]; }
            }
            if (reject) gm = gm > last_h ? gm : last_h;
            else { last_h = merit; gm = gm > merit ? gm : merit; }
            g.sync();
        }
        if (hist && g.rank() == 0) hist[it] = gm;
        shown = gm;
        bool stop = false;
        if (gm < a.pr.absolute_tolerance) { stop = true; exitcode = 1; }
        else if (fabs(gm - global_last) < a.pr.relative_tolerance * global_last) { stop = true; exitcode = 2; }
        global_last = gm;
        if (stop) { iterations = it; break; }
    }
    if (a.out.hinge_sol)
        for (int i = 5 * h0 + g.rank(); i < 5 * h1; i += g.size()) a.out.hinge_sol[i] = a.ws.hsol[i];
    if (g.rank() == 0) { st->iterations = iterations; st->exitcode = exitcode; st->merit = shown; }
    g.sync();
}

// device clock in microseconds (the global nanosecond timer)
__device__ __forceinline__ double device_us() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return 1e-3 * (double)t;
}

template <class G>
__device__ void solve_scene_body(const StepArgs& a, const G& g, int s, int post, double* w_smem, int smem_bodies);

// The proximal solve of one scene (gauss_seidel_solver.py:14 / solver_interface.py:123); with profiling on,
// its device time goes to the scene's statistics (added to the FP32 phase's time when one ran).
template <class G>
__device__ void solve_scene(const StepArgs& a, const G& g, int s, int post, double* w_smem, int smem_bodies) {
    if (!post && a.ws.fin32[s]) return;   // finished by the FP32 phase
    const bool timed = !post && a.pr.profiling;
    const double t0 = timed ? device_us() : 0.0;
    solve_scene_body(a, g, s, post, w_smem, smem_bodies);
    if (!post && g.rank() == 0) {
        rb_scene_stats* st = a.out.stats + s;
        const bool fp32_phase = a.pr.precision != RB_PRECISION_FP64 && a.ws.sweeps32[s] >= 0;
        if (!timed) { st->solve_start_us = 0.0; st->solve_us = 0.0; }
        else if (fp32_phase) st->solve_us += device_us() - t0;
        else { st->solve_start_us = t0; st->solve_us = device_us() - t0; }
    }
}

template <class G>
__device__ void solve_scene_body(const StepArgs& a, const G& g, int s, int post, double* w_smem, int smem_bodies) {
    if (!post && a.bd.n_hinges > 0 && a.bd.scene_hinge_start[s + 1] > a.bd.scene_hinge_start[s]) {
        solve_scene_hinges(a, g, s, w_smem, smem_bodies);
        return;
    }
    const int scheme = post ? RB_SCHEME_RIGID_GS : a.pr.scheme;
    const bool rigid = scheme == RB_SCHEME_RIGID_GS;
    const bool jacobi = scheme == RB_SCHEME_JACOBI || scheme == RB_SCHEME_JACOBI_HYBRID;
    const int max_it = a.pr.max_iterations;
    // the accepted impulses x and the sweep's new ones y: two arrays that change places when a sweep is
    // accepted (a rolled-back sweep leaves x as it is); the solution goes to sol at the end
    double* x = a.ws.x;
    double* sol = post ? a.ws.xold : a.out.contact_sol;
    double* y = a.ws.xold;
    const double* b = a.ws.b;
    double* r = a.ws.r;
    const SceneRange R = scene_range(a, s);
    const int K = R.c1 - R.c0;
    rb_scene_stats* st = a.out.stats + s;
    double* hist = (!post && a.out.residuals && a.pr.profiling) ? a.out.residuals + (size_t)s * a.caps.max_iterations
                                                                : nullptr;
    if (g.rank() == 0) {
        if (!post) {
            st->n_contacts = K; st->contact_start = R.c0; st->iterations = -1; st->exitcode = -1;
            st->merit = 0.0; st->residual = 0.0; st->post_iterations = -1; st->post_exitcode = -1;
            st->n_levels = 0; st->fp32_sweeps = 0;
        } else {
            st->post_iterations = -1; st->post_exitcode = -1;
        }
    }
    if (hist) for (int i = g.rank(); i < max_it; i += g.size()) hist[i] = INFINITY;
    if (K == 0) { g.sync(); return; }
    if (post) {   // steppers.py:32: no solve when no contact is deeper than min_gap
        bool any = false;
        for (int k = R.c0 + g.rank(); k < R.c1; k += g.size()) any |= (b[4 * k] != 0.0);
        if (!g.any(any)) return;
    }
    const bool coloured = !post && !jacobi &&
                          (scheme == RB_SCHEME_COLOURED_GS || a.pr.ordering == RB_ORDER_COLOURED);
    // FP32 modes: the scene's FP32 phase left its iterate in x and its level order in lev_order / lev_ptr
    const int sweeps32 = (!post && a.pr.precision != RB_PRECISION_FP64) ? a.ws.sweeps32[s] : -1;
    const int L = jacobi ? 0 : sweeps32 >= 0 ? a.ws.nlev[s]
                : (coloured ? scene_colours(a, g, R, s) : scene_levels_any(a, g, R, s, w_smem, smem_bodies));
    if (!post && g.rank() == 0) st->n_levels = L;
    const Solve64 v = scene_setup64(a, g, R, s, L, w_smem, smem_bodies);
    const bool by_residual = !post && a.pr.termination != RB_TERMINATE_MERIT;
    const bool fixed_r = !post && a.pr.termination == RB_TERMINATE_RESIDUAL_FIXED_R;
    const int interval = a.pr.residual_interval > 1 ? a.pr.residual_interval : 1;
    double last = INFINITY, global_last = INFINITY, shown = 0.0;
    int iterations = max_it, exitcode = 0;
    bool w_is_wjt_x = false;   // w already holds WJT x for the current x (left by the residual pass)
    // FP32 modes: test the FP32 iterate in FP64, then refine it in FP64 with the sweeps left
    int loop_max = max_it;
    if (sweeps32 >= 0) {
        const double res0 = scene_residual(a, g, v, x);
        w_is_wjt_x = true;
        shown = res0;
        if (g.rank() == 0) st->fp32_sweeps = sweeps32;
        if (res0 <= a.pr.residual_tolerance || a.pr.precision == RB_PRECISION_FP32 || sweeps32 >= max_it) {
            for (int i = 4 * R.c0 + g.rank(); i < 4 * R.c1; i += g.size()) sol[i] = x[i];
            g.sync();
            const bool ok = res0 <= a.pr.residual_tolerance;
            if (g.rank() == 0) {
                st->iterations = ok ? max(sweeps32 - 1, 0) : max_it;
                st->exitcode = ok ? 3 : 0;
                st->merit = res0;
                st->residual = res0;
            }
            g.sync();
            return;
        }
        loop_max = max_it - sweeps32;   // the sweeps the FP32 phase left over
    }
    for (int it = 0; it < loop_max; ++it) {
        if (!w_is_wjt_x) scene_wjt(g, v, x);   // every sweep starts from w = WJT x (contacts.py:72)
        double m = 0.0;
        if (jacobi) {               // proximal_contact/jacobi_solver.py:41-79, a quad per contact
            const bool hybrid = scheme == RB_SCHEME_JACOBI_HYBRID;
            const int q = g.rank() & 3, slot = g.rank() >> 2, nslot = g.size() >> 2;
            Contact64 c;
            contact64_load(v, contact64_meta(v, slot, K), q, b, r, x, c);
            for (int i = 0; i < K; i += nslot) {
                const double jw = contact64_jw(c, W64<false>(v.w));
                const double xq = c.xq, xn_old = c.x[0];
                const double bq = c.b, rq = c.r, mu = c.mu;
                const int4 me = c.me;
                contact64_load(v, contact64_meta(v, i + nslot + slot, K), q, b, r, x, c);
                double z[4];
                const double zq = xq - rq * (jw + bq);
                quad_gather(zq, z);
                const double xn = z[0] > 0.0 ? z[0] : 0.0;
                double scale;
                const int kind = prox_factor(z, mu, hybrid ? xn : xn_old, scale);
                if (!(me.w & kMetaIdle)) {
                    const double xnew = q == 0 ? xn : prox_apply(kind, scale, zq);
                    y[4 * (size_t)me.x + q] = xnew;
                    m = nanmax(m, fabs(xnew - xq));
                }
            }
            g.sync();
        } else {
            m = gs_sweep_levels(g, v, b, r, x, y, post != 0);
        }
        // merit = ||y - x||_inf (problem.py:53); the fixed-r rule never looks at it
        const double merit = fixed_r ? 0.0 : g.max(m);
        const bool check = by_residual && (!fixed_r || (it + 1) % interval == 0 || it + 1 == loop_max);
        const double res = check ? scene_residual(a, g, v, y) : 0.0;
        int decision = 0;   // 0 accept, 1 reject, 2 keep x, 3 take y
        bool stop = false, inc = false;
        if (rigid) {        // gauss_seidel_solver.py:439-482
            double gm;
            if (merit > last) { decision = 1; gm = last > 0.0 ? last : 0.0; }
            else {
                inc = last - merit < a.pr.too_small_merit_change;
                last = merit;
                gm = merit > 0.0 ? merit : 0.0;
            }
            if (gm < a.pr.absolute_tolerance) { stop = true; exitcode = 1; }
            else if (fabs(gm - global_last) < a.pr.relative_tolerance * global_last) { stop = true; exitcode = 2; }
            global_last = gm;
            shown = gm;
        } else {            // solver_interface.py:88-113 then :50-69
            if (merit < a.pr.absolute_tolerance) { stop = true; exitcode = 1; }
            else if (fabs(merit - last) < a.pr.relative_tolerance * last) { stop = true; exitcode = 2; }
            if (!stop) {
                if (merit > last) decision = 1;
                else { inc = last - merit < a.pr.too_small_merit_change; last = merit; }
            } else decision = 2;
            shown = merit;
        }
        if (by_residual && !check) {   // fixed r between residual tests: accept the sweep
            stop = false; exitcode = 0; decision = 0; inc = false;
        } else if (by_residual) {      // stop only on the complementarity residual
            shown = res;
            if (res <= a.pr.residual_tolerance) { stop = true; exitcode = 3; decision = 3; }
            else if (fixed_r) { stop = false; exitcode = 0; decision = 0; inc = false; }
            else {
                stop = false;
                exitcode = 0;
                if (decision == 2) {   // a merit test would have stopped: apply the accept/reject rule
                    if (merit > last) decision = 1;
                    else { inc = last - merit < a.pr.too_small_merit_change; last = merit; decision = 0; }
                }
            }
        }
        if (hist && g.rank() == 0) hist[it] = shown;
        if (decision == 1 || (decision == 0 && inc)) {
            const double nu = decision == 1 ? a.pr.nu_reduce : a.pr.nu_increase;
            for (int i = 4 * R.c0 + g.rank(); i < 4 * R.c1; i += g.size()) r[i] = nu * r[i];
        }
        // accepted, or converged by residual: the new iterate is the solution so far
        if (decision == 0 || decision == 3) { double* t = x; x = y; y = t; }
        // the residual pass computed w = WJT y; unless y was rolled back that is the next sweep's start
        w_is_wjt_x = check && decision != 1;
        g.sync();
        if (stop) { iterations = it; break; }
    }
    if (sweeps32 >= 0) iterations = exitcode == 3 ? sweeps32 + iterations : max_it;
    if (x != sol) {
        for (int i = 4 * R.c0 + g.rank(); i < 4 * R.c1; i += g.size()) sol[i] = x[i];
        g.sync();
    }
    if (by_residual && exitcode != 3) shown = scene_residual(a, g, v, x);   // residual of what is returned
    if (g.rank() == 0) {
        if (!post) {
            st->iterations = iterations; st->exitcode = exitcode; st->merit = shown;
            if (by_residual) st->residual = shown;
        } else {
            st->post_iterations = iterations; st->post_exitcode = exitcode;
        }
    }
    g.sync();
}

// ---------------------------------------------------------------------------------------------------------
// FP32 phase of the FP32 precision modes.  A scene's whole contact problem is copied into shared memory as
// FP32 in a compact form and swept there, level by level (or colour by colour), with the fixed-r rule until
// the FP32 residual meets the tolerance, stalls near FP32 rounding, or the sweep budget is spent; the iterate
// is then tested in FP64 and, if it misses the tolerance, refined by the same team with FP64 sweeps (the
// budget left).
//
// Compact form.  A contact's Jacobian rows are [lin_lo | ang_lo | lin_hi | ang_hi] with lin_hi = -lin_lo
// (the frame direction, zero on the torsion row) and W J^T = (m^-1 lin, I_w^-1 ang) per body, so a contact
// stores per row q three float4s, (lin_lo, b), (ang_lo, 1/diag) and (ang_hi, mu), and its four impulses in one more, in a
// record of kS32Floats; a body stores its accumulator w (6), m^-1, a fixed flag and the world inverse
// inertia (6, symmetric), in a record of kS32BodyFloats (all fixed bodies share one with m^-1 = I^-1 = 0).  The update
// of w after a contact changes by dx is m^-1 sum_q lin_q dx_q (negated on the hi side) and I^-1 sum_q ang_q dx_q.
//
// Execution.  A team takes scenes from its size class's queue: one warp for scenes of up to the mid slab (s32_sweep), a
// 128-thread block above (s32_sweep_turns), a 512-thread block for the scenes whose rows stay in L2 (s32_sweep_ring, or
// s32_sweep when there are too many bodies for the ring).  The four classes' launches run concurrently on separate streams.
// ---------------------------------------------------------------------------------------------------------
constexpr int kQueueFp32 = 5;                        // counters[5..8]: scene queues of the four size classes
constexpr int kClassEnd32 = 9;                       // counters[9..12]: end of each class's range in list32
constexpr int kFp32Block = 128;                      // threads per block of the large slab's launch
constexpr int kFp32L2Block = 512;                    // threads of the launch for the scenes beyond any slab
constexpr int kFp32LargeSmem = 224 * 1024;           // slab of a block team (one scene per SM)
constexpr int kS32SmallSlab = 28 * 1024;             // slab of a warp team, small class (8 scenes per SM)
constexpr int kS32MidSlab = 56 * 1024;               // slab of a warp team, mid class (4 scenes per SM)
// relative residual below which a stalled FP32 iteration may have met FP32 rounding
constexpr float kFp32Floor = 1e-5f;
// residual tests without a 5 % improvement after which an FP32 round ends in a defect correction (with the
// test every 4 sweeps: 64 sweeps; Gauss-Seidel often progresses by less than 5 % in 12 sweeps near 1e-6).
// A round that did not lower the FP64 residual by kS32RoundGain doubles the next round's window (up to
// kS32StallTestsMax): a scene whose Gauss-Seidel iteration itself has stalled keeps sweeping in FP32 with
// rare corrections, as FP64 sweeps would stall on it just the same
constexpr float kS32FarFactor = 100.0f;   // residual / tolerance above which tests are spaced twice as far
constexpr int kS32StallTests = 16;
constexpr int kS32StallTestsMax = 512;
constexpr double kS32RoundGain = 0.9;

// A scene's FP32 copy.  Only the free bodies with contacts have records ("slots", in body order), followed by one
// that stands for every fixed body, so there are at most min(bodies, 2 K) of them.
struct S32Scene {
    char* c;       // kS32Floats per contact, in level order, as thirteen float4s: (lin, b) of the four rows, then
                   // (ang_lo, 1/diag), then (ang_hi, mu), then the four impulses; the torsion row's lin is zero
    char* body;    // kS32BodyFloats per slot: (w_lin, m^-1), (w_ang, fixed), I^-1 (xx, xy, xz, yy, yz, zz), padding
    char* lohi;    // per contact in level order: slots lo | hi << 16, each with its top bit set for a fixed body
    char* pos;     // level-order position of each contact (scene-local contact index -> position), while loading
    char* bptr;    // per slot: start of its contact list in blist (n_free + 1)
    char* blist;   // per slot, its contacts in ascending order: level-order position << 1 | side (2K)
    char* steps;   // the sweep's steps: first position | contacts << 16 | flags; over pos, once that is used
    char* x;       // the impulses: float4s `xs` bytes apart (in the records, or, with the rows in a ring, on their own)
    char* ring;    // room for kRingSteps steps' records, when the rows come from L2 through it, else null
    uint32_t xs;
    int K, n_free, n_steps, warps;
};
// The rows of a scene too large for a slab stay in L2.  When the slab has room for them beside the bodies, the impulses
// and the indices, they come through a ring of six steps' records, three of each group, copied four steps ahead
// (s32_sweep_ring).
constexpr int kRingSteps = 6, kRingWarps = 4;
constexpr int kRingRecord = 192;   // a record without its impulses
constexpr int kRingSlot = 8 * kRingWarps * kRingRecord;
constexpr uint32_t kStep32Ends = 1u << 31, kStep32Wide = 1u << 30;
constexpr uint32_t kStep32Turns = 1u << 29;   // the next step is of the other width
__host__ __device__ inline size_t s32_align(size_t v) { return (v + 15) & ~size_t(15); }
// shared memory of a scene's FP32 copy with nr body records (and nb bodies); with in_l2 the contact rows, the
// level-order positions and the per-body contact lists live in global memory (L2) and only the bodies, body indices
// and level and list starts stay on chip
__host__ __device__ inline size_t s32_bytes(int K, int nb, bool in_l2 = false, bool bodies_global = false) {
    return (in_l2 ? 0 : s32_align(sizeof(float) * (size_t)K * kS32Floats) + s32_align(sizeof(uint16_t) * (size_t)K) +
                        s32_align(sizeof(uint32_t) * 2 * (size_t)K)) +
           (bodies_global ? 0 : s32_align(sizeof(float) * (size_t)nb * kS32BodyFloats)) +
           s32_align(sizeof(uint32_t) * (size_t)K) +
           s32_align(sizeof(uint16_t) * (size_t)(K + 1)) + s32_align(sizeof(uint16_t) * (size_t)(nb + 1));
}
// body records a scene can need
__host__ __device__ inline int s32_records(int K, int nb) { return nb < 2 * K ? nb : 2 * K; }
// shared memory of a scene whose rows come through the ring (the other arrays as with in_l2, and the impulses)
__host__ __device__ inline size_t s32_ring_bytes(int K, int nr) {
    return s32_align(sizeof(float) * (size_t)nr * kS32BodyFloats) + s32_align(sizeof(uint32_t) * (size_t)K) +
           s32_align(sizeof(uint16_t) * (size_t)(nr + 1)) + s32_align(4 * sizeof(float) * (size_t)K) +
           (size_t)kRingSteps * kRingSlot;
}
// with l2, the contact rows, positions, steps and body lists go to the workspace; with bodies_global the body
// records too (the scene's team is the only reader and writer, so block barriers keep them consistent)
__device__ __forceinline__ S32Scene s32_carve(char* base, int K, int nr, const StepArgs* l2 = nullptr, int c0 = 0,
                                              int s = 0, bool bodies_global = false, int b0 = 0, bool ring = false) {
    S32Scene f;
    size_t o = 0;
    auto take = [&](size_t bytes) { char* p = base + o; o += s32_align(bytes); return p; };
    f.c = l2 ? reinterpret_cast<char*>(l2->ws.c32 + kS32Floats * (size_t)c0) : take(sizeof(float) * (size_t)K * kS32Floats);
    f.body = (l2 && bodies_global) ? reinterpret_cast<char*>(l2->ws.body32 + kS32BodyFloats * (size_t)b0)
                                   : take(sizeof(float) * (size_t)nr * kS32BodyFloats);
    f.lohi = take(sizeof(uint32_t) * (size_t)K);
    // positions, then room of their size: together a word per contact for the steps (in L2: the level cursors)
    f.pos = l2 ? reinterpret_cast<char*>(l2->ws.pos32 + c0) : take(sizeof(uint16_t) * (size_t)K);
    if (!ring) take(sizeof(uint16_t) * (size_t)(K + 1));
    f.steps = l2 ? reinterpret_cast<char*>(l2->ws.lev_cur + c0 + s) : f.pos;
    f.bptr = take(sizeof(uint16_t) * (size_t)(nr + 1));
    f.blist = l2 ? reinterpret_cast<char*>(l2->ws.blist32 + 2 * (size_t)c0) : take(sizeof(uint32_t) * 2 * (size_t)K);
    f.x = ring ? take(4 * sizeof(float) * (size_t)K) : f.c + 192;
    f.xs = ring ? 16u : (uint32_t)sizeof(float) * kS32Floats;
    f.ring = ring ? take((size_t)kRingSteps * kRingSlot) : nullptr;
    f.K = K;
    f.n_free = f.n_steps = 0;
    f.warps = 1;
    return f;
}

// Addresses of a scene's copy: in shared memory by that space's own loads and stores (kept in program order, which
// is the order the sweep wants them issued in), in L2 by ordinary ones.
struct ShPtr {
    uint32_t p;
    __device__ __forceinline__ explicit ShPtr(char* q) : p((uint32_t)__cvta_generic_to_shared(q)) {}
    __device__ __forceinline__ ShPtr(uint32_t q, int) : p(q) {}
    __device__ __forceinline__ ShPtr operator+(uint32_t o) const { return ShPtr(p + o, 0); }
    __device__ __forceinline__ float4 f4() const {
        float4 v;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(p) : "memory");
        return v;
    }
    __device__ __forceinline__ float2 f2() const {
        float2 v;
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(p) : "memory");
        return v;
    }
    __device__ __forceinline__ float f1() const {
        float v;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p) : "memory");
        return v;
    }
    __device__ __forceinline__ uint32_t u32() const {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
        return v;
    }
    __device__ __forceinline__ uint32_t u16() const {
        uint32_t v;
        asm volatile("{.reg .u16 t; ld.shared.u16 t, [%1]; cvt.u32.u16 %0, t;}" : "=r"(v) : "r"(p) : "memory");
        return v;
    }
    __device__ __forceinline__ void set(float v) const { asm volatile("st.shared.f32 [%0], %1;" ::"r"(p), "f"(v) : "memory"); }
    __device__ __forceinline__ void set(float4 v) const {
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
    }
};
struct GlPtr {
    char* p;
    __device__ __forceinline__ explicit GlPtr(char* q) : p(q) {}
    __device__ __forceinline__ GlPtr operator+(uint32_t o) const { return GlPtr(p + o); }
    __device__ __forceinline__ float4 f4() const { return *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ float2 f2() const { return *reinterpret_cast<const float2*>(p); }
    __device__ __forceinline__ float f1() const { return *reinterpret_cast<const float*>(p); }
    __device__ __forceinline__ uint32_t u32() const { return *reinterpret_cast<const uint32_t*>(p); }
    __device__ __forceinline__ uint32_t u16() const { return *reinterpret_cast<const uint16_t*>(p); }
    __device__ __forceinline__ void set(float v) const { *reinterpret_cast<float*>(p) = v; }
    __device__ __forceinline__ void set(float4 v) const { *reinterpret_cast<float4*>(p) = v; }
};
constexpr uint32_t kC32 = sizeof(float) * kS32Floats, kB32 = sizeof(float) * kS32BodyFloats;   // record strides
// a contact record's offsets: piece j (0..2) of row q at 64 j + 16 q, and the impulses
constexpr uint32_t kX32 = 192;

// Warps that sweep a step of a scene of these levels: the number (a power of two, up to max_warps) with the least cost.
// In a slab (one or two warps) a level of up to eight contacts a warp is a step of quads and a wider one steps of a lane
// per contact; in tens of cycles a step by turns takes 400-420 with quads (14 to 600 contacts) and 515 with lanes (547
// contacts on six levels).  With the rows in L2 (in_l2; scenes with too many bodies for the ring, whose warps are given)
// wide levels are cut into more steps of quads.  200 sweeps of 5441 contacts on 193 levels with one, two, four and eight
// warps: 82.0, 53.3, 38.8 and 40.3 ms; of 7503 on 201: 133, 78.6, 52.8, 52.0; of 3288 on 70: 32.8, 19.7, 13.3, 12.4;
// of 1248 on 56: 5.4, 5.3, 5.5, 5.3.  The rule takes eight in the first three, so it is off the best by 4 % at most there.
// Every warp of the block counts for itself.
__device__ __forceinline__ int s32_warps(const int* ptr, int L, int max_warps, bool in_l2) {
    int cost[4] = {0, 0, 0, 0};
    const int quads[4] = {in_l2 ? 120 : 40, in_l2 ? 125 : 42, 112, 140};   // the last two in L2 alone
    const int lanes[2] = {50, 52};
    for (int l = threadIdx.x & 31; l < L; l += 32) {
        const int n = ptr[l + 1] - ptr[l];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const int q = 8 << w;
            cost[w] += in_l2 ? (n + q - 1) / q * quads[w] : n <= q ? quads[w] : (n + 4 * q - 1) / (4 * q) * lanes[w & 1];
        }
    }
    int best = 1, least = INT_MAX;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const int c = __reduce_add_sync(0xffffffffu, cost[w]);
        if ((1 << w) <= max_warps && c < least) { least = c; best = 1 << w; }
    }
    return best;
}

// copy scene R into the team's slab as FP32, contacts in level order; returns the number of levels
template <class G>
__device__ __forceinline__ int s32_load(const StepArgs& a, const G& g, const SceneRange& R, int s, S32Scene& f,
                                        bool coloured, bool in_l2, int16_t* scratch) {
    const int K = f.K;
    // levels by relaxation in shared memory when a scratch is given (the rows' room, not yet filled)
    const int L = coloured ? scene_colours(a, g, R, s)
                : scratch ? scene_levels_smem(a, g, R, s, scratch) : scene_levels(a, g, R, s);
    const int* order = a.ws.lev_order + R.c0;
    float* c = reinterpret_cast<float*>(f.c);
    // a lane per row (a quad per contact), all of whose values load together: with a lane per float4 group of a row, the
    // groups' branches each waited for L2 in turn (260 thousand cycles for 600 contacts, a tenth of 100 sweeps)
#pragma unroll 2
    for (int t = g.rank(); t < 4 * K; t += g.size()) {
        const int i = t >> 2, q = t & 3;
        const size_t k = (size_t)order[i];
        const double2* J = reinterpret_cast<const double2*>(a.ws.J + 48 * k + 2 * q);
        const double2 j0 = J[0], j1 = J[4], j2 = J[8], j4 = J[16], j5 = J[20];   // columns 0..5 and 8..11 of row q
        const double b = a.ws.b[4 * k + q], diag = a.ws.diag[4 * k + q], x = a.ws.x[4 * k + q], mu = a.ws.mu[k];
        float4* o = reinterpret_cast<float4*>(c + kS32Floats * (size_t)i) + q;
        o[0] = q < 3 ? make_float4((float)j0.x, (float)j0.y, (float)j1.x, (float)b) : make_float4(0.0f, 0.0f, 0.0f, (float)b);
        o[4] = make_float4((float)j1.y, (float)j2.x, (float)j2.y, (float)(1.0 / diag));
        o[8] = make_float4((float)j4.y, (float)j5.x, (float)j5.y, (float)mu);
        reinterpret_cast<float*>(f.x + (size_t)f.xs * i)[q] = (float)x;
    }
    // the slots: the free bodies with contacts in body order (their lists in bc_list then follow one another)
    const int e0 = a.ws.bc_ptr[R.b0];
    uint16_t* bptr = reinterpret_cast<uint16_t*>(f.bptr);
    const int n = scene_touched(a, g, R, [&](int at, int b, int p0, int) {
        bptr[at] = (uint16_t)(p0 - e0);
        reinterpret_cast<int*>(f.body + kB32 * (size_t)at)[0] = b;   // whose record it is, until the record is filled
    });
    g.sync();
    for (int i = g.rank(); i < n; i += g.size()) {
        float* B = reinterpret_cast<float*>(f.body + kB32 * (size_t)i);
        const int b = reinterpret_cast<const int*>(B)[0];
        const double* Wi = a.ws.Winv + 9 * (size_t)b;
        B[3] = (float)(1.0 / a.bd.mass[b]);
        B[7] = 0.0f;
        B[8] = (float)Wi[0]; B[9] = (float)Wi[1]; B[10] = (float)Wi[2];
        B[11] = (float)Wi[4]; B[12] = (float)Wi[5]; B[13] = (float)Wi[8];
    }
    f.n_free = n;
    if (g.rank() == 0) bptr[n] = (uint16_t)(a.ws.bc_ptr[R.b1] - e0);
    if (n < s32_records(K, R.b1 - R.b0) && g.rank() < kS32BodyFloats)   // the fixed bodies' record
        reinterpret_cast<float*>(f.body + kB32 * (size_t)n)[g.rank()] = g.rank() == 7 ? 1.0f : 0.0f;
    g.sync();   // slots complete
    uint16_t* pos = reinterpret_cast<uint16_t*>(f.pos);
    uint32_t* lohi = reinterpret_cast<uint32_t*>(f.lohi);
#pragma unroll 4
    for (int i = g.rank(); i < K; i += g.size()) {
        const int k = order[i];
        pos[k - R.c0] = (uint16_t)i;
        const int lo = a.ws.lohi[2 * k], hi = a.ws.lohi[2 * k + 1];
        lohi[i] = (uint32_t)(a.bd.fixed[lo] ? 0x8000 | n : a.ws.bc_fill[lo]) |
                  ((uint32_t)(a.bd.fixed[hi] ? 0x8000 | n : a.ws.bc_fill[hi]) << 16);
    }
    g.sync();   // pos complete
    // per-body contact lists (the residual's w = W J^T x), positions in level order
    uint32_t* blist = reinterpret_cast<uint32_t*>(f.blist);
    const int entries = a.ws.bc_ptr[R.b1] - e0;
#pragma unroll 4
    for (int e = g.rank(); e < entries; e += g.size()) {
        const int code = a.ws.bc_list[e0 + e];
        blist[e] = ((uint32_t)pos[(code >> 1) - R.c0] << 1) | (uint32_t)(code & 1);
    }
    g.sync();   // pos used: the steps take its room
    const int* ptr = a.ws.lev_ptr + R.c0 + s;
    f.warps = f.ring ? kRingWarps : s32_warps(ptr, L, in_l2 ? g.size() >> 5 : g.size() >> 6, in_l2);
    uint32_t* steps = reinterpret_cast<uint32_t*>(f.steps);
    f.n_steps = sweep_steps(g, ptr, L, in_l2 ? 0 : 8 * f.warps, in_l2 ? 8 * f.warps : 32 * f.warps, [&](int at, int start, int count, bool ends, bool wide) {
        steps[at] = (uint32_t)start | ((uint32_t)count << 16) | (ends ? kStep32Ends : 0u) | (wide && !in_l2 ? kStep32Wide : 0u);
    });
    g.sync();
    for (int i = g.rank(); i < f.n_steps; i += g.size())   // (reads only the widths of others, which stay)
        if (((steps[i] ^ steps[i + 1 < f.n_steps ? i + 1 : 0]) & kStep32Wide) != 0) atomicOr(steps + i, kStep32Turns);
    g.sync();
    return L;
}

// w = W J^T x: two lanes per slot, one for the linear and one for the angular components, each body's contacts
// summed in ascending order
template <class P, class G>
__device__ __noinline__ void s32_rebuild_w(const G g, const S32Scene f) {
    const P c(f.c), body(f.body), bptr(f.bptr), blist(f.blist), xp(f.x);
    const int ang = g.rank() & 1;
    for (int i = g.rank() >> 1; i < f.n_free; i += g.size() >> 1) {
        uint32_t e = (bptr + 2u * i).u16();
        const uint32_t e1 = (bptr + (2u * i + 2u)).u16();
        const P B = body + kB32 * i;
        float S[3] = {0.f, 0.f, 0.f};
        float4 v[2][4], x[2];   // two contacts at a time: their loads are under way together
        auto fetch = [&](int t, uint32_t code) {
            const uint32_t side = code & 1u;
            const P col = c + (kC32 * (code >> 1) + (ang ? 64u + 64u * side : 0u));
#pragma unroll
            for (int k = 0; k < 4; ++k) v[t][k] = (col + 16u * k).f4();
            x[t] = (xp + f.xs * (code >> 1)).f4();
            const float sg = !ang && side ? -1.0f : 1.0f;   // lin_hi = -lin_lo
            x[t] = make_float4(sg * x[t].x, sg * x[t].y, sg * x[t].z, sg * x[t].w);
        };
        auto add = [&](int t) {
            const float xs[4] = {x[t].x, x[t].y, x[t].z, x[t].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                S[0] = fmaf(v[t][k].x, xs[k], S[0]);
                S[1] = fmaf(v[t][k].y, xs[k], S[1]);
                S[2] = fmaf(v[t][k].z, xs[k], S[2]);
            }
        };
        uint32_t code0 = (blist + 4u * e).u32(), code1 = (blist + 4u * min(e + 1u, e1 - 1u)).u32();
        for (; e + 1u < e1; e += 2u) {
            fetch(0, code0);
            fetch(1, code1);
            code0 = (blist + 4u * min(e + 2u, e1 - 1u)).u32();
            code1 = (blist + 4u * min(e + 3u, e1 - 1u)).u32();
            add(0);
            add(1);
        }
        if (e < e1) { fetch(0, code0); add(0); }
        const float4 I0 = (B + 32u).f4();
        const float2 I1 = (B + 48u).f2();
        if (ang) {
            (B + 16u).set(make_float4(fmaf(I0.x, S[0], fmaf(I0.y, S[1], I0.z * S[2])),
                                      fmaf(I0.y, S[0], fmaf(I0.w, S[1], I1.x * S[2])),
                                      fmaf(I0.z, S[0], fmaf(I1.x, S[1], I1.y * S[2])), 0.0f));
        } else {
            const float m = (B + 12u).f1();
            B.set(make_float4(m * S[0], m * S[1], m * S[2], m));
        }
    }
    g.sync();
}

// J_q . [w_lo; w_hi] of a contact's row q: three partial sums, then their total (the torsion row's lin is zero)
__device__ __forceinline__ float s32_jw(float4 r0, float4 r1, float4 r2, float4 l0, float4 l1, float4 h0, float4 h1) {
    const float lin = fmaf(r0.x, l0.x - h0.x, fmaf(r0.y, l0.y - h0.y, r0.z * (l0.z - h0.z)));
    const float alo = fmaf(r1.x, l1.x, fmaf(r1.y, l1.y, r1.z * l1.z));
    const float ahi = fmaf(r2.x, h1.x, fmaf(r2.y, h1.y, r2.z * h1.z));
    return (lin + alo) + ahi;
}
__device__ __forceinline__ void quad_gather(float z, float* o) {
    const int base = (threadIdx.x & 31) & ~3;
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = __shfl_sync(0xffffffffu, z, base | i);
}

// w = W J^T x, then the FP32 residual ||x - prox(x - D^-1 (A x + b))||_inf / max(1, ||x||_inf), a quad per contact
template <class P, class G>
__device__ __noinline__ float s32_residual(const G g, const S32Scene f) {
    s32_rebuild_w<P>(g, f);
    const P c(f.c), body(f.body), lohi(f.lohi), xp(f.x);
    const int q = g.rank() & 3, nslot = g.size() >> 2;
    float m = 0.0f, xm = 0.0f;
    for (int i0 = 0; i0 < f.K; i0 += nslot) {
        const int at = i0 + (g.rank() >> 2), i = min(at, f.K - 1);
        const uint32_t lh = (lohi + 4u * i).u32();
        const P rec = c + kC32 * i, row = rec + 16u * q;
        const P Bl = body + kB32 * (lh & 0x7fffu), Bh = body + kB32 * ((lh >> 16) & 0x7fffu);
        const float4 r0 = row.f4(), r1 = (row + 64u).f4(), r2 = (row + 128u).f4();
        const float4 l0 = Bl.f4(), l1 = (Bl + 16u).f4(), h0 = Bh.f4(), h1 = (Bh + 16u).f4();
        const float x = (xp + (f.xs * i + 4u * q)).f1();
        float z[4];
        const float zq = x - r1.w * (s32_jw(r0, r1, r2, l0, l1, h0, h1) + r0.w);
        quad_gather(zq, z);
        const float pn = fmaxf(z[0], 0.0f);
        const float radius = r2.w * pn;
        const float sqr = fmaf(z[1], z[1], fmaf(z[2], z[2], z[3] * z[3]));
        const float fr = pn <= 0.0f ? 0.0f : (sqr <= radius * radius ? zq : zq * (radius * rsqrtf(sqr)));
        const float d = x - (q == 0 ? pn : fr);
        if (at < f.K) {
            m = nanmax(m, fabsf(d));
            xm = fmaxf(xm, fabsf(x));
        }
    }
    double mres = (double)m, mx = (double)xm;
    g.max2(mres, mx);
    return (float)(mres / (mx > 1.0 ? mx : 1.0));
}

// n_sweeps projected Gauss-Seidel sweeps over the levels, as one sequence of steps.  A narrow step takes a quad of
// lanes per contact: lane q computes z_q from the current w, the four z meet by shuffles and every lane applies the
// prox (branch-free); the lane then forms one 3-vector of the update -- lin columns for the lo and the hi body (lanes
// 0 and 1), ang_lo (2), ang_hi (3) -- applies that part of W to it and stores its float4 of w (the linear lanes apply
// m^-1 as a diagonal matrix).  A wide step takes one lane per contact, which computes all four rows as independent
// chains and updates both bodies.  Every expression has the same operands in the same order, so both give the same
// bits.
//
// Bound by one contact's chain (~250 cycles: row product, reciprocal root, update, shared-memory store and load) and by
// the instructions of a step, which one warp issues every ~2.5 cycles: ~150 with a quad per contact, ~250 with a lane.
// A step of quads takes ~420 cycles and one of lanes ~700, but the quads of four warps hold one another up in the
// shared-memory pipe (four 128-byte wavefronts a load: 560 cycles).  (One lane per contact at every level, its rows
// loaded after the level's barrier: ~570 cycles.)  The values of the next step's
// contact are loaded as soon as the current ones are used up, its indices a step before that, and the loads and
// shuffles, which share one queue, are issued in the order of their need.
template <class P, class G>
__device__ __noinline__ void s32_sweep(const G g, const S32Scene f, float rscale, int n_sweeps) {
    const P c(f.c), body(f.body), lohi(f.lohi), steps(f.steps);
    const int rank = g.rank(), last = f.n_steps - 1;
    auto step = [&](int j) { return (steps + 4u * j).u32(); };
    auto after = [&](int j) { return j < last ? j + 1 : 0; };   // the sequence goes on from sweep to sweep
    int j = 0;
    uint32_t st0 = step(0);
#pragma unroll 1
    for (int left = n_sweeps * f.n_steps; left > 0;) {
        if (!(st0 & kStep32Wide)) {
            // a run of narrow steps
            const int q = rank & 3, slot = rank >> 2;
            const bool linear = q < 2;
            const uint32_t hi_shift = (q & 1) ? 16u : 0u;          // lanes 1 and 3 update the hi body
            const uint32_t fixed_bit = 0x8000u << hi_shift;
            const uint32_t part = linear ? 0u : 16u;                // their float4 of w
            const uint32_t col = linear ? 0u : 64u * (uint32_t)(q - 1);   // the piece whose columns the lane sums
            const float sg = q == 1 ? -1.0f : 1.0f;
            auto at = [&](uint32_t st) { return min((int)(st & 0x7fffu) + slot, f.K - 1); };
            int j2 = after(after(j));
            uint32_t st1 = step(after(j));
            P rec = c + kC32 * at(st0);
            uint32_t lh = (lohi + 4u * at(st0)).u32();
            float4 r0 = (rec + 16u * q).f4(), r1 = (rec + (64u + 16u * q)).f4(), r2 = (rec + (128u + 16u * q)).f4();
            float4 x = (rec + kX32).f4();
            float xq = (rec + (kX32 + 4u * q)).f1();
            int i_next = at(st1);
            uint32_t lh_next = (lohi + 4u * i_next).u32();
            bool more;
#pragma unroll 1
            do {
                const P Bl = body + kB32 * (lh & 0x7fffu), Bh = body + kB32 * ((lh >> 16) & 0x7fffu);
                const float4 l0 = Bl.f4(), h0 = Bh.f4(), l1 = (Bl + 16u).f4(), h1 = (Bh + 16u).f4();
                const float zq = xq - rscale * r1.w * (s32_jw(r0, r1, r2, l0, l1, h0, h1) + r0.w);
                float z[4];
                quad_gather(zq, z);
                const P cl = rec + col;
                const float4 v0 = cl.f4(), v1 = (cl + 16u).f4(), v2 = (cl + 32u).f4(), v3 = (cl + 48u).f4();
                const P B = body + kB32 * ((lh >> hi_shift) & 0x7fffu);
                const float4 own = (B + part).f4();
                const float4 I0 = (B + 32u).f4();
                const float2 I1 = (B + 48u).f2();
                const float xn = fmaxf(z[0], 0.0f);
                // prox onto the friction ball of radius mu xn
                const float radius = r2.w * xn;
                const float sqr = fmaf(z[1], z[1], fmaf(z[2], z[2], z[3] * z[3]));
                float scale = sqr > radius * radius ? radius * rsqrtf(sqr) : 1.0f;
                if (xn <= 0.0f) scale = 0.0f;
                const uint32_t st2 = step(j2);
                j2 = after(j2);
                const P rec_next = c + kC32 * i_next;
                r0 = (rec_next + 16u * q).f4(); r1 = (rec_next + (64u + 16u * q)).f4(); r2 = (rec_next + (128u + 16u * q)).f4();
                const float f1 = z[1] * scale, f2 = z[2] * scale, f3 = z[3] * scale;
                const float d0 = xn - x.x, d1 = f1 - x.y, d2 = f2 - x.z, d3 = f3 - x.w;
                const float yq = q == 0 ? xn : zq * scale;
                // the lane's part of W: m^-1 on the diagonal (negative for the hi body: lin_hi = -lin_lo), or I^-1
                const float m = sg * own.w;
                const float wxx = linear ? m : I0.x, wxy = linear ? 0.0f : I0.y, wxz = linear ? 0.0f : I0.z;
                const float wyy = linear ? m : I0.w, wyz = linear ? 0.0f : I1.x, wzz = linear ? m : I1.y;
                const float S0 = fmaf(v3.x, d3, fmaf(v2.x, d2, fmaf(v1.x, d1, v0.x * d0)));
                const float S1 = fmaf(v3.y, d3, fmaf(v2.y, d2, fmaf(v1.y, d1, v0.y * d0)));
                const float S2 = fmaf(v3.z, d3, fmaf(v2.z, d2, fmaf(v1.z, d1, v0.z * d0)));
                const float4 n = make_float4(own.x + fmaf(wxx, S0, fmaf(wxy, S1, wxz * S2)),
                                             own.y + fmaf(wxy, S0, fmaf(wyy, S1, wyz * S2)),
                                             own.z + fmaf(wxz, S0, fmaf(wyz, S1, wzz * S2)), own.w);
                // the fixed bodies' record is only read; an idle quad writes nothing
                const bool mine = slot < (int)((st0 >> 16) & 0x1fffu);
                if (mine && !(lh & fixed_bit)) (B + part).set(n);
                if (mine) (rec + (kX32 + 4u * q)).set(yq);
                // after the stores of all four lanes: a scene of one step sweeps the same contacts again, and each lane
                // loads what the other three of its quad stored
                __syncwarp();
                x = (rec_next + kX32).f4();
                xq = (rec_next + (kX32 + 4u * q)).f1();
                if (st0 & kStep32Ends) g.sync();
                more = --left > 0 && !(st0 & kStep32Turns);
                st0 = st1; st1 = st2;
                rec = rec_next;
                lh = lh_next;
                i_next = at(st2);
                lh_next = (lohi + 4u * i_next).u32();
                j = after(j);
            } while (more);
        } else {
            // a run of wide steps
            auto at = [&](uint32_t st) { return min((int)(st & 0x7fffu) + rank, f.K - 1); };
            uint32_t st1 = step(after(j));
            P rec = c + kC32 * at(st0);
            uint32_t lh = (lohi + 4u * at(st0)).u32();
            float4 r[12];
#pragma unroll
            for (int t = 0; t < 12; ++t) r[t] = (rec + 16u * t).f4();
            float4 x = (rec + kX32).f4();
            bool more;
#pragma unroll 1
            do {
                const P Bl = body + kB32 * (lh & 0x7fffu), Bh = body + kB32 * ((lh >> 16) & 0x7fffu);
                const float4 l0 = Bl.f4(), h0 = Bh.f4(), l1 = (Bl + 16u).f4(), h1 = (Bh + 16u).f4();
                const float xs[4] = {x.x, x.y, x.z, x.w};
                float z[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 r0 = r[k], r1 = r[4 + k], r2 = r[8 + k];
                    float lin = 0.0f;
                    if (k < 3) lin = fmaf(r0.x, l0.x - h0.x, fmaf(r0.y, l0.y - h0.y, r0.z * (l0.z - h0.z)));
                    const float alo = fmaf(r1.x, l1.x, fmaf(r1.y, l1.y, r1.z * l1.z));
                    const float ahi = fmaf(r2.x, h1.x, fmaf(r2.y, h1.y, r2.z * h1.z));
                    z[k] = xs[k] - rscale * r1.w * (((lin + alo) + ahi) + r0.w);
                }
                const float mu = r[8].w;
                float4 v[12];   // the rows once more, for the update: the next ones take r
#pragma unroll
                for (int t = 0; t < 12; ++t) v[t] = (rec + 16u * t).f4();
                const float4 Il0 = (Bl + 32u).f4(), Ih0 = (Bh + 32u).f4();
                const float2 Il1 = (Bl + 48u).f2(), Ih1 = (Bh + 48u).f2();
                const P rec_next = c + kC32 * at(st1);
                const uint32_t lh_next = (lohi + 4u * at(st1)).u32();
#pragma unroll
                for (int t = 0; t < 12; ++t) r[t] = (rec_next + 16u * t).f4();
                const float xn = fmaxf(z[0], 0.0f);
                const float radius = mu * xn;
                const float sqr = fmaf(z[1], z[1], fmaf(z[2], z[2], z[3] * z[3]));
                float scale = sqr > radius * radius ? radius * rsqrtf(sqr) : 1.0f;
                if (xn <= 0.0f) scale = 0.0f;
                const float f1 = z[1] * scale, f2 = z[2] * scale, f3 = z[3] * scale;
                const float d0 = xn - x.x, d1 = f1 - x.y, d2 = f2 - x.z, d3 = f3 - x.w;
                // the three sums of the update (the torsion row has no linear columns)
                const float L0 = fmaf(v[2].x, d2, fmaf(v[1].x, d1, v[0].x * d0));
                const float L1 = fmaf(v[2].y, d2, fmaf(v[1].y, d1, v[0].y * d0));
                const float L2 = fmaf(v[2].z, d2, fmaf(v[1].z, d1, v[0].z * d0));
                const float A0 = fmaf(v[7].x, d3, fmaf(v[6].x, d2, fmaf(v[5].x, d1, v[4].x * d0)));
                const float A1 = fmaf(v[7].y, d3, fmaf(v[6].y, d2, fmaf(v[5].y, d1, v[4].y * d0)));
                const float A2 = fmaf(v[7].z, d3, fmaf(v[6].z, d2, fmaf(v[5].z, d1, v[4].z * d0)));
                const float H0 = fmaf(v[11].x, d3, fmaf(v[10].x, d2, fmaf(v[9].x, d1, v[8].x * d0)));
                const float H1 = fmaf(v[11].y, d3, fmaf(v[10].y, d2, fmaf(v[9].y, d1, v[8].y * d0)));
                const float H2 = fmaf(v[11].z, d3, fmaf(v[10].z, d2, fmaf(v[9].z, d1, v[8].z * d0)));
                const float ml = l0.w, mh = -h0.w;
                const bool mine = rank < (int)((st0 >> 16) & 0x1fffu);
                if (mine && !(lh & 0x8000u)) {
                    Bl.set(make_float4(l0.x + ml * L0, l0.y + ml * L1, l0.z + ml * L2, ml));
                    (Bl + 16u).set(make_float4(l1.x + fmaf(Il0.x, A0, fmaf(Il0.y, A1, Il0.z * A2)),
                                               l1.y + fmaf(Il0.y, A0, fmaf(Il0.w, A1, Il1.x * A2)),
                                               l1.z + fmaf(Il0.z, A0, fmaf(Il1.x, A1, Il1.y * A2)), 0.0f));
                }
                if (mine && !(lh & 0x80000000u)) {
                    Bh.set(make_float4(h0.x + mh * L0, h0.y + mh * L1, h0.z + mh * L2, h0.w));
                    (Bh + 16u).set(make_float4(h1.x + fmaf(Ih0.x, H0, fmaf(Ih0.y, H1, Ih0.z * H2)),
                                               h1.y + fmaf(Ih0.y, H0, fmaf(Ih0.w, H1, Ih1.x * H2)),
                                               h1.z + fmaf(Ih0.z, H0, fmaf(Ih1.x, H1, Ih1.y * H2)), 0.0f));
                }
                if (mine) (rec + kX32).set(make_float4(xn, f1, f2, f3));
                x = (rec_next + kX32).f4();
                if (st0 & kStep32Ends) g.sync();
                more = --left > 0 && !(st0 & kStep32Turns);
                j = after(j);
                st0 = st1;
                st1 = step(after(j));
                rec = rec_next;
                lh = lh_next;
            } while (more);
        }
    }
}

// n_sweeps sweeps of a slab scene by two groups of f.warps warps that take the steps by turns (as gs_sweep_turns does in
// FP64): while one computes a step, the other loads all that its next step's contacts do not have from w, so that only
// the chain itself -- the accumulators' loads, the row products, the prox, the update and its stores -- lies between the
// barriers.  The steps and their expressions are s32_sweep's: a quad of lanes per contact, or in a wide step a lane.
// A step's impulses are stored after its barrier, so a sweep has at least five steps (kTurnsSteps): the next one to load
// them, five or more steps on, has by then passed a barrier that the storing group reached later.
__device__ __noinline__ void s32_sweep_turns(const S32Scene f, float rscale, int n_sweeps) {
    const ShPtr c(f.c), body(f.body), lohi(f.lohi), steps(f.steps);
    const int half = 32 * f.warps, group = (int)threadIdx.x >= half, rank = threadIdx.x - group * half;
    const int q = rank & 3, quad = rank >> 2;
    const bool linear = q < 2;
    const uint32_t hi_shift = (q & 1) ? 16u : 0u;          // lanes 1 and 3 update the hi body
    const uint32_t fixed_bit = 0x8000u << hi_shift;
    const uint32_t part = linear ? 0u : 16u;                // their float4 of w
    const uint32_t col = linear ? 0u : 64u * (uint32_t)(q - 1);   // the piece whose columns the lane sums
    const float sg = q == 1 ? -1.0f : 1.0f;
    const int n_steps = f.n_steps, total = n_sweeps * n_steps;
    auto at = [&](uint32_t st) { return min((int)(st & 0x7fffu) + ((st & kStep32Wide) ? rank : quad), f.K - 1); };
    int place = group < n_steps ? group : 0;   // the step's place in its sweep
    uint32_t st_next = (steps + 4u * place).u32();
    uint32_t lh_next = (lohi + 4u * at(st_next)).u32();
#pragma unroll 1
    for (int j = group; j < total; j += 2) {
        const uint32_t st = st_next, lh = lh_next;
        const ShPtr rec = c + kC32 * at(st);
        const ShPtr Bl = body + kB32 * (lh & 0x7fffu), Bh = body + kB32 * ((lh >> 16) & 0x7fffu);
        place += 2;
        while (place >= n_steps) place -= n_steps;
        st_next = (steps + 4u * place).u32();
        const int count = (int)((st >> 16) & 0x1fffu);
        if (!(st & kStep32Wide)) {
            const float4 r0 = (rec + 16u * q).f4(), r1 = (rec + (64u + 16u * q)).f4(), r2 = (rec + (128u + 16u * q)).f4();
            const ShPtr cl = rec + col;
            const float4 v0 = cl.f4(), v1 = (cl + 16u).f4(), v2 = (cl + 32u).f4(), v3 = (cl + 48u).f4();
            const ShPtr B = body + kB32 * ((lh >> hi_shift) & 0x7fffu);
            const float4 I0 = (B + 32u).f4();
            const float2 I1 = (B + 48u).f2();
            const float wxy = linear ? 0.0f : I0.y, wxz = linear ? 0.0f : I0.z, wyz = linear ? 0.0f : I1.x;
            const bool mine = quad < count, put = mine && !(lh & fixed_bit);
            lh_next = (lohi + 4u * at(st_next)).u32();
            const float rs = rscale * r1.w;
            const float4 x = (rec + kX32).f4();
            const float xq = (rec + (kX32 + 4u * q)).f1();
            if (j > 0) turn_wait(group, 2 * half);
            const float4 l0 = Bl.f4(), h0 = Bh.f4(), l1 = (Bl + 16u).f4(), h1 = (Bh + 16u).f4();
            const float4 own = (B + part).f4();
            const float zq = xq - rs * (s32_jw(r0, r1, r2, l0, l1, h0, h1) + r0.w);
            float z[4];
            quad_gather(zq, z);
            // the lane's part of W: m^-1 on the diagonal (negative for the hi body: lin_hi = -lin_lo), or I^-1
            const float m = sg * own.w;
            const float wxx = linear ? m : I0.x, wyy = linear ? m : I0.w, wzz = linear ? m : I1.y;
            const float xn = fmaxf(z[0], 0.0f);
            // prox onto the friction ball of radius mu xn
            const float radius = r2.w * xn;
            const float sqr = fmaf(z[1], z[1], fmaf(z[2], z[2], z[3] * z[3]));
            float scale = sqr > radius * radius ? radius * rsqrtf(sqr) : 1.0f;
            if (xn <= 0.0f) scale = 0.0f;
            const float f1 = z[1] * scale, f2 = z[2] * scale, f3 = z[3] * scale;
            const float d0 = xn - x.x, d1 = f1 - x.y, d2 = f2 - x.z, d3 = f3 - x.w;
            const float S0 = fmaf(v3.x, d3, fmaf(v2.x, d2, fmaf(v1.x, d1, v0.x * d0)));
            const float S1 = fmaf(v3.y, d3, fmaf(v2.y, d2, fmaf(v1.y, d1, v0.y * d0)));
            const float S2 = fmaf(v3.z, d3, fmaf(v2.z, d2, fmaf(v1.z, d1, v0.z * d0)));
            const float4 n = make_float4(own.x + fmaf(wxx, S0, fmaf(wxy, S1, wxz * S2)),
                                         own.y + fmaf(wxy, S0, fmaf(wyy, S1, wyz * S2)),
                                         own.z + fmaf(wxz, S0, fmaf(wyz, S1, wzz * S2)), own.w);
            // the fixed bodies' record is only read; an idle quad writes nothing
            if (put) (B + part).set(n);
            if (j + 1 < total) turn_done(group, 2 * half);
            if (mine) (rec + (kX32 + 4u * q)).set(q == 0 ? xn : zq * scale);
        } else {
            float4 r[12];
#pragma unroll
            for (int t = 0; t < 12; ++t) r[t] = (rec + 16u * t).f4();
            const float4 Il0 = (Bl + 32u).f4(), Ih0 = (Bh + 32u).f4();
            const float2 Il1 = (Bl + 48u).f2(), Ih1 = (Bh + 48u).f2();
            const bool mine = rank < count;
            lh_next = (lohi + 4u * at(st_next)).u32();
            const float4 x = (rec + kX32).f4();
            if (j > 0) turn_wait(group, 2 * half);
            const float4 l0 = Bl.f4(), h0 = Bh.f4(), l1 = (Bl + 16u).f4(), h1 = (Bh + 16u).f4();
            const float xs[4] = {x.x, x.y, x.z, x.w};
            float z[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 r0 = r[k], r1 = r[4 + k], r2 = r[8 + k];
                float lin = 0.0f;
                if (k < 3) lin = fmaf(r0.x, l0.x - h0.x, fmaf(r0.y, l0.y - h0.y, r0.z * (l0.z - h0.z)));
                const float alo = fmaf(r1.x, l1.x, fmaf(r1.y, l1.y, r1.z * l1.z));
                const float ahi = fmaf(r2.x, h1.x, fmaf(r2.y, h1.y, r2.z * h1.z));
                z[k] = xs[k] - rscale * r1.w * (((lin + alo) + ahi) + r0.w);
            }
            const float xn = fmaxf(z[0], 0.0f);
            const float radius = r[8].w * xn;
            const float sqr = fmaf(z[1], z[1], fmaf(z[2], z[2], z[3] * z[3]));
            float scale = sqr > radius * radius ? radius * rsqrtf(sqr) : 1.0f;
            if (xn <= 0.0f) scale = 0.0f;
            const float f1 = z[1] * scale, f2 = z[2] * scale, f3 = z[3] * scale;
            const float d0 = xn - x.x, d1 = f1 - x.y, d2 = f2 - x.z, d3 = f3 - x.w;
            // the three sums of the update (the torsion row has no linear columns)
            const float L0 = fmaf(r[2].x, d2, fmaf(r[1].x, d1, r[0].x * d0));
            const float L1 = fmaf(r[2].y, d2, fmaf(r[1].y, d1, r[0].y * d0));
            const float L2 = fmaf(r[2].z, d2, fmaf(r[1].z, d1, r[0].z * d0));
            const float A0 = fmaf(r[7].x, d3, fmaf(r[6].x, d2, fmaf(r[5].x, d1, r[4].x * d0)));
            const float A1 = fmaf(r[7].y, d3, fmaf(r[6].y, d2, fmaf(r[5].y, d1, r[4].y * d0)));
            const float A2 = fmaf(r[7].z, d3, fmaf(r[6].z, d2, fmaf(r[5].z, d1, r[4].z * d0)));
            const float H0 = fmaf(r[11].x, d3, fmaf(r[10].x, d2, fmaf(r[9].x, d1, r[8].x * d0)));
            const float H1 = fmaf(r[11].y, d3, fmaf(r[10].y, d2, fmaf(r[9].y, d1, r[8].y * d0)));
            const float H2 = fmaf(r[11].z, d3, fmaf(r[10].z, d2, fmaf(r[9].z, d1, r[8].z * d0)));
            const float ml = l0.w, mh = -h0.w;
            if (mine && !(lh & 0x8000u)) {
                Bl.set(make_float4(l0.x + ml * L0, l0.y + ml * L1, l0.z + ml * L2, ml));
                (Bl + 16u).set(make_float4(l1.x + fmaf(Il0.x, A0, fmaf(Il0.y, A1, Il0.z * A2)),
                                           l1.y + fmaf(Il0.y, A0, fmaf(Il0.w, A1, Il1.x * A2)),
                                           l1.z + fmaf(Il0.z, A0, fmaf(Il1.x, A1, Il1.y * A2)), 0.0f));
            }
            if (mine && !(lh & 0x80000000u)) {
                Bh.set(make_float4(h0.x + mh * L0, h0.y + mh * L1, h0.z + mh * L2, h0.w));
                (Bh + 16u).set(make_float4(h1.x + fmaf(Ih0.x, H0, fmaf(Ih0.y, H1, Ih0.z * H2)),
                                           h1.y + fmaf(Ih0.y, H0, fmaf(Ih0.w, H1, Ih1.x * H2)),
                                           h1.z + fmaf(Ih0.z, H0, fmaf(Ih1.x, H1, Ih1.y * H2)), 0.0f));
            }
            if (j + 1 < total) turn_done(group, 2 * half);
            if (mine) (rec + kX32).set(make_float4(xn, f1, f2, f3));
        }
        __syncwarp();   // a quad's impulses are stored by its four lanes and loaded by each of them
    }
}
constexpr int kTurnsSteps = 5;

// The float4 of w that lane q updates, of the four that it has.  With two groups of four warps the shared-memory pipe is
// what a step waits for, and loading it again costs more than the choice (clock-counted 570 against 517 cycles a step); with two groups
// of one or two warps it is the other way round (424 against 434).
__device__ __forceinline__ float4 s32_own(int q, float4 l0, float4 l1, float4 h0, float4 h1) {
    const bool hi = q & 1, linear = q < 2;
    return make_float4(linear ? (hi ? h0.x : l0.x) : (hi ? h1.x : l1.x), linear ? (hi ? h0.y : l0.y) : (hi ? h1.y : l1.y),
                       linear ? (hi ? h0.z : l0.z) : (hi ? h1.z : l1.z), linear ? (hi ? h0.w : l0.w) : 0.0f);
}

// The narrow steps of s32_sweep_turns for a scene whose rows come through the ring.  Each group has three of its slots and
// a warp that copies its steps' records, contiguous in level order, into them (asynchronous 16-byte copies, one group a
// step): a step's records are asked for two of the group's own steps ahead, four of the sweep's.  A barrier of the group
// and its copying warp tells the one that the rows are there and the other that the slot before is free: a group has all
// of a step's rows in registers before it waits for its turn.  A scene comes here with more than 600 contacts (its copy
// is too large for a slab), so a sweep has more steps than kTurnsSteps.
//
// Bound by the shared-memory pipe of its SM: a warp's step takes about 80 wavefronts of 128 bytes, and eight warps share
// the pipe with the copies.  1566 contacts in 80 steps, 200 sweeps and their tests: 5540 us, 6250 with the records as they
// lie in L2 (13 float4s apart, two of a quad's columns in one bank), 6310 with all four warps on every step and one ring.
// (Clock-counted copies of the kernel, whose registers fall otherwise: 517 cycles a step, 687 with records as in L2.)
//
// A group of four pieces (lin, ang_lo, ang_hi of the four rows) is kept turned by its number, so that neither the quads'
// loads of a row each nor those of a column, of two contacts at a time, meet twice in a bank.
__host__ __device__ constexpr uint32_t ring_piece(int group, int row) { return 64u * group + 16u * ((row + group) & 3); }
__device__ __forceinline__ void ring_sync(int group) {   // written with their numbers, as in turn_wait
    if (group) asm volatile("bar.sync 4, %0;" ::"n"(32 * kRingWarps + 32) : "memory");
    else asm volatile("bar.sync 3, %0;" ::"n"(32 * kRingWarps + 32) : "memory");
}
__device__ __noinline__ void s32_sweep_ring(const S32Scene f, float rscale, int n_sweeps) {
    constexpr int half = 32 * kRingWarps, kPlaces = kRingSteps / 2;
    const GlPtr steps(f.steps);
    const int n_steps = f.n_steps, total = n_sweeps * n_steps;
    auto on = [&](int step) { return step + 2 < n_steps ? step + 2 : step + 2 - n_steps; };
    auto next_place = [&](int p) { return p + 1 < kPlaces ? p + 1 : 0; };
    if (threadIdx.x >= 2 * half) {   // a group's copying warp
        const int group = ((int)threadIdx.x - 2 * half) >> 5, lane = threadIdx.x & 31;
        const ShPtr ring = ShPtr(f.ring) + (uint32_t)kRingSlot * (kPlaces * group);
        int step = group, place = 0;
        uint32_t st = (steps + 4u * step).u32();
        uint32_t src[3], dst[3];   // three times 32 pieces are those of eight records
        for (int a = 0; a < 3; ++a) {
            const int t = lane + 32 * a, r = t / 12, p = t % 12;
            src[a] = kC32 * r + 16u * p;
            dst[a] = kRingRecord * r + ring_piece(p >> 2, p & 3);
        }
        auto copy = [&]() {   // the records of the group's next step
            const char* from = f.c + (size_t)kC32 * (st & 0x7fffu);
            const int pieces = 12 * (int)((st >> 16) & 0x1fffu);
            step = on(step);
            st = (steps + 4u * step).u32();
            const uint32_t to = (ring + (uint32_t)kRingSlot * place).p;
#pragma unroll
            for (int m = 0; m < 3 * kRingWarps; ++m)
                if (lane + 32 * m < pieces)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::
                                 "r"(to + dst[m % 3] + 8 * kRingRecord * (m / 3)), "l"(from + src[m % 3] + 8 * kC32 * (m / 3)) : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
            place = next_place(place);
        };
        copy();
        copy();
        for (int j = group; j < total; j += 2) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            ring_sync(group);
            copy();
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        return;
    }
    const ShPtr body(f.body), lohi(f.lohi), xp(f.x);
    const int group = (int)threadIdx.x >= half, rank = threadIdx.x - group * half;
    const int q = rank & 3, slot = rank >> 2;
    const ShPtr ring = ShPtr(f.ring) + (uint32_t)(kRingSlot * (kPlaces * group) + kRingRecord * slot);
    const bool linear = q < 2;
    const uint32_t hi_shift = (q & 1) ? 16u : 0u;
    const uint32_t fixed_bit = 0x8000u << hi_shift;
    const uint32_t part = linear ? 0u : 16u;
    const float sg = q == 1 ? -1.0f : 1.0f;
    const uint32_t row0 = ring_piece(0, q), row1 = ring_piece(1, q), row2 = ring_piece(2, q);
    const int cg = linear ? 0 : q - 1;   // the group of pieces whose columns the lane sums
    const uint32_t col0 = ring_piece(cg, 0), col1 = ring_piece(cg, 1), col2 = ring_piece(cg, 2), col3 = ring_piece(cg, 3);
    auto at = [&](uint32_t st) { return min((int)(st & 0x7fffu) + slot, f.K - 1); };
    int step = group, place = 0;
    uint32_t st_next = (steps + 4u * step).u32();
    int i_next = at(st_next);
    uint32_t lh_next = (lohi + 4u * i_next).u32();
#pragma unroll 1
    for (int j = group; j < total; j += 2) {
        const uint32_t st = st_next, lh = lh_next;
        const int i = i_next;
        step = on(step);
        st_next = (steps + 4u * step).u32();
        const ShPtr Bl = body + kB32 * (lh & 0x7fffu), Bh = body + kB32 * ((lh >> 16) & 0x7fffu);
        const ShPtr B = body + kB32 * ((lh >> hi_shift) & 0x7fffu);
        const bool mine = slot < (int)((st >> 16) & 0x1fffu), put = mine && !(lh & fixed_bit);
        const ShPtr rec = ring + (uint32_t)kRingSlot * place;
        place = next_place(place);
        ring_sync(group);
        const float4 r0 = (rec + row0).f4(), r1 = (rec + row1).f4(), r2 = (rec + row2).f4();
        const float xq = (xp + (16u * i + 4u * q)).f1();
        const float4 v0 = (rec + col0).f4(), v1 = (rec + col1).f4(), v2 = (rec + col2).f4(), v3 = (rec + col3).f4();
        const float4 x = (xp + 16u * i).f4();
        const float4 I0 = (B + 32u).f4();
        const float2 I1 = (B + 48u).f2();
        const float wxy = linear ? 0.0f : I0.y, wxz = linear ? 0.0f : I0.z, wyz = linear ? 0.0f : I1.x;
        const float rs = rscale * r1.w;
        i_next = at(st_next);
        lh_next = (lohi + 4u * i_next).u32();
        if (j > 0) turn_wait(group, 2 * half);
        const float4 l0 = Bl.f4(), h0 = Bh.f4(), l1 = (Bl + 16u).f4(), h1 = (Bh + 16u).f4();
        const float4 own = s32_own(q, l0, l1, h0, h1);
        const float zq = xq - rs * (s32_jw(r0, r1, r2, l0, l1, h0, h1) + r0.w);
        float z[4];
        quad_gather(zq, z);
        const float m = sg * own.w;
        const float wxx = linear ? m : I0.x, wyy = linear ? m : I0.w, wzz = linear ? m : I1.y;
        const float xn = fmaxf(z[0], 0.0f);
        const float radius = r2.w * xn;
        const float sqr = fmaf(z[1], z[1], fmaf(z[2], z[2], z[3] * z[3]));
        float scale = sqr > radius * radius ? radius * rsqrtf(sqr) : 1.0f;
        if (xn <= 0.0f) scale = 0.0f;
        const float f1 = z[1] * scale, f2 = z[2] * scale, f3 = z[3] * scale;
        const float d0 = xn - x.x, d1 = f1 - x.y, d2 = f2 - x.z, d3 = f3 - x.w;
        const float S0 = fmaf(v3.x, d3, fmaf(v2.x, d2, fmaf(v1.x, d1, v0.x * d0)));
        const float S1 = fmaf(v3.y, d3, fmaf(v2.y, d2, fmaf(v1.y, d1, v0.y * d0)));
        const float S2 = fmaf(v3.z, d3, fmaf(v2.z, d2, fmaf(v1.z, d1, v0.z * d0)));
        const float4 n = make_float4(own.x + fmaf(wxx, S0, fmaf(wxy, S1, wxz * S2)),
                                     own.y + fmaf(wxy, S0, fmaf(wyy, S1, wyz * S2)),
                                     own.z + fmaf(wxz, S0, fmaf(wyz, S1, wzz * S2)), own.w);
        if (put) (B + part).set(n);
        if (j + 1 < total) turn_done(group, 2 * half);
        if (mine) (xp + (16u * i + 4u * q)).set(q == 0 ? xn : zq * scale);
        __syncwarp();   // a quad's impulses are stored by its four lanes and loaded by each of them
    }
}

// n_sweeps sweeps by as many of the team's warps as the scene's levels keep busy
template <class P, class G>
__device__ __forceinline__ void s32_sweep_team(const G& g, const S32Scene& f, float rscale, int n_sweeps) {
    if (std::is_same_v<G, WarpGroup>) {
        s32_sweep<P>(WarpGroup{}, f, rscale, n_sweeps);
    } else if (std::is_same_v<P, GlPtr> && f.ring) {
        if (threadIdx.x < 64 * (kRingWarps + 1)) s32_sweep_ring(f, rscale, n_sweeps);
    } else if (std::is_same_v<P, ShPtr> && f.n_steps >= kTurnsSteps) {
        if ((int)threadIdx.x < 64 * f.warps) s32_sweep_turns(f, rscale, n_sweeps);
    } else if (f.warps == 1) {
        if (threadIdx.x < 32) s32_sweep<P>(WarpGroup{}, f, rscale, n_sweeps);
    } else if ((int)threadIdx.x < 32 * f.warps) {
        s32_sweep<P>(SubGroup{32 * f.warps}, f, rscale, n_sweeps);
    }
    g.sync();
}

// One proximal Jacobi sweep (proximal_contact/jacobi_solver.py:41-57) on the FP32 copy: every contact's new
// impulse from the accumulators w = W J^T x of the previous iterate, a quad per contact as in the Gauss-Seidel
// sweep (any order: no contact reads another's new impulse), then w rebuilt from the new impulses.  hybrid
// (jacobi_solver.py:60-79): the friction ball's radius uses the new normal impulse instead of the previous one.
template <class P, class G>
__device__ __noinline__ void s32_sweep_jacobi(const G g, const S32Scene f, float rscale, bool hybrid) {
    const P c(f.c), body(f.body), lohi(f.lohi);
    const int q = g.rank() & 3, nslot = g.size() >> 2;
    for (int i0 = 0; i0 < f.K; i0 += nslot) {
        const int at = i0 + (g.rank() >> 2), i = min(at, f.K - 1);
        const uint32_t lh = (lohi + 4u * i).u32();
        const P rec = c + kC32 * i, row = rec + 16u * q;
        const P Bl = body + kB32 * (lh & 0x7fffu), Bh = body + kB32 * ((lh >> 16) & 0x7fffu);
        const float4 r0 = row.f4(), r1 = (row + 64u).f4(), r2 = (row + 128u).f4();
        const float4 l0 = Bl.f4(), l1 = (Bl + 16u).f4(), h0 = Bh.f4(), h1 = (Bh + 16u).f4();
        const float x = (rec + kX32 + 4u * q).f1();
        float z[4];
        const float zq = x - rscale * r1.w * (s32_jw(r0, r1, r2, l0, l1, h0, h1) + r0.w);
        quad_gather(zq, z);
        const float xn_old = __shfl_sync(0xffffffffu, x, (threadIdx.x & 31) & ~3);
        const float xn = fmaxf(z[0], 0.0f), bound = hybrid ? xn : xn_old;
        const float radius = r2.w * bound;
        const float sqr = fmaf(z[1], z[1], fmaf(z[2], z[2], z[3] * z[3]));
        const float fr = bound <= 0.0f ? 0.0f : (sqr <= radius * radius ? zq : zq * (radius * rsqrtf(sqr)));
        if (at < f.K) (rec + kX32 + 4u * q).set(q == 0 ? xn : fr);
    }
    g.sync();
    s32_rebuild_w<P>(g, f);
}

// FP64 check of the FP32 iterate and defect correction of the FP32 problem.  With x the current FP32 iterate,
// evaluates A x + b in FP64 (J, W J^T and b of the FP64 problem, w in the scene's global FP64 accumulators)
// and in FP32 (the shared copy), adds the difference to the FP32 b, and returns the FP64 residual
// ||x - prox(x - D^-1 (A x + b))||_inf / max(1, ||x||_inf).  The FP32 sweeps that follow then converge to the
// FP64 problem's solution: at the current x the corrected FP32 problem has the FP64 problem's residual.  The
// FP32 w must hold W J^T x for this x (the residual test just before rebuilt it).
template <class P, class G>
__device__ __forceinline__ double s32_correct(const StepArgs& a, const G& g, const SceneRange& R, const S32Scene& f,
                                              bool correct = true) {
    const P c(f.c), body(f.body), lohi(f.lohi), bptr(f.bptr), blist(f.blist), xp(f.x);
    const int K = f.K;
    const int* order = a.ws.lev_order + R.c0;
    double* w64 = a.ws.w + 6 * (size_t)R.b0;   // by slot; the scene's FP64 accumulators, unused until the FP64 solve
    for (int i = g.rank(); i < 6 * f.n_free; i += g.size()) {   // a thread per component
        const int bl = i / 6, d = i - 6 * bl;
        double acc = 0.0;
        const uint32_t e1 = (bptr + (2u * bl + 2u)).u16();
        for (uint32_t e = (bptr + 2u * bl).u16(); e < e1; ++e) {
            const uint32_t code = (blist + 4u * e).u32();
            double W[4];
            w_column(a.ws.WJT, order[code >> 1], 6 * (int)(code & 1u) + d, W);
            const float4 x = (xp + f.xs * (code >> 1)).f4();
            acc = fma(W[0], (double)x.x, acc);
            acc = fma(W[1], (double)x.y, acc);
            acc = fma(W[2], (double)x.z, acc);
            acc = fma(W[3], (double)x.w, acc);
        }
        w64[i] = acc;
    }
    if (f.n_free < s32_records(K, R.b1 - R.b0) && g.rank() < 6) w64[6 * f.n_free + g.rank()] = 0.0;
    g.sync();
    double m = 0.0, xm = 0.0;
    const int q = g.rank() & 3, nslot = g.size() >> 2;
    for (int i0 = 0; i0 < K; i0 += nslot) {   // a quad per contact
        const int at = i0 + (g.rank() >> 2), i = min(at, K - 1);
        const size_t k = (size_t)order[i];
        const uint32_t lh = (lohi + 4u * i).u32();
        const double* wl = w64 + 6 * (lh & 0x7fffu);
        const double* wh = w64 + 6 * ((lh >> 16) & 0x7fffu);
        const double2* J = reinterpret_cast<const double2*>(a.ws.J + 48 * k + 2 * q);
        double v64 = a.ws.b[4 * k + q];
#pragma unroll
        for (int t = 0; t < 6; ++t) {
            const double2 j2 = J[4 * t];
            const double* w = t < 3 ? wl + 2 * t : wh + 2 * t - 6;
            v64 = fma(j2.x, w[0], v64);
            v64 = fma(j2.y, w[1], v64);
        }
        const P rec = c + kC32 * i, row = rec + 16u * q;
        if (correct && at < K) {
            const P Bl = body + kB32 * (lh & 0x7fffu), Bh = body + kB32 * ((lh >> 16) & 0x7fffu);
            const float4 r0 = row.f4();
            const float v32 = s32_jw(r0, (row + 64u).f4(), (row + 128u).f4(), Bl.f4(), (Bl + 16u).f4(), Bh.f4(), (Bh + 16u).f4()) + r0.w;
            (row + 12u).set(r0.w + (float)(v64 - (double)v32));
        }
        const double x = (double)(xp + (f.xs * i + 4u * q)).f1();
        const double zq = x - v64 / a.ws.diag[4 * k + q];
        double z[4];
        quad_gather(zq, z);
        const double pn = z[0] > 0.0 ? z[0] : 0.0;
        double scale;
        const int kind = prox_factor(z, a.ws.mu[k], pn, scale);
        const double d = x - (q == 0 ? pn : prox_apply(kind, scale, zq));
        if (at < K) {
            m = nanmax(m, fabs(d));
            xm = fmax(xm, fabs(x));
        }
    }
    g.max2(m, xm);
    g.sync();
    return m / (xm > 1.0 ? xm : 1.0);
}

// size class of a scene's FP32 copy: 0 and 1 warp teams with small and mid slabs, 2 block teams with the
// large slab, 3 block teams with the contact rows in L2; -1 for a scene the FP32 phase leaves to FP64
__host__ __device__ inline int s32_class(int K, int nb, size_t small_slab, size_t mid_slab) {
    if (K == 0 || K > 32767 || nb > 32767) return -1;   // 16-bit positions and list offsets
    const int nr = s32_records(K, nb);
    const size_t bytes = s32_bytes(K, nr);
    if (bytes <= small_slab) return 0;
    if (bytes <= mid_slab) return 1;
    if (bytes <= (size_t)kFp32LargeSmem) return 2;
    const bool bodies_global = s32_bytes(K, nb, true) > (size_t)kFp32LargeSmem;
    return s32_bytes(K, nb, true, bodies_global) <= (size_t)kFp32LargeSmem ? 3 : -1;
}

// Per-scene FP32 bookkeeping of the step, and the scene list of each size class, longest expected chain
// first, so that every team's next scene is one of its class and the scenes that bound the step start first.
// The expected chain of a scene is its previous step's levels x sweeps (the solve length in level steps,
// the sweeps floored at half the cap), read before this step resets them; without a plausible history (first
// step, a scene new to its slot) it is estimated from the contact count.  The order decides only which team takes which scene and when, never a
// result.  One block.
constexpr int kClassBuckets = 64;
__global__ void __launch_bounds__(1024) k_fp32_classes(const StepArgs a, size_t small_slab, size_t mid_slab) {
    __shared__ int cnt[4 * kClassBuckets];
    const int S = a.bd.n_scenes;
    // no lists after an overflow: the contact ranges are not valid then, and the solvers do not run
    const bool fp32 = !a.ws.counters[kAbort];
    const int max_it = a.pr.max_iterations;
    for (int t = threadIdx.x; t < 4 * kClassBuckets; t += blockDim.x) cnt[t] = 0;
    __syncthreads();
    auto slot = [&](int s) -> int {   // class x buckets + expected-chain bucket (descending), or -1
        const SceneRange R = scene_range(a, s);
        const int K = R.c1 - R.c0;
        const int c = s32_class(K, R.b1 - R.b0, small_slab, mid_slab);
        if (c < 0) return -1;
        // previous levels x sweeps, the sweeps floored at half the cap: whether a scene converges early varies
        // from step to step, and one that converged last step may run to the cap in this one
        const int Lp = a.ws.nlev[s], Sp = a.ws.sweeps32[s];
        const bool known = Lp > 0 && Lp <= K && Sp > 0 && Sp <= max_it;
        const float w = known ? (float)Lp * (float)max(Sp, max_it / 2) : 0.25f * (float)K * (float)max_it;
        const int lg = (int)(2.0f * log2f(w + 1.0f));   // buckets of a factor 2^(1/2)
        return kClassBuckets * c + kClassBuckets - 1 - min(lg, kClassBuckets - 1);
    };
    if (fp32)
        for (int s = threadIdx.x; s < S; s += blockDim.x) {
            const int t = slot(s);
            if (t >= 0) atomicAdd(&cnt[t], 1);
        }
    __syncthreads();
    if (fp32 && threadIdx.x == 0) {   // counts -> starts; class ends to the counters
        int run = 0;
        for (int t = 0; t < 4 * kClassBuckets; ++t) {
            const int n = cnt[t];
            cnt[t] = run;
            run += n;
            if ((t % kClassBuckets) == kClassBuckets - 1) a.ws.counters[kClassEnd32 + t / kClassBuckets] = run;
        }
    }
    __syncthreads();
    for (int s = threadIdx.x; s < S; s += blockDim.x) {   // the thread that keyed scene s places and resets it
        if (fp32) {
            const int t = slot(s);
            if (t >= 0) a.ws.list32[atomicAdd(&cnt[t], 1)] = s;
        }
        a.ws.sweeps32[s] = -1;
        a.ws.fin32[s] = 0;
    }
}

template <class G>
__device__ __forceinline__ int team_next(const G& g, int* counter, int* slot) {
    if constexpr (std::is_same_v<G, WarpGroup>) {
        int s = 0;
        if (g.rank() == 0) s = atomicAdd(counter, 1);
        return __shfl_sync(0xffffffffu, s, 0);
    } else {
        if (g.rank() == 0) *slot = atomicAdd(counter, 1);
        __syncthreads();
        const int s = *slot;
        __syncthreads();
        return s;
    }
}

// the FP64 solve of a scene as a call of its own, so that it does not raise the FP32 kernel's registers
template <class G>
__device__ __noinline__ void solve_scene_call(const StepArgs& a, const G& g, int s) {
    solve_scene(a, g, s, 0, nullptr, 0);
}

// FP32 phase for the scenes whose compact copy takes lo_bytes < bytes <= slab bytes, a block per scene.  kL2: the scenes
// too large for any slab, with their contact rows in global memory (L2-resident) and the rest of the copy in the slab.
// The small and mid slabs' scenes take one warp each (G = WarpGroup): by turns their steps are a little shorter (396
// against ~430 cycles), but the team's barriers in every residual test take more than that (32-box tower, 200 sweeps:
// 530 us with one warp, 638 with two).
template <class G, bool kL2, int kThreads>
__global__ void __launch_bounds__(kThreads, 1) k_solve_fp32(const StepArgs a, int queue, size_t lo_bytes, size_t slab) {
    extern __shared__ __align__(16) char f32_smem[];
    __shared__ double red[33];
    __shared__ int ired[33];
    __shared__ int next_slot;
    if (a.ws.counters[kAbort]) return;
    G g;
    if constexpr (std::is_same_v<G, BlockGroup>) { g.red = red; g.ired = ired; }
    using P = std::conditional_t<kL2, GlPtr, ShPtr>;
    char* my_slab = f32_smem;
    const int max_it = a.pr.max_iterations;
    const int interval = a.pr.residual_interval > 1 ? a.pr.residual_interval : 1;
    // the FP32 sweeps aim a little below the tolerance when an FP64 test follows, so that the FP32 problem
    // rarely meets it while the FP64 one misses it
    const float tol = (float)(a.pr.precision == RB_PRECISION_FP32_REFINE ? 0.5 * a.pr.residual_tolerance
                                                                        : a.pr.residual_tolerance);
    // sweeps reserved for the FP64 refinement
    const int reserve = a.pr.precision == RB_PRECISION_FP32_REFINE ? min(max(a.pr.refine_iterations, 0), max_it) : 0;
    const int budget = max_it - reserve;
    double rs = a.pr.scheme == RB_SCHEME_RIGID_GS ? 1.0 : 0.1;   // the r of the scheme: r = rs / diag
    if (a.pr.relaxation > 0.0) rs *= a.pr.relaxation;
    const float rscale = (float)rs;
    const bool coloured = a.pr.scheme == RB_SCHEME_COLOURED_GS || a.pr.ordering == RB_ORDER_COLOURED;
    const bool jacobi = a.pr.scheme == RB_SCHEME_JACOBI || a.pr.scheme == RB_SCHEME_JACOBI_HYBRID;
    const bool hybrid = a.pr.scheme == RB_SCHEME_JACOBI_HYBRID;
    const int cls = queue - kQueueFp32;
    const int list0 = cls == 0 ? 0 : a.ws.counters[kClassEnd32 + cls - 1];
    const int list1 = a.ws.counters[kClassEnd32 + cls];
    for (;;) {
        const int idx = list0 + team_next(g, a.ws.counters + queue, &next_slot);
        if (idx >= list1) break;
        const int s = a.ws.list32[idx];
        const SceneRange R = scene_range(a, s);
        const int K = R.c1 - R.c0, nb = R.b1 - R.b0;
        if (K == 0 || K > 32767 || nb > 32767) continue;   // 16-bit positions and list offsets
        const int nr = s32_records(K, nb);
        bool bodies_global = false;
        if (kL2) {   // the scenes no slab holds whole: contact rows in L2, and the bodies too if they do not fit
            if (s32_bytes(K, nr) <= lo_bytes) continue;
            bodies_global = s32_bytes(K, nr, true) > slab;
            if (s32_bytes(K, nr, true, bodies_global) > slab) continue;
        } else {
            const size_t bytes = s32_bytes(K, nr);
            if (bytes <= lo_bytes || bytes > slab) continue;
        }
        const double t0 = a.pr.profiling ? device_us() : 0.0;
        const bool ring = kL2 && !jacobi && s32_ring_bytes(K, nr) <= slab;
        S32Scene f = s32_carve(my_slab, K, nr, kL2 ? &a : nullptr, R.c0, s, bodies_global, R.b0, ring);
        // scratch for the level relaxation: the rows' room of the slab, or with rows in L2 what the slab has left
        int16_t* scratch = nullptr;
        if (!kL2) {   // a contact record's bytes per contact there, more than s32_level_scratch needs
            scratch = reinterpret_cast<int16_t*>(f.c);
        } else {
            const size_t off = (s32_bytes(K, nr, true, bodies_global) + 15) & ~size_t(15);
            if (ring) scratch = reinterpret_cast<int16_t*>(f.x);   // 16 bytes a contact and the ring after them
            else if (off + s32_level_scratch(K) <= slab) scratch = reinterpret_cast<int16_t*>(my_slab + off);
        }
        const int L = s32_load(a, g, R, s, f, coloured, kL2, scratch);
        if (g.rank() == 0) a.ws.nlev[s] = L;
        float res = s32_residual<P>(g, f);   // the warm-started iterate may already be good enough
        float best = res;
        int sweeps = 0, stalls = 0, window = kS32StallTests;
        // far above the tolerance (and the stall floor) the residual is tested half as often: no stop and no
        // stall can be decided there, and each test rebuilds w
        // (unsigned: twice any interval fits)
        auto gap = [&](float r) { return r > kS32FarFactor * tol ? 2u * (unsigned)interval : (unsigned)interval; };
        unsigned next_test = gap(res);
        // sweeps of one call, whose steps are counted in 32 bits
        const unsigned most = (unsigned)(INT_MAX / f.n_steps);
        double r64 = -1.0;            // FP64 residual of the current iterate, once evaluated
        double r64_round = INFINITY;  // FP64 residual after the previous correction round
        for (;;) {
            const int round_start = sweeps;
            while (res > tol && sweeps < budget) {
                // as far as the next test
                const unsigned n = jacobi ? 1u : min(min(next_test, (unsigned)(budget - sweeps)), most);
                if (jacobi) s32_sweep_jacobi<P>(g, f, rscale, hybrid);
                else s32_sweep_team<P>(g, f, rscale, (int)n);
                sweeps += (int)n;
                next_test -= n;
                if (next_test == 0 || sweeps == budget) {
                    res = s32_residual<P>(g, f);
                    next_test = gap(res);
                    // a round ends once the residual, already small, stops improving for a while (the FP32
                    // problem's own rounding, or slow progress a defect correction may speed up).  Above the
                    // floor a pause is the Gauss-Seidel iteration itself (it is not monotone), so go on.
                    if (res < 0.95f * best) { best = res; stalls = 0; }
                    else if (best < kFp32Floor && ++stalls >= window) break;
                }
            }
            // FP32 + refinement: test in FP64; if the FP32 answer misses the tolerance in FP64, correct the FP32
            // problem's b by the FP64 defect and sweep on in FP32.  FP64 sweeps take over only when the FP32
            // problem meets the tolerance and the FP64 one does not (the FP32 sweeps can do no more).
            if (a.pr.precision != RB_PRECISION_FP32_REFINE || sweeps >= budget) break;
            r64 = s32_correct<P>(a, g, R, f);
            if (r64 <= a.pr.residual_tolerance) break;
            if (sweeps == round_start) break;   // r64 stays valid for x
            if (r64 > kS32RoundGain * r64_round) window = min(2 * window, kS32StallTestsMax);
            r64_round = fmin(r64_round, r64);
            r64 = -1.0;   // the sweeps that follow change the iterate
            res = s32_residual<P>(g, f);
            next_test = gap(res);
            best = res;
            stalls = 0;
        }
        // the FP64 residual of the iterate decides whether FP64 sweeps follow; when none do, this kernel
        // finishes the scene (solution, statistics), and when some do, this team runs them right away, so
        // the FP64 solver launched after the FP32 phase skips the scene either way
        if (r64 < 0.0) r64 = s32_correct<P>(a, g, R, f, false);
        const bool finished = r64 <= a.pr.residual_tolerance || sweeps >= max_it ||
                              a.pr.precision == RB_PRECISION_FP32;
        for (int t = g.rank(); t < 4 * K; t += g.size()) {   // back to contact order
            const int i = t >> 2, q = t & 3;
            const size_t k4 = 4 * (size_t)a.ws.lev_order[R.c0 + i] + q;
            const double xv = (double)(P(f.x) + (f.xs * i + 4u * q)).f1();
            a.ws.x[k4] = xv;
            if (finished) a.out.contact_sol[k4] = xv;
        }
        if (finished && a.out.residuals && a.pr.profiling)
            for (int i = g.rank(); i < max_it; i += g.size()) a.out.residuals[(size_t)s * a.caps.max_iterations + i] = INFINITY;
        if (g.rank() == 0) {
            a.ws.sweeps32[s] = sweeps;
            a.ws.fin32[s] = finished ? 1 : 0;
            rb_scene_stats* st = a.out.stats + s;
            st->solve_start_us = t0;
            st->solve_us = a.pr.profiling ? device_us() - t0 : 0.0;
            if (finished) {
                const bool ok = r64 <= a.pr.residual_tolerance;
                st->n_contacts = K; st->contact_start = R.c0;
                st->iterations = ok ? max(sweeps - 1, 0) : max_it;
                st->exitcode = ok ? 3 : 0;
                st->merit = r64; st->residual = r64;
                st->post_iterations = -1; st->post_exitcode = -1;
                st->n_levels = L; st->fp32_sweeps = sweeps;
            }
        }
        g.sync();
        if (!kL2 && !finished) {   // FP64 sweeps with the budget left, by this team at once (w in global memory)
            solve_scene_call(a, g, s);
            if (g.rank() == 0) a.ws.fin32[s] = 1;
            g.sync();
        }
    }
}

constexpr int kSolveBlock = 256;   // threads per scene in the block solver, at most
constexpr int kWarpSceneMaxContacts = 2048;
constexpr int kWarpSceneMaxBodies = 384;
constexpr int kSolveWarpsPerBlock = 4;

__device__ __forceinline__ int scene_contacts(const StepArgs& a, int s) {
    const SceneRange R = scene_range(a, s);
    return R.c1 - R.c0;
}

// scenes with at most kWarpSceneMaxContacts contacts and warp_bodies bodies: one warp each
__global__ void __launch_bounds__(32 * kSolveWarpsPerBlock) k_solve_warps(const StepArgs a, int post, int warp_bodies) {
    extern __shared__ __align__(16) double wsm[];
    if (a.ws.counters[kAbort]) return;
    const WarpGroup g;
    const int wib = threadIdx.x >> 5;
    double* w_smem = warp_bodies > 0 ? wsm + (size_t)wib * 6 * (warp_bodies + 1) : nullptr;
    for (int s = blockIdx.x * kSolveWarpsPerBlock + wib; s < a.bd.n_scenes; s += gridDim.x * kSolveWarpsPerBlock) {
        const int nb = a.bd.scene_start[s + 1] - a.bd.scene_start[s];
        if (scene_contacts(a, s) > kWarpSceneMaxContacts || nb > warp_bodies) continue;
        solve_scene(a, g, s, post, w_smem, warp_bodies + 1);
    }
}

// the other scenes: one block each; the body accumulators are on chip up to smem_bodies bodies
__global__ void __launch_bounds__(kSolveBlock) k_solve_blocks(const StepArgs a, int post, int warp_bodies, int smem_bodies) {
    extern __shared__ __align__(16) double wsm[];
    __shared__ double red[33];
    __shared__ int ired[33];
    if (a.ws.counters[kAbort]) return;
    const BlockGroup g = {red, ired};
    for (int s = blockIdx.x; s < a.bd.n_scenes; s += gridDim.x) {
        const int nb = a.bd.scene_start[s + 1] - a.bd.scene_start[s];
        if (scene_contacts(a, s) <= kWarpSceneMaxContacts && nb <= warp_bodies) continue;
        solve_scene(a, g, s, post, wsm, smem_bodies);
    }
}

// ---------------------------------------------------------------------------------------------------------
// integration (state_storage.py:239 velocity_update, :251 position_update)
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void position_update(double* xb, const double* ub, double dt) {
    for (int i = 0; i < 3; ++i) xb[i] = xb[i] + ub[i] * dt;
    const double qw[4] = {0.0, ub[3], ub[4], ub[5]};
    double q[4] = {xb[3], xb[4], xb[5], xb[6]}, dq[4], qn[4];
    quat_prod(qw, q, dq);
    for (int i = 0; i < 4; ++i) qn[i] = q[i] + (dq[i] * dt) * 0.5;
    quat_unit(qn, xb + 3);
}

// six lanes per body, one velocity component each (the sums over a body's contacts are chains of 4 additions a
// contact); the first of them moves the body
__global__ void k_integrate(const StepArgs a) {
    if (a.ws.counters[kAbort]) return;
    int d;
    const int b = body_of_six(a.bd.n_bodies, d);
    const bool fixed = b < 0 || a.bd.fixed[b];
    double ud = 0.0;
    if (b >= 0) {
        double du = a.ws.du[6 * b + d];
        const int e0 = a.ws.bc_ptr[b], e1 = a.ws.bc_ptr[b + 1];
        if (!fixed && e1 > e0) du = du + body_wjt_dot(a.ws, e0, e1, d, a.out.contact_sol);   // steppers.py:84-85
        if (a.bd.n_hinges > 0 && !fixed && a.ws.hbody_ptr[b + 1] > a.ws.hbody_ptr[b]) {
            // then the hinge problem's WJT sol (hinges.py:52), hinges ascending, 5 rows each
            double t = 0.0;
            for (int e = a.ws.hbody_ptr[b]; e < a.ws.hbody_ptr[b + 1]; ++e) {
                const int code = a.ws.hbody_list[e];
                const int k = code >> 1, side = code & 1;
                const double* Wk = a.ws.hWJT + 60 * (size_t)k + 6 * side;
                for (int row = 0; row < 5; ++row) t += Wk[12 * row + d] * a.ws.hsol[5 * (size_t)k + row];
            }
            du = du + t;
        }
        ud = a.bd.u[6 * b + d] + du;
        a.bd.u[6 * b + d] = ud;
    }
    double ub[6];
    gather_six(ud, ub);
    if (fixed || d != 0) return;
    position_update(a.bd.x + 7 * b, ub, a.pr.dt);
    bool finite = true;
    for (int i = 0; i < 7; ++i) finite &= isfinite(a.bd.x[7 * b + i]);
    for (int i = 0; i < 6; ++i) finite &= isfinite(ub[i]);
    if (!finite) atomicOr(a.out.status, RB_STATUS_NONFINITE);
}

// post-stabilisation problem (post_stabilization.py:30-104): b = gap on deep normal rows, r = 1/diag
__global__ void k_post_setup(const StepArgs a) {
    if (a.ws.counters[kAbort]) return;
    const int K = a.ws.counters[kNContacts];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += gridDim.x * blockDim.x) {
        const double g = a.out.contact_g[k];
        for (int row = 0; row < 4; ++row) {
            a.ws.b[4 * k + row] = (row == 0 && g < -a.pr.min_gap_value) ? g : 0.0;
            a.ws.r[4 * k + row] = 1.0 / a.ws.diag[4 * k + row];
            a.ws.x[4 * k + row] = 0.0;
            a.ws.xold[4 * k + row] = 0.0;
        }
    }
}
__global__ void k_post_apply(const StepArgs a) {
    if (a.ws.counters[kAbort]) return;
    int d;
    const int b = body_of_six(a.bd.n_bodies, d);
    // every non-fixed body of a corrected scene is updated (and its quaternion renormalised), contacts or not;
    // a scene with post_iterations < 0 had nothing to correct
    const bool moves = b >= 0 && !a.bd.fixed[b] &&
                       a.out.stats[scene_of(a.bd.scene_start, a.bd.n_scenes, b)].post_iterations >= 0;
    double dr[6];
    gather_six(moves ? body_wjt_dot(a.ws, a.ws.bc_ptr[b], a.ws.bc_ptr[b + 1], d, a.ws.xold) : 0.0, dr);
    if (moves && d == 0) position_update(a.bd.x + 7 * b, dr, 1.0);
}

// energies and largest penetration (state_storage.py:188, contacts.py:222)
// one warp per scene: the deepest gap and the pair / candidate counts by warp reductions (order-free), the
// energy sums by lane 0 in body order (their rounding follows state_storage.py:188-237)
__device__ __forceinline__ void scene_summary(const StepArgs& a, int s) {
    const int lane = threadIdx.x & 31;
    rb_scene_stats* st = a.out.stats + s;
    const SceneRange R = scene_range(a, s);
    double gap = 0.0;
    for (int k = R.c0 + lane; k < R.c1; k += 32) gap = fmin(gap, a.out.contact_g[k]);
    for (int o = 16; o > 0; o >>= 1) gap = fmin(gap, __shfl_xor_sync(0xffffffffu, gap, o));
    const int p0 = a.ws.pair_cnt[R.b0], p1 = a.ws.pair_cnt[R.b1];
    int ovl = 0, cand = 0;
    if (a.pr.profiling)
        for (int p = p0 + lane; p < p1; p += 32) { ovl += a.ws.pair_ovl[p]; cand += a.ws.pair_n_items[p]; }
    for (int o = 16; o > 0; o >>= 1) {
        ovl += __shfl_xor_sync(0xffffffffu, ovl, o);
        cand += __shfl_xor_sync(0xffffffffu, cand, o);
    }
    if (lane != 0) return;
    st->max_penetration = -gap;
    st->n_pairs = p1 - p0;
    st->n_candidates = cand;
    st->n_leaf_overlaps = ovl;
    if (!a.pr.profiling) return;
    int has_gravity = 0;
    for (int f = a.bd.scene_force_start[s]; f < a.bd.scene_force_start[s + 1]; ++f)
        if (a.bd.force_kind[f] == 0) has_gravity = 1;
    // the per-body terms come from k_body_energy
    double kinetic = 0.0, potential = 0.0;
#pragma unroll 8
    for (int b = R.b0; b < R.b1; ++b) {
        if (a.bd.fixed[b]) continue;
        if (has_gravity) potential += a.ws.eterm[2 * (size_t)b + 1];
        kinetic += a.ws.eterm[2 * (size_t)b];
    }
    st->kinetic_energy = kinetic;
    st->potential_energy = potential;
}

// per-body energy terms of a profiled step (StateStorage.compute_total_energy, state_storage.py:188-237):
// 0.5 (m v.v + w.(I_w w)) and m g (up . r) with the scene's summed gravity
__global__ void k_body_energy(const StepArgs a) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= a.bd.n_bodies || a.ws.counters[kAbort]) return;
    double* out = a.ws.eterm + 2 * (size_t)b;
    if (a.bd.fixed[b]) { out[0] = 0.0; out[1] = 0.0; return; }
    const int s = scene_of(a.bd.scene_start, a.bd.n_scenes, b);
    double G[3] = {0.0, 0.0, 0.0};
    int has_gravity = 0;
    for (int f = a.bd.scene_force_start[s]; f < a.bd.scene_force_start[s + 1]; ++f)
        if (a.bd.force_kind[f] == 0) {
            const double* fp = a.bd.force_params + 4 * f;
            for (int i = 0; i < 3; ++i) G[i] = G[i] + fp[1 + i] * fp[0];
            has_gravity = 1;
        }
    const double* xb = a.bd.x + 7 * b;
    double Rm[9], Iw[9], Ib[3] = {a.bd.inertia[3 * b], a.bd.inertia[3 * b + 1], a.bd.inertia[3 * b + 2]};
    quat_to_matrix(xb + 3, Rm);
    update_inertia_tensor(Rm, Ib, Iw);
    const double m = a.bd.mass[b];
    double pot = 0.0;
    if (has_gravity) {
        const d3 Gv = d3{G[0], G[1], G[2]};
        const double ln = norm3_np(Gv);
        const d3 up = d3{G[0] / ln, G[1] / ln, G[2] / ln};
        const double g = norm3_np(Gv);
        const double h = dot3_np(up, ld3(xb));
        pot = m * g * h;
    }
    const d3 v = ld3(a.bd.u + 6 * b), w = ld3(a.bd.u + 6 * b + 3);
    const double wIw = dot3_np(w, gemv3_np(Iw, w));
    out[0] = 0.5 * (m * dot3_np(v, v) + wIw);
    out[1] = pot;
}

// The end of the step: the scenes' summaries by the first blocks, and by the others this step's contact keys and impulses
// kept for the next step's warm start; one thread writes the totals.
__global__ void __launch_bounds__(128) k_outputs(const StepArgs a, int summary_blocks) {
    const int ab = a.ws.counters[kAbort];
    if ((int)blockIdx.x < summary_blocks) {
        const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        if (s < a.bd.n_scenes && !ab) scene_summary(a, s);
        return;
    }
    const int at = (blockIdx.x - summary_blocks) * blockDim.x + threadIdx.x;
    if (at == 0) {
        if (a.out.n_contacts_total) *a.out.n_contacts_total = a.ws.counters[kNContacts];
        if (a.out.needed) {   // a stage after an overflow did not run: its total is reported as 0
            a.out.needed[0] = a.ws.counters[kNPairs];
            a.out.needed[1] = (ab & RB_STATUS_PAIR_OVERFLOW) ? 0 : a.ws.counters[kNItems];
            a.out.needed[2] = (ab & (RB_STATUS_PAIR_OVERFLOW | RB_STATUS_ITEM_OVERFLOW)) ? 0 : a.ws.counters[kNContacts];
        }
    }
    if (ab || !a.out.cache_key || !a.out.cache_sol || !a.out.cache_count) return;
    const int K = min(a.ws.counters[kNContacts], a.caps.contact_capacity);
    for (int k = at; k < K; k += (gridDim.x - summary_blocks) * blockDim.x) {
        a.out.cache_key[2 * k] = a.ws.ckey[2 * k];
        a.out.cache_key[2 * k + 1] = a.ws.ckey[2 * k + 1];
        for (int row = 0; row < 4; ++row) a.out.cache_sol[4 * k + row] = a.out.contact_sol[4 * k + row];
    }
    if (at == 0) *a.out.cache_count = K;
}

// ---------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------
thread_local std::string g_error;

// phase events of the last profiled step (host-side CUDA events; no device memory)
struct ProfileEvents {
    cudaEvent_t ev[8];
    bool created = false;
    bool recorded = false;
};
thread_local ProfileEvents g_prof;

static void prof_mark(bool on, int i, cudaStream_t st) {
    if (!on) return;
    if (!g_prof.created) {
        for (int k = 0; k < 8; ++k) cudaEventCreate(&g_prof.ev[k]);
        g_prof.created = true;
    }
    cudaEventRecord(g_prof.ev[i], st);
    if (i == 6) g_prof.recorded = true;
}

static int fail(int code, const std::string& msg) {
    g_error = msg;
    return code;
}

static inline int blocks_for(int64_t n, int block) { return (int)((n + block - 1) / block > 0 ? (n + block - 1) / block : 1); }

}  // namespace rb

using namespace rb;

extern "C" {

int rb_abi_version(void) { return RB_ABI_VERSION; }

const char* rb_last_error(void) { return rb::g_error.c_str(); }

int rb_topology_sizes(int32_t n_bodies, const int32_t* body_shape, int32_t n_shapes, const int32_t* v_off,
                      const int32_t* t_off, int64_t* out) {
    if (n_bodies < 0 || n_shapes <= 0 || !body_shape || !v_off || !t_off || !out)
        return fail(RB_ERR_ARG, "rb_topology_sizes: bad argument");
    int64_t nv = 0, nt = 0, nc = 0;
    for (int b = 0; b < n_bodies; ++b) {
        const int s = body_shape[b];
        if (s < 0 || s >= n_shapes) return fail(RB_ERR_ARG, "rb_topology_sizes: shape index out of range");
        nv += v_off[s + 1] - v_off[s];
        const int t = t_off[s + 1] - t_off[s];
        nt += t;
        nc += (t + 31) / 32;
    }
    out[0] = nv; out[1] = nt; out[2] = nc;
    return RB_OK;
}

int rb_workspace_bytes(const rb_bodies* bd, const rb_caps* caps, size_t* bytes) {
    if (!bd || !caps || !bytes) return fail(RB_ERR_ARG, "rb_workspace_bytes: null argument");
    if (bd->n_bodies < 0 || bd->n_body_vertices < 0 || bd->n_body_triangles < 0 || bd->n_clusters < 0 ||
        caps->pair_capacity < 0 || caps->item_capacity < 0 || caps->contact_capacity < 0)
        return fail(RB_ERR_ARG, "rb_workspace_bytes: negative size");
    if (bd->n_hinges < 0) return fail(RB_ERR_ARG, "rb_workspace_bytes: negative hinge count");
    *bytes = rb::layout(nullptr, nullptr, bd->n_bodies, bd->n_body_vertices, bd->n_body_triangles, bd->n_clusters,
                        caps->pair_capacity, caps->item_capacity, caps->contact_capacity, bd->n_scenes,
                        bd->n_hinges);
    return RB_OK;
}

}  // extern "C"

namespace {
// Largest dynamic shared memory of each solver kernel, granted once per device.  Done outside the launch
// sequence so that a step can be captured into a CUDA graph once the device has seen one uncaptured step.
std::mutex g_attr_mutex;
bool g_attr_done[64] = {false};
int ensure_kernel_attributes() {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return fail(RB_ERR_CUDA, "rb_step: no current device");
    std::lock_guard<std::mutex> lock(g_attr_mutex);
    if (g_attr_done[dev]) return RB_OK;
    const int warp_max = kSolveWarpsPerBlock * 6 * (int)sizeof(double) * (kWarpSceneMaxBodies + 1);
    const int block_max = 6 * (int)sizeof(double) * kSolveSmemBodies;
    e = cudaFuncSetAttribute(k_solve_warps, cudaFuncAttributeMaxDynamicSharedMemorySize, warp_max);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_solve_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, block_max);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_solve_fp32<WarpGroup, false, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kS32MidSlab);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_solve_fp32<BlockGroup, false, kFp32Block>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFp32LargeSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_solve_fp32<BlockGroup, true, kFp32L2Block>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFp32LargeSmem);
    if (e != cudaSuccess) return fail(RB_ERR_CUDA, std::string("rb_step: cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    g_attr_done[dev] = true;
    return RB_OK;
}

// Side streams of the FP32 size classes, per host thread and device: kSideSets sets, all made on the thread's
// first step on the device (an uncaptured call).  Each caller stream gets a set of its own (round robin over
// the sets, so steps on different streams run their solves concurrently); a step forks its set from its
// stream with an event and joins it back, which a stream capture records as parallel branches.
constexpr int kSideStreams = 4;
constexpr int kSideSets = 4;
struct SideStreams {
    cudaStream_t s[kSideStreams] = {};
    cudaEvent_t fork = nullptr, join[kSideStreams] = {};
};
struct SideSets {
    SideStreams set[kSideSets];
    const void* key[kSideSets] = {};
    int next = 0;
    bool made = false;
};
thread_local SideSets g_side[64];
int side_streams(cudaStream_t caller, SideStreams** out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fail(RB_ERR_CUDA, "rb_step: no current device");
    SideSets& ss = g_side[dev];
    if (!ss.made) {
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < kSideSets && e == cudaSuccess; ++k) {
            SideStreams& t = ss.set[k];
            e = cudaEventCreateWithFlags(&t.fork, cudaEventDisableTiming);
            for (int c = 0; c < kSideStreams && e == cudaSuccess; ++c) {
                e = cudaStreamCreateWithFlags(&t.s[c], cudaStreamNonBlocking);
                if (e == cudaSuccess) e = cudaEventCreateWithFlags(&t.join[c], cudaEventDisableTiming);
            }
        }
        if (e != cudaSuccess) return fail(RB_ERR_CUDA, std::string("rb_step: side streams: ") + cudaGetErrorString(e));
        ss.made = true;
    }
    int k = 0;
    while (k < kSideSets && ss.key[k] != (const void*)caller) ++k;
    if (k == kSideSets) {   // a caller stream not seen before takes the next set
        k = ss.next;
        ss.next = (ss.next + 1) % kSideSets;
        ss.key[k] = (const void*)caller;
    }
    *out = &ss.set[k];
    return RB_OK;
}
}  // namespace

extern "C" {

int rb_step(const rb_shapes* sh, const rb_bodies* bd, const rb_caps* caps, const rb_params* pr,
            const rb_outputs* out, void* workspace, size_t workspace_bytes, void* stream_ptr) {
    if (!sh || !bd || !caps || !pr || !out || !workspace) return fail(RB_ERR_ARG, "rb_step: null argument");
    if (bd->n_bodies <= 0 || bd->n_scenes <= 0) return fail(RB_ERR_ARG, "rb_step: empty scene batch");
    if (!bd->x || !bd->u || !out->contact_ids || !out->stats || !out->status)
        return fail(RB_ERR_ARG, "rb_step: null state or output buffer");
    if (pr->scheme < 0 || pr->scheme > RB_SCHEME_COLOURED_GS)
        return fail(RB_ERR_UNSUPPORTED, "rb_step: unknown solver scheme");
    if (pr->ordering != RB_ORDER_SERIAL && pr->ordering != RB_ORDER_COLOURED)
        return fail(RB_ERR_ARG, "rb_step: unknown contact ordering");
    if (bd->n_hinges < 0 || (bd->n_hinges > 0 && (!bd->scene_hinge_start || !bd->hinge_bodies || !bd->hinge_frames)))
        return fail(RB_ERR_ARG, "rb_step: hinge arrays missing");
    if (bd->n_hinges > 0 && (pr->scheme != RB_SCHEME_RIGID_GS || pr->termination != RB_TERMINATE_MERIT ||
                             pr->ordering != RB_ORDER_SERIAL || pr->precision != RB_PRECISION_FP64))
        return fail(RB_ERR_UNSUPPORTED, "rb_step: hinge joints are solved with the reference stepper's rule only "
                                        "(rigid Gauss-Seidel, merit termination, serial order, FP64)");
    // launch shapes
    const int small_slab = pr->fp32_small_slab > 0 ? pr->fp32_small_slab : kS32SmallSlab;
    const int mid_slab = pr->fp32_mid_slab > 0 ? pr->fp32_mid_slab : kS32MidSlab;
    const int mid_blocks = pr->mid_blocks > 0 ? pr->mid_blocks : 148 * 16;
    const int narrow_blocks = pr->narrow_blocks > 0 ? pr->narrow_blocks : 148 * 8;
    const int narrow_threads = pr->narrow_threads > 0 ? pr->narrow_threads : 256;
    if (small_slab % 16 || mid_slab % 16 || small_slab < 4096 || small_slab >= mid_slab || mid_slab > kS32MidSlab)
        return fail(RB_ERR_ARG, "rb_step: FP32 slabs must be multiples of 16 with 4096 <= small < mid <= 57344");
    if (mid_blocks > 65535 || narrow_blocks > 65535 ||
        (narrow_threads != 64 && narrow_threads != 128 && narrow_threads != 256))
        return fail(RB_ERR_ARG, "rb_step: launch shape out of range");
    if (pr->max_iterations < 0 || pr->max_iterations > caps->max_iterations)
        return fail(RB_ERR_ARG, "rb_step: max_iterations exceeds rb_caps.max_iterations");
    if (!(pr->dt > 0.0)) return fail(RB_ERR_ARG, "rb_step: dt must be positive");
    if (pr->precision != RB_PRECISION_FP64 && pr->termination != RB_TERMINATE_RESIDUAL_FIXED_R)
        return fail(RB_ERR_UNSUPPORTED, "rb_step: FP32 precision needs the fixed-r residual rule");
    if (pr->precision < RB_PRECISION_FP64 || pr->precision > RB_PRECISION_FP32)
        return fail(RB_ERR_ARG, "rb_step: unknown precision");
    if (sh->max_shape_triangles <= 0 || sh->max_shape_triangles > 32 * kMaxClustersPerShape)
        return fail(RB_ERR_ARG, "rb_step: max_shape_triangles must be in 1..16384");
    size_t need = 0;
    int rc = rb_workspace_bytes(bd, caps, &need);
    if (rc != RB_OK) return rc;
    if (workspace_bytes < need) return fail(RB_ERR_WORKSPACE, "rb_step: workspace too small");
    rc = ensure_kernel_attributes();
    if (rc != RB_OK) return rc;
    const int64_t n_body_vertices = bd->n_body_vertices, n_body_triangles = bd->n_body_triangles,
                  n_clusters = bd->n_clusters;
    cudaStream_t st = (cudaStream_t)stream_ptr;
    StepArgs a;
    a.sh = *sh; a.bd = *bd; a.caps = *caps; a.pr = *pr; a.out = *out;
    rb::layout(&a.ws, (char*)workspace, bd->n_bodies, n_body_vertices, n_body_triangles, n_clusters,
               caps->pair_capacity, caps->item_capacity, caps->contact_capacity, bd->n_scenes, bd->n_hinges);
    if (n_body_vertices <= 0 || n_body_triangles <= 0 || n_clusters <= 0)
        return fail(RB_ERR_ARG, "rb_step: bodies without geometry");
    const int N = bd->n_bodies;
    const int G = 148 * 8;
    const bool prof = pr->profiling != 0;
    prof_mark(prof, 0, st);
    k_bodies<<<blocks_for(std::max(N + 1, std::max(bd->n_scenes, 16)), 128), 128, 0, st>>>(a); note_launch();
    k_world_vertices<<<blocks_for(n_body_vertices, 256), 256, 0, st>>>(a, (int)n_body_vertices); note_launch();
    k_clusters<<<blocks_for(32 * n_clusters, kBlock), kBlock, 0, st>>>(a, (int)n_clusters); note_launch();
    k_roots<<<blocks_for(32 * (int64_t)N, kBlock), kBlock, 0, st>>>(a); note_launch();
    prof_mark(prof, 1, st);
    // broad phase
    k_pairs<false><<<blocks_for(32 * (int64_t)N, kBlock), kBlock, 0, st>>>(a); note_launch();
    scan_total(a.ws.pair_cnt, nullptr, N, a.ws.scan_tmp,
               ScanTotal{a.ws.counters, kNPairs, caps->pair_capacity, RB_STATUS_PAIR_OVERFLOW, out->status}, st);
    k_pairs<true><<<blocks_for(32 * (int64_t)N, kBlock), kBlock, 0, st>>>(a); note_launch();
    // mid phase
    {
        const int max_clusters = (sh->max_shape_triangles + 31) / 32;
        const size_t mid_smem = (size_t)kWarpsPerBlock * 3 * sizeof(uint32_t) * max_clusters;
        k_mid<<<mid_blocks, kBlock, mid_smem, st>>>(a, max_clusters); note_launch();
        // shapes of up to four clusters (128 triangles) make no wide pair
        if (max_clusters * max_clusters > kMidLight) {
            k_mid_wide<<<148 * 4, 32 * kMidWideWarps, mid_wide_bytes(max_clusters), st>>>(a, max_clusters); note_launch();
        }
    }
    prof_mark(prof, 2, st);
    // narrow phase
    // The search on the FP32 grid copy makes the FP64 search's decisions (near-ties go to FP64 lookups), so it finds the
    // same contacts; with FP64 lookups rid of their divisions it is the slower one, for its error bounds and second
    // lookups (512 piles with a grid per body 1284 against 710 us, 4096-body lattice 213 against 137).  It runs only
    // where it is checked against the FP64 search (profiling bit 2); every other step, profiled or not, runs the latter.
    if (pr->precision != RB_PRECISION_FP64 && sh->grid32 && (pr->profiling & 2)) {
        k_narrow<true><<<narrow_blocks, narrow_threads, 0, st>>>(a); note_launch();
    } else {
        k_narrow<false><<<narrow_blocks, narrow_threads, 0, st>>>(a); note_launch();
    }
    prof_mark(prof, 3, st);
    // reduction and compaction
    k_dedup<<<2 * G, kBlock, 0, st>>>(a); note_launch();
    scan_total(a.ws.pair_cont, a.ws.counters + kNPairs, caps->pair_capacity, a.ws.scan_tmp,
               ScanTotal{a.ws.counters, kNContacts, caps->contact_capacity, RB_STATUS_CONTACT_OVERFLOW, out->status}, st);
    k_emit<<<2 * G, kBlock, 0, st>>>(a); note_launch();
    prof_mark(prof, 4, st);
    // contact problem
    k_contacts<<<2 * G, 128, 0, st>>>(a); note_launch();   // a thread per contact row
    if (bd->n_hinges > 0) {   // the hinge problem of every scene that has hinges
        k_hinge_lists<<<blocks_for(bd->n_scenes, 64), 64, 0, st>>>(a); note_launch();
        k_hinges<<<blocks_for(bd->n_hinges, 128), 128, 0, st>>>(a); note_launch();
    }
    scan(a.ws.bc_ptr, nullptr, N, a.ws.scan_tmp, st);
    k_body_contacts_fill<<<G, 256, 0, st>>>(a); note_launch();
    k_body_contacts_sort<<<blocks_for(32 * (int64_t)N, 128), 128, 0, st>>>(a); note_launch();
    // solve, integrate, post-stabilise
    // small scenes: one warp each with its body accumulators in shared memory; large scenes: one block each
    // a warp per scene only pays off once the scenes alone fill the GPU (>= 32 per SM); otherwise blocks
    const int warp_bodies = bd->n_scenes < 148 * 32 ? 0
                          : (bd->max_scene_bodies < kWarpSceneMaxBodies ? bd->max_scene_bodies : kWarpSceneMaxBodies);
    const size_t warp_smem = (size_t)kSolveWarpsPerBlock * 6 * sizeof(double) * (warp_bodies > 0 ? warp_bodies + 1 : 1);
    const int wg = (bd->n_scenes + kSolveWarpsPerBlock - 1) / kSolveWarpsPerBlock;
    const int smem_bodies = std::min(std::max(bd->max_scene_bodies, 0), kSolveSmemBodies - 1) + 1;   // + 1: fixed bodies
    const size_t block_smem = (size_t)6 * sizeof(double) * smem_bodies;
    const int bg = bd->n_scenes < 148 * 16 ? bd->n_scenes : 148 * 16;
    // Threads of a scene's block: a scene that has an SM to itself takes as many warps as the registers allow (255 a
    // thread), so that wide levels and the rebuilds of w have them; more scenes than SMs share them, two blocks to an SM
    // or, with scenes so small or so many that two warps each do better, four, where the accumulators leave room for as
    // many.  A batch whose largest scene is more than four times the mean waits for that scene: it takes the most threads
    // too.  (Measured, ms a step with 128 and with 64 threads: 300 piles of 8-200 bodies 57 and 74, 600 101 and 128, 1500
    // 67.8 and 68.7, 4000 107 and 105; 600 piles of 30-60 bodies 66 and 54, 600 of 4-30 25.7 and 25.4, 1500 20.4 and 17.2.
    // 400 piles of up to 200 bodies and one of 5000: 454 with 64, 131 with 256; 300 of up to 40 and one of 1500: 729, 251.)
    const int share = (int)std::min<size_t>((bd->n_scenes + 147) / 148, (227 * 1024) / (block_smem + 2048));
    const bool uneven = (int64_t)bd->max_scene_bodies * bd->n_scenes > 4 * (int64_t)N;
    const bool small = bd->max_scene_bodies <= 64 || bd->n_scenes > 8 * 148;
    const int solve_threads = share <= 1 || uneven ? kSolveBlock : share == 2 || !small ? kSolveBlock / 2 : kSolveBlock / 4;
    if (pr->precision != RB_PRECISION_FP64) {
        k_fp32_classes<<<1, 1024, 0, st>>>(a, small_slab, mid_slab); note_launch();
        // FP32 phase, four size classes side by side: warp teams with small slabs (28 KB unless tuned), warp
        // teams with mid slabs (56 KB), block teams with 224 KB (1 per SM), and 512-thread block teams for the
        // scenes beyond that, whose contact rows stay in L2
        SideStreams* ss = nullptr;
        rc = side_streams(st, &ss);
        if (rc != RB_OK) return rc;
        cudaEventRecord(ss->fork, st);
        for (int c = 0; c < kSideStreams; ++c) cudaStreamWaitEvent(ss->s[c], ss->fork, 0);
        k_solve_fp32<BlockGroup, true, kFp32L2Block><<<148, kFp32L2Block, (size_t)kFp32LargeSmem, ss->s[3]>>>(
            a, kQueueFp32 + 3, kFp32LargeSmem, kFp32LargeSmem); note_launch();
        k_solve_fp32<BlockGroup, false, kFp32Block><<<148, kFp32Block, (size_t)kFp32LargeSmem, ss->s[2]>>>(
            a, kQueueFp32 + 2, mid_slab, kFp32LargeSmem); note_launch();
        // warp teams as one-warp blocks: a team's slab is released as soon as the team finds its queue empty
        // (in blocks of four teams the slowest held all four slabs), so the small class fills the room the mid
        // class leaves; as many blocks per SM as the shared memory (227 KB) allows, up to 32
        const int small_per_sm = std::min(32, (227 * 1024) / small_slab);
        const int mid_per_sm = std::max(1, std::min(32, (227 * 1024) / mid_slab));
        k_solve_fp32<WarpGroup, false, 32><<<148 * mid_per_sm, 32, (size_t)mid_slab, ss->s[1]>>>(
            a, kQueueFp32 + 1, small_slab, mid_slab); note_launch();
        k_solve_fp32<WarpGroup, false, 32><<<148 * small_per_sm, 32, (size_t)small_slab, ss->s[0]>>>(
            a, kQueueFp32, 0, small_slab); note_launch();
        for (int c = 0; c < kSideStreams; ++c) {
            cudaEventRecord(ss->join[c], ss->s[c]);
            cudaStreamWaitEvent(st, ss->join[c], 0);
        }
    }
    if (warp_bodies > 0) { k_solve_warps<<<wg, 32 * kSolveWarpsPerBlock, warp_smem, st>>>(a, 0, warp_bodies); note_launch(); }
    k_solve_blocks<<<bg, solve_threads, block_smem, st>>>(a, 0, warp_bodies, smem_bodies); note_launch();
    prof_mark(prof, 5, st);
    k_integrate<<<blocks_for(32 * ((N + 4) / (int64_t)5), 128), 128, 0, st>>>(a); note_launch();
    if (pr->use_post_stabilization) {
        k_post_setup<<<G, 128, 0, st>>>(a); note_launch();
        if (warp_bodies > 0) { k_solve_warps<<<wg, 32 * kSolveWarpsPerBlock, warp_smem, st>>>(a, 1, warp_bodies); note_launch(); }
        k_solve_blocks<<<bg, solve_threads, block_smem, st>>>(a, 1, warp_bodies, smem_bodies); note_launch();
        k_post_apply<<<blocks_for(32 * ((N + 4) / (int64_t)5), 128), 128, 0, st>>>(a); note_launch();
    }
    if (prof) { k_body_energy<<<blocks_for(N, 128), 128, 0, st>>>(a); note_launch(); }
    const int summary_blocks = blocks_for(32 * (int64_t)bd->n_scenes, 128);
    k_outputs<<<summary_blocks + G, 128, 0, st>>>(a, summary_blocks); note_launch();
    prof_mark(prof, 6, st);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(RB_ERR_CUDA, std::string("rb_step: ") + cudaGetErrorString(e));
    return RB_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------------
// rb_step_noalloc: the same step with its temporaries in a fixed scratch array of this library
// ---------------------------------------------------------------------------------------------------------
namespace {

// Scratch of rb_step_noalloc.  In host code this name only stands for the array: the kernels receive the
// device address looked up with cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_noalloc_scratch[RB_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_ptr[kMaxDevices] = {nullptr};

// device address of the scratch array on the current device, looked up once per device
int noalloc_scratch(void** ptr) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(RB_ERR_CUDA, std::string("rb_step_noalloc: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return fail(RB_ERR_UNSUPPORTED, "rb_step_noalloc: device index out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return fail(RB_ERR_CUDA, std::string("rb_step_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
        g_noalloc_ptr[dev] = p;
    }
    *ptr = g_noalloc_ptr[dev];
    return RB_OK;
}

}  // namespace

extern "C" {

int rb_step_noalloc(const rb_shapes* sh, const rb_bodies* bd, const rb_caps* caps, const rb_params* pr,
                    const rb_outputs* out, void* stream) {
    if (!sh || !bd || !caps || !pr || !out) return fail(RB_ERR_ARG, "rb_step_noalloc: null argument");
    size_t need = 0;
    int rc = rb_workspace_bytes(bd, caps, &need);
    if (rc != RB_OK) return rc;
    if (need > (size_t)RB_NOALLOC_SCRATCH_BYTES)
        return fail(RB_ERR_WORKSPACE, "rb_step_noalloc: this batch needs " + std::to_string(need) +
                                          " bytes of scratch, more than the " +
                                          std::to_string((size_t)RB_NOALLOC_SCRATCH_BYTES) +
                                          " bytes available; use rb_step with a workspace");
    void* scratch = nullptr;
    rc = noalloc_scratch(&scratch);
    if (rc != RB_OK) return rc;
    // rb_step clears the counters and per-body tallies it needs at the start of every step, so the
    // previous call's contents of the shared array do no harm
    return rb_step(sh, bd, caps, pr, out, scratch, (size_t)RB_NOALLOC_SCRATCH_BYTES, stream);
}

int64_t rb_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

int rb_profile_times(float* out, int32_t n) {
    if (!out || n < 7) return fail(RB_ERR_ARG, "rb_profile_times: need room for 7 values");
    if (!g_prof.recorded) return fail(RB_ERR_ARG, "rb_profile_times: no profiled step on this thread");
    cudaError_t e = cudaEventSynchronize(g_prof.ev[6]);
    if (e != cudaSuccess) return fail(RB_ERR_CUDA, std::string("rb_profile_times: ") + cudaGetErrorString(e));
    for (int i = 0; i < 6; ++i) cudaEventElapsedTime(out + i, g_prof.ev[i], g_prof.ev[i + 1]);
    cudaEventElapsedTime(out + 6, g_prof.ev[0], g_prof.ev[6]);
    return RB_OK;
}

}  // extern "C"
