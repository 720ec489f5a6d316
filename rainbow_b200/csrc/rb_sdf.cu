// rb_sdf.cu -- signed distance grid of a closed triangle mesh (shape set-up).
//
// Replaces the igl.signed_distance call of grid3.py:338 (create_signed_distance).  For every grid node:
//   distance = min over triangles of |p - closest point on the triangle| (Voronoi-region case analysis of
//              Ericson, Real-Time Collision Detection, 2005, section 5.1.5);
//   sign     = negative when the generalized winding number |w| > 1/2, w = sum of the triangles' signed
//              solid angles / 4 pi (Van Oosterom & Strackee, IEEE TBME 1983).
// One thread per node; triangles are streamed through shared memory in tiles.
#include <cuda_runtime.h>

#include <string>

#include "rainbow_b200.h"
#include "rb_device.cuh"
#include "rb_internal.h"

namespace {

using rb::d3;

__device__ __forceinline__ double dot(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ d3 scale(d3 a, double s) { return d3{a.x * s, a.y * s, a.z * s}; }

__device__ d3 closest_point(d3 p, d3 a, d3 b, d3 c) {
    const d3 ab = rb::sub(b, a), ac = rb::sub(c, a), ap = rb::sub(p, a);
    const double d1 = dot(ab, ap), d2 = dot(ac, ap);
    if (d1 <= 0.0 && d2 <= 0.0) return a;
    const d3 bp = rb::sub(p, b);
    const double d3v = dot(ab, bp), d4 = dot(ac, bp);
    if (d3v >= 0.0 && d4 <= d3v) return b;
    const double vc = d1 * d4 - d3v * d2;
    if (vc <= 0.0 && d1 >= 0.0 && d3v <= 0.0) {
        const double v = d1 / (d1 - d3v);
        return rb::add(a, scale(ab, v));
    }
    const d3 cp = rb::sub(p, c);
    const double d5 = dot(ab, cp), d6 = dot(ac, cp);
    if (d6 >= 0.0 && d5 <= d6) return c;
    const double vb = d5 * d2 - d1 * d6;
    if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) {
        const double w = d2 / (d2 - d6);
        return rb::add(a, scale(ac, w));
    }
    const double va = d3v * d6 - d5 * d4;
    if (va <= 0.0 && (d4 - d3v) >= 0.0 && (d5 - d6) >= 0.0) {
        const double w = (d4 - d3v) / ((d4 - d3v) + (d5 - d6));
        return rb::add(b, scale(rb::sub(c, b), w));
    }
    const double denom = 1.0 / (va + vb + vc);
    const double v = vb * denom, w = vc * denom;
    return rb::add(a, rb::add(scale(ab, v), scale(ac, w)));
}

constexpr int kTile = 128;
constexpr int kSdfBlock = 128;

// signed solid angle of the triangle at the origin as the angle of the complex number (den, num), times two
__device__ __forceinline__ void solid_angle(d3 A, d3 B, d3 C, double la, double lb, double lc, double& num, double& den) {
    num = dot(A, rb::cross_np(B, C));
    den = la * lb * lc + dot(A, B) * lc + dot(B, C) * la + dot(C, A) * lb;
}

// the same from the squares of the lengths, with fused products
__device__ __forceinline__ double dot_fused(d3 a, d3 b) { return fma(a.z, b.z, fma(a.y, b.y, a.x * b.x)); }
__device__ __forceinline__ void solid_angle_fused(d3 A, d3 B, d3 C, double a2, double b2, double c2, double& size,
                                                  double& num, double& den) {
    const double la = rb::sqrt_chain(a2), lb = rb::sqrt_chain(b2), lc = rb::sqrt_chain(c2);
    const d3 n = d3{fma(B.y, C.z, -(B.z * C.y)), fma(B.z, C.x, -(B.x * C.z)), fma(B.x, C.y, -(B.y * C.x))};
    num = dot_fused(A, n);
    size = la * lb * lc;
    den = fma(dot_fused(C, A), lb, fma(dot_fused(B, C), la, fma(dot_fused(A, B), lc, size)));
}

// one tile of triangles in shared memory: corners, and a sphere around each (centroid, radius)
struct SdfTile {
    double corner[kTile][9];
    double ball[kTile][4];
};
__device__ __forceinline__ void sdf_tile(SdfTile& tile, const double* __restrict__ V, const int32_t* __restrict__ T,
                                         int n_tri, int t0, bool balls) {
    __syncthreads();
    for (int e = threadIdx.x; e < kTile * 9; e += blockDim.x) {
        const int t = t0 + e / 9, c = (e % 9) / 3, axis = e % 3;
        tile.corner[e / 9][e % 9] = t < n_tri ? V[3 * T[3 * t + c] + axis] : 0.0;
    }
    __syncthreads();
    if (!balls) return;
    for (int t = threadIdx.x; t < kTile; t += blockDim.x) {
        const double* q = tile.corner[t];
        const d3 a = rb::ld3(q), b = rb::ld3(q + 3), c = rb::ld3(q + 6);
        const d3 g = scale(rb::add(rb::add(a, b), c), 1.0 / 3.0);
        const d3 u = rb::sub(a, g), v = rb::sub(b, g), w = rb::sub(c, g);
        rb::st3(tile.ball[t], g);
        tile.ball[t][3] = sqrt(fmax(dot(u, u), fmax(dot(v, v), dot(w, w))));
    }
    __syncthreads();
}

// distance and sign of node `node` of a grid (meta: min[3], max[3], spacing[3], I, J, K) around the mesh
// (V, T with n_tri triangles); every thread of the block calls it (the triangle tiles go through shared memory).
//
// Bound by FP64 arithmetic over (node, triangle) pairs.  The sign needs only whether |w| > 1/2, so the solid angles are
// not summed as arcs: their complex numbers are multiplied, the turns across the negative real axis counted, and one
// arc taken at the end (exponents are taken out on the way).  A node so near an edge of a triangle that its number's
// modulus is below 1e-4 of its scale, or with a sum within 1e-3 of the threshold, takes the plain sum (a factor's angle
// is otherwise right to 1e-11, w with any number of triangles that memory holds to 1e-3).  The distance's minimum is
// taken over squares, and a triangle is passed over when the sphere around it is farther than the nearest vertex or
// point so far.  Both give the values of the plain form: an arc, four roots and the closest point for every triangle
// took 11.8 ms a pass for 96 grids of 32^3 around boxes and 448-triangle spheres, this one 6.1 (5.8 with lengths to
// 2^-39 only, which bounded w to 3e-4 for 16384 triangles and not at all for more).
__device__ __forceinline__ void sdf_node(const double* __restrict__ V, const int32_t* __restrict__ T, int n_tri,
                                         const double* __restrict__ meta, int64_t node, double* __restrict__ values) {
    __shared__ SdfTile tile;
    const int I = (int)meta[9], J = (int)meta[10], K = (int)meta[11];
    const int64_t n_nodes = (int64_t)I * J * K;
    const bool mine = node < n_nodes;
    d3 p = d3{meta[0], meta[1], meta[2]};   // (a thread past the last node goes along with the first)
    if (mine) {
        const int i = (int)(node % I), j = (int)((node / I) % J), k = (int)(node / ((int64_t)I * J));
        // grid3.py:88 get_node_coord: min + spacing * (i, j, k)
        p = d3{meta[0] + meta[6] * (double)i, meta[1] + meta[7] * (double)j, meta[2] + meta[8] * (double)k};
    }
    // winding number, and the nearest vertex
    double re = 1.0, im = 0.0, near2 = INFINITY;
    int turns = 0;
    bool unsure = false;
    for (int t0 = 0; t0 < n_tri; t0 += kTile) {
        sdf_tile(tile, V, T, n_tri, t0, false);
        const int nt = min(kTile, n_tri - t0);
        for (int t = 0; t < nt; ++t) {
            const double* q = tile.corner[t];
            const d3 A = rb::sub(rb::ld3(q), p), B = rb::sub(rb::ld3(q + 3), p), C = rb::sub(rb::ld3(q + 6), p);
            const double a2 = dot_fused(A, A), b2 = dot_fused(B, B), c2 = dot_fused(C, C);
            near2 = fmin(near2, fmin(a2, fmin(b2, c2)));
            double size, num, den;
            solid_angle_fused(A, B, C, a2, b2, c2, size, num, den);
            // (so put that a NaN is unsure; a zero imaginary part left of zero has no side)
            unsure |= !(fabs(num) + fabs(den) >= 1e-4 * size) || (num == 0.0 && den < 0.0);
            const double r = fma(re, den, -(im * num)), m = fma(re, num, im * den);
            // both factors' angles on one side and the product on the other: past the negative real axis
            if (im >= 0.0 && num >= 0.0 && m < 0.0) ++turns;
            else if (im < 0.0 && num < 0.0 && m >= 0.0) --turns;
            const int e = max(__double2hiint(r) & 0x7ff00000, __double2hiint(m) & 0x7ff00000);
            const double s = __hiloint2double(0x7fe00000 - e, 0);   // 2^-exponent of the larger part
            re = r * s; im = m * s;
        }
    }
    double wind = 2.0 * (atan2(im, re) + 2.0 * M_PI * (double)turns);
    if (__syncthreads_or(unsure || !(fabs(fabs(wind) / (4.0 * M_PI) - 0.5) > 1e-3))) {   // some node's plain sum
        const bool again = unsure || !(fabs(fabs(wind) / (4.0 * M_PI) - 0.5) > 1e-3);
        double sum = 0.0;
        for (int t0 = 0; t0 < n_tri; t0 += kTile) {
            sdf_tile(tile, V, T, n_tri, t0, false);
            const int nt = min(kTile, n_tri - t0);
            if (again)
                for (int t = 0; t < nt; ++t) {
                    const double* q = tile.corner[t];
                    const d3 A = rb::sub(rb::ld3(q), p), B = rb::sub(rb::ld3(q + 3), p), C = rb::sub(rb::ld3(q + 6), p);
                    double num, den;
                    solid_angle(A, B, C, sqrt(dot(A, A)), sqrt(dot(B, B)), sqrt(dot(C, C)), num, den);
                    sum += 2.0 * atan2(num, den);
                }
        }
        if (again) wind = sum;
    }
    // distance: the square's minimum over the triangles whose sphere comes as near as the best so far
    double best2 = INFINITY, reach = sqrt(near2);
    for (int t0 = 0; t0 < n_tri; t0 += kTile) {
        sdf_tile(tile, V, T, n_tri, t0, true);
        const int nt = min(kTile, n_tri - t0);
        for (int t = 0; t < nt; ++t) {
            const double* s = tile.ball[t];
            const d3 u = rb::sub(p, rb::ld3(s));
            const double far = s[3] + reach;
            if (dot_fused(u, u) > 1.000001 * (far * far)) continue;
            const double* q = tile.corner[t];
            const d3 dq = rb::sub(p, closest_point(p, rb::ld3(q), rb::ld3(q + 3), rb::ld3(q + 6)));
            const double d2 = dot(dq, dq);
            if (d2 < best2) { best2 = d2; reach = fmin(reach, sqrt(d2)); }
        }
    }
    const double best = sqrt(best2);
    if (mine) values[node] = (fabs(wind) / (4.0 * M_PI) > 0.5) ? -best : best;
}

// The node a thread takes of its block's 128: 4 runs of 8 a warp, 32 apart, so that with about 32 nodes to a grid's
// row a warp is a patch of 8 x 4 and its lanes pass over much the same triangles
__device__ __forceinline__ int sdf_place() {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    return 32 * (lane >> 3) + 8 * warp + (lane & 7);
}

__global__ void __launch_bounds__(kSdfBlock) k_sdf(const double* __restrict__ V, const int32_t* __restrict__ T,
                                                   int n_tri, const double* __restrict__ meta,
                                                   double* __restrict__ values) {
    sdf_node(V, T, n_tri, meta, (int64_t)blockIdx.x * kSdfBlock + sdf_place(), values);
}

// many grids in one launch: block b belongs to the shape s with block_off[s] <= b < block_off[s + 1]
__global__ void __launch_bounds__(kSdfBlock) k_sdf_many(int n_shapes, const double* __restrict__ V,
                                                        const int32_t* __restrict__ v_off,
                                                        const int32_t* __restrict__ T,
                                                        const int32_t* __restrict__ t_off,
                                                        const double* __restrict__ meta,
                                                        const int64_t* __restrict__ g_off,
                                                        const int64_t* __restrict__ block_off,
                                                        double* __restrict__ values) {
    const int64_t b = blockIdx.x;
    int lo = 0, hi = n_shapes;   // the last s with block_off[s] <= b
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (block_off[mid] <= b) lo = mid; else hi = mid;
    }
    const int s = lo;
    const int64_t node = (b - block_off[s]) * kSdfBlock + sdf_place();
    sdf_node(V + 3 * (size_t)v_off[s], T + 3 * (size_t)t_off[s], t_off[s + 1] - t_off[s], meta + 12 * (size_t)s,
             node, values + g_off[s]);
}

}  // namespace

extern "C" int rb_signed_distance_grid(const double* V, int32_t n_vertices, const int32_t* T, int32_t n_triangles,
                                       const double* grid_meta_dev, double* values, void* stream) {
    if (!V || !T || !grid_meta_dev || !values || n_vertices <= 0 || n_triangles <= 0) {
        rb::g_error = "rb_signed_distance_grid: bad argument";
        return RB_ERR_ARG;
    }
    // the node count is read on the device from grid_meta; the launch covers the largest grid allowed here
    double meta[12];
    cudaError_t e = cudaMemcpyAsync(meta, grid_meta_dev, sizeof(meta), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) {
        rb::g_error = std::string("rb_signed_distance_grid: ") + cudaGetErrorString(e);
        return RB_ERR_CUDA;
    }
    const int64_t n_nodes = (int64_t)meta[9] * (int64_t)meta[10] * (int64_t)meta[11];
    if (meta[9] < 2 || meta[10] < 2 || meta[11] < 2 || n_nodes > (int64_t)1 << 30) {
        rb::g_error = "rb_signed_distance_grid: grid size out of range";
        return RB_ERR_ARG;
    }
    const int block = kSdfBlock;
    k_sdf<<<(unsigned)((n_nodes + block - 1) / block), block, 0, (cudaStream_t)stream>>>(V, T, n_triangles,
                                                                                      grid_meta_dev, values);
    rb::note_launch();
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        rb::g_error = std::string("rb_signed_distance_grid: ") + cudaGetErrorString(e);
        return RB_ERR_CUDA;
    }
    return RB_OK;
}

extern "C" int rb_signed_distance_grids(int32_t n_shapes, const double* V, const int32_t* v_off, const int32_t* T,
                                        const int32_t* t_off, const double* grid_meta, const int64_t* g_off,
                                        const int64_t* block_off, int64_t total_blocks, double* values,
                                        void* stream) {
    if (n_shapes <= 0 || !V || !v_off || !T || !t_off || !grid_meta || !g_off || !block_off || !values ||
        total_blocks <= 0 || total_blocks > INT32_MAX) {
        rb::g_error = "rb_signed_distance_grids: bad argument";
        return RB_ERR_ARG;
    }
    k_sdf_many<<<(unsigned)total_blocks, kSdfBlock, 0, (cudaStream_t)stream>>>(n_shapes, V, v_off, T, t_off,
                                                                             grid_meta, g_off, block_off, values);
    rb::note_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        rb::g_error = std::string("rb_signed_distance_grids: ") + cudaGetErrorString(e);
        return RB_ERR_CUDA;
    }
    return RB_OK;
}
