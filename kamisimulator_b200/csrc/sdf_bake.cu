// sdf_bake.cu -- the body SDF grid baked from a closed triangle mesh on the GPU.
//
// KamiSimulator bakes the head's SDF on the CPU: Discregrid's TriangleMeshDistance resampled by a
// CubicLagrangeDiscreteGrid (utilities/Geometry.cpp:5-35), then sampled at the grid nodes by
// PNMesh::StoreSDFQueries (PNMesh.cpp:109-173).  Here every node gets the exact signed distance
// to the mesh, the function that grid approximates:
//   * nearest point: the triangle with the smallest squared distance, the first of them on a tie, among
//     all triangles; clusters of neighbouring triangles that cannot hold it are skipped (sdf_bake_kernel).
//     Closest point on a triangle and its Voronoi feature (vertex, edge or face) after Ericson,
//     Real-Time Collision Detection (2005), 5.1.5;
//   * sign: the angle-weighted pseudonormal of that feature (Baerentzen and Aanaes, "Signed
//     distance computation using the angle weighted pseudonormal", IEEE TVCG 11(3), 2005), the
//     sign rule of TriangleMeshDistance::signed_distance;
//   * gradient: inside (distance < 0) the unit gradient of the distance, (nearest - x) / |d|;
//     elsewhere the unit direction from the grid centre, as StoreSDFQueries sets it (zero at a
//     node exactly at the centre, where the reference divides 0 by 0).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "kami_vbd.h"
#include "vbd_common.cuh"
#include "vbd_host.h"

namespace kami {
namespace {

constexpr int BAKE_THREADS = 256;
constexpr int BAKE_WARPS = BAKE_THREADS / 32;
constexpr int BAKE_CLUSTER = 16;  // triangles per cluster
constexpr int BX = 4, BY = 4, BZ = 2;  // nodes of a brick: one warp's lanes

// Neighbouring triangles, in the order of their centroids along a Morton curve.
struct BakeCluster {
    float lo[3], hi[3];  // box of the vertices
    float e1;            // relative and absolute error of a computed closest point, both per squared
    float e2;            // distance (below)
};

// Closest point on triangle (a, b, c) to p and its feature: 0, 1, 2 = vertex a, b, c; 3, 4, 5 =
// edge ab, bc, ca; 6 = face.  Returns the squared distance.
__device__ __forceinline__ float closest_on_triangle(float3 p, float3 a, float3 b, float3 c, float3& cp, int& f) {
    const float3 ab = b - a, ac = c - a, ap = p - a;
    const float d1 = dot3(ab, ap), d2 = dot3(ac, ap);
    if (d1 <= 0.f && d2 <= 0.f) {
        cp = a;
        f = 0;
    } else {
        const float3 bp = p - b;
        const float d3 = dot3(ab, bp), d4 = dot3(ac, bp);
        if (d3 >= 0.f && d4 <= d3) {
            cp = b;
            f = 1;
        } else {
            const float vc = d1 * d4 - d3 * d2;
            if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
                cp = a + (d1 / (d1 - d3)) * ab;
                f = 3;
            } else {
                const float3 cpp = p - c;
                const float d5 = dot3(ab, cpp), d6 = dot3(ac, cpp);
                if (d6 >= 0.f && d5 <= d6) {
                    cp = c;
                    f = 2;
                } else {
                    const float vb = d5 * d2 - d1 * d6;
                    if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
                        cp = a + (d2 / (d2 - d6)) * ac;
                        f = 5;
                    } else {
                        const float va = d3 * d6 - d5 * d4;
                        if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
                            cp = b + ((d4 - d3) / ((d4 - d3) + (d5 - d6))) * (c - b);
                            f = 4;
                        } else {
                            const float den = 1.f / (va + vb + vc);
                            cp = a + (vb * den) * ab + (vc * den) * ac;
                            f = 6;
                        }
                    }
                }
            }
        }
    }
    const float3 d = p - cp;
    return dot3(d, d);
}

// A node's signed distance and gradient from its nearest triangle bt, feature bf and point bcp.
__device__ __forceinline__ void bake_node(float3 x, float3 centre, float best, int bt, int bf, float3 bcp, int64_t node,
                                          const int32_t* __restrict__ tris, const float4* __restrict__ face_n,
                                          const float4* __restrict__ edge_n, const float4* __restrict__ vert_n,
                                          float* __restrict__ phi, float* __restrict__ grad) {
    if (bt < 0) {  // no finite distance (the host rejects non-finite vertices, so this is a guard)
        phi[node] = NAN;
        grad[3 * node] = grad[3 * node + 1] = grad[3 * node + 2] = 0.f;
        return;
    }
    const float dist = sqrtf(best);
    float4 pn;
    if (bf < 3)
        pn = vert_n[tris[3 * bt + bf]];
    else if (bf < 6)
        pn = edge_n[3 * bt + (bf - 3)];
    else
        pn = face_n[bt];
    const float3 u = x - bcp;
    const float s = (u.x * pn.x + u.y * pn.y + u.z * pn.z) >= 0.f ? 1.f : -1.f;
    const float d = s * dist;
    phi[node] = d;
    float3 g;
    if (d < 0.f) {
        g = (bcp - x) * (1.f / dist);
    } else {
        const float3 r = x - centre;
        const float l = sqrtf(dot3(r, r));
        g = l > 0.f ? r * (1.f / l) : f3(0.f, 0.f, 0.f);
    }
    grad[3 * node] = g.x;
    grad[3 * node + 1] = g.y;
    grad[3 * node + 2] = g.z;
}

// Whether a cluster holds no triangle whose computed squared distance from a point of the box [p0, p1] is
// best or less.  closest_on_triangle's point lies on the triangle up to the rounding of its coordinates
// (`slack`), except in the face case, whose barycentric weights come from differences of products: with u
// the unit roundoff, L the longest edge, A the area and D the distance of the farthest vertex, each is off by
// at most E = 72 u L^2 D^2 / (4 A^2) of their sum, so the point by 8 E L while E <= 1/2.  A cluster with a
// larger E (slivers, or small triangles very far away) is never skipped: its computed distances may be
// anything, and the nearest computed one is what the bake returns.  e1, e2: the largest E / D^2 and
// 8 E L / D^2 of the cluster.
__device__ __forceinline__ bool bake_skips(const BakeCluster& c, float3 p0, float3 p1, float slack, float best) {
    const float ax = fmaxf(fmaxf(c.lo[0] - p1.x, p0.x - c.hi[0]), 0.f), bx = fmaxf(c.hi[0] - p0.x, p1.x - c.lo[0]);
    const float ay = fmaxf(fmaxf(c.lo[1] - p1.y, p0.y - c.hi[1]), 0.f), by = fmaxf(c.hi[1] - p0.y, p1.y - c.lo[1]);
    const float az = fmaxf(fmaxf(c.lo[2] - p1.z, p0.z - c.hi[2]), 0.f), bz = fmaxf(c.hi[2] - p0.z, p1.z - c.lo[2]);
    const float far2 = bx * bx + by * by + bz * bz;
    const float lb = sqrtf(ax * ax + ay * ay + az * az) * 0.9999f - c.e2 * far2 - slack;
    return c.e1 * far2 <= 0.5f && lb > 0.f && lb * lb > best;  // false when anything is NaN
}

// One CTA per brick of 4 x 4 x 2 nodes: a warp's lanes are the nodes, the 8 warps share the clusters.  The
// cluster nearest to the brick gives every node a distance; the clusters that may hold a smaller one for some
// node are listed and tested, each lane's own distance sparing whole warps some of the list.  Bound by the
// closest-point arithmetic, about 100 instructions a node and triangle, so the test count decides: 20,480
// triangles and 64^3 nodes took 15.7 ms when every node tested every triangle, and 1.87 with this.
// Clusters of 16: with larger ones more triangles are tested for nothing, with smaller ones more boxes.
__global__ void __launch_bounds__(BAKE_THREADS) sdf_bake_kernel(const float* __restrict__ tv, int nt,
                                                                const int32_t* __restrict__ order,
                                                                const BakeCluster* __restrict__ clusters, int nc,
                                                                const int32_t* __restrict__ tris,
                                                                const float4* __restrict__ face_n,
                                                                const float4* __restrict__ edge_n,
                                                                const float4* __restrict__ vert_n, int nx, int ny, int nz,
                                                                float3 lo, float3 ds, float3 centre, float slack,
                                                                float* __restrict__ phi, float* __restrict__ grad) {
    __shared__ float s_best[BAKE_WARPS][32];
    __shared__ float3 s_cp[BAKE_WARPS][32];
    __shared__ int s_bt[BAKE_WARPS][32], s_bf[BAKE_WARPS][32];
    __shared__ float s_near[BAKE_WARPS];
    __shared__ int s_arg[BAKE_WARPS], s_list[BAKE_THREADS], s_count;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t gx = (nx + BX - 1) / BX, gy = (ny + BY - 1) / BY, gz = (nz + BZ - 1) / BZ;
    for (int64_t brick = blockIdx.x; brick < gx * gy * gz; brick += gridDim.x) {
        const int64_t i0 = brick % gx * BX, j0 = brick / gx % gy * BY, k0 = brick / (gx * gy) * BZ;
        const int64_t ni = i0 + lane % BX, nj = j0 + lane / BX % BY, nk = k0 + lane / (BX * BY);
        const bool active = ni < nx && nj < ny && nk < nz;
        // lanes beyond the grid repeat its last nodes
        const int64_t i = min(ni, (int64_t)nx - 1), j = min(nj, (int64_t)ny - 1), k = min(nk, (int64_t)nz - 1);
        const int64_t node = i + nx * (j + ny * k);
        const float3 x = f3(lo.x + ds.x * (float)i, lo.y + ds.y * (float)j, lo.z + ds.z * (float)k);
        const float3 p0 = f3(lo.x + ds.x * (float)i0, lo.y + ds.y * (float)j0, lo.z + ds.z * (float)k0);
        const float3 p1 = f3(lo.x + ds.x * (float)min(i0 + BX - 1, (int64_t)nx - 1),
                             lo.y + ds.y * (float)min(j0 + BY - 1, (int64_t)ny - 1),
                             lo.z + ds.z * (float)min(k0 + BZ - 1, (int64_t)nz - 1));
        float best = INFINITY;
        int bt = -1, bf = 0;
        float3 bcp = x;
        const auto test = [&](int q) {  // the q-th triangle in the clusters' order
            const float* T = tv + 9 * (int64_t)q;
            const int t = order[q];
            float3 cp;
            int f;
            const float d2 = closest_on_triangle(x, f3(T[0], T[1], T[2]), f3(T[3], T[4], T[5]), f3(T[6], T[7], T[8]), cp, f);
            if (d2 < best || (d2 == best && t < bt)) {
                best = d2;
                bt = t;
                bf = f;
                bcp = cp;
            }
        };
        // the cluster whose centre is nearest to the brick's
        float near = INFINITY;
        int arg = 0;
        for (int c = threadIdx.x; c < nc; c += BAKE_THREADS) {
            const BakeCluster& C = clusters[c];
            const float3 d = f3((C.lo[0] + C.hi[0]) - (p0.x + p1.x), (C.lo[1] + C.hi[1]) - (p0.y + p1.y),
                                (C.lo[2] + C.hi[2]) - (p0.z + p1.z));
            const float d2 = dot3(d, d);
            if (d2 < near) {
                near = d2;
                arg = c;
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float n2 = __shfl_xor_sync(~0u, near, o);
            const int a2 = __shfl_xor_sync(~0u, arg, o);
            if (n2 < near || (n2 == near && a2 < arg)) {
                near = n2;
                arg = a2;
            }
        }
        if (lane == 0) {
            s_near[warp] = near;
            s_arg[warp] = arg;
        }
        __syncthreads();
        near = s_near[0];
        arg = s_arg[0];
        for (int w = 1; w < BAKE_WARPS; w++)
            if (s_near[w] < near) {
                near = s_near[w];
                arg = s_arg[w];
            }
        const int first_end = min((arg + 1) * BAKE_CLUSTER, nt);
        for (int q = arg * BAKE_CLUSTER + warp; q < first_end; q += BAKE_WARPS) test(q);
        s_best[warp][lane] = best;
        __syncthreads();
        float mine = s_best[0][lane];  // this node's distance so far, a bound for every warp
        for (int w = 1; w < BAKE_WARPS; w++) mine = fminf(mine, s_best[w][lane]);
        float all = mine;  // and the brick's
#pragma unroll
        for (int o = 16; o; o >>= 1) all = fmaxf(all, __shfl_xor_sync(~0u, all, o));
        for (int base = 0; base < nc; base += BAKE_THREADS) {
            if (threadIdx.x == 0) s_count = 0;
            __syncthreads();
            const int c = base + threadIdx.x;
            const bool keep = c < nc && c != arg && !bake_skips(clusters[c], p0, p1, slack, all);
            const unsigned m = __ballot_sync(~0u, keep);
            int at = 0;
            if (lane == 0 && m) at = atomicAdd(&s_count, __popc(m));
            at = __shfl_sync(~0u, at, 0) + __popc(m & ((1u << lane) - 1));
            if (keep) s_list[at] = c;
            __syncthreads();
            for (int e = warp; e < s_count; e += BAKE_WARPS) {
                const int l = s_list[e];
                if (__all_sync(~0u, bake_skips(clusters[l], x, x, slack, fminf(best, mine)))) continue;
                const int end = min((l + 1) * BAKE_CLUSTER, nt);
                for (int q = l * BAKE_CLUSTER; q < end; q++) test(q);
            }
            __syncthreads();
        }
        s_best[warp][lane] = best;
        s_bt[warp][lane] = bt;
        s_bf[warp][lane] = bf;
        s_cp[warp][lane] = bcp;
        __syncthreads();
        if (warp == 0) {
            for (int w = 1; w < BAKE_WARPS; w++) {
                const float d2 = s_best[w][lane];
                const int t = s_bt[w][lane];
                if (d2 < best || (d2 == best && t < bt && t >= 0)) {
                    best = d2;
                    bt = t;
                    bf = s_bf[w][lane];
                    bcp = s_cp[w][lane];
                }
            }
            if (active) bake_node(x, centre, best, bt, bf, bcp, node, tris, face_n, edge_n, vert_n, phi, grad);
        }
        __syncthreads();
    }
}

struct D3 {
    double x, y, z;
};
inline D3 sub(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
inline D3 add(D3 a, D3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
inline D3 mul(double s, D3 a) { return {s * a.x, s * a.y, s * a.z}; }
inline double dotd(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
inline D3 crossd(D3 a, D3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
inline double lend(D3 a) { return std::sqrt(dotd(a, a)); }

kami_status bake_fail(kami_status st, const std::string& msg) {
    set_last_error(msg.c_str());
    return st;
}

}  // namespace
}  // namespace kami

using namespace kami;

extern "C" kami_status kami_sdf_bake(const float* vertices, int32_t num_vertices, const int32_t* triangles,
                                     int32_t num_triangles, const int32_t dims[3], const float grid_min[3],
                                     const float grid_max[3], float* phi, float* grad, int32_t memory, int32_t device) {
    if (!vertices || !triangles || !dims || !grid_min || !grid_max || !phi || !grad || num_vertices < 3 || num_triangles < 1)
        return bake_fail(KAMI_ERR_INVALID_ARGUMENT, "need a mesh of >= 3 vertices and >= 1 triangle, dims, bounds and outputs");
    if (memory != KAMI_MEMORY_HOST && memory != KAMI_MEMORY_DEVICE) return bake_fail(KAMI_ERR_INVALID_ARGUMENT, "bad memory kind");
    for (int a = 0; a < 3; a++) {
        if (dims[a] <= 0) return bake_fail(KAMI_ERR_INVALID_ARGUMENT, "dims must be > 0");
        if (!(grid_max[a] > grid_min[a])) return bake_fail(KAMI_ERR_INVALID_ARGUMENT, "grid_max must exceed grid_min");
    }
    const int64_t total = (int64_t)dims[0] * dims[1] * dims[2];
    for (int64_t q = 0; q < 3LL * num_vertices; q++)
        if (!std::isfinite(vertices[q])) return bake_fail(KAMI_ERR_INVALID_ARGUMENT, "non-finite mesh vertex");
    // pseudonormals, in double: faces; vertices weighted by the incident angles; edges the sum of
    // their faces' normals (TriangleMeshDistance.h:364-421 builds the same three sets)
    const int32_t nv = num_vertices, nt = num_triangles;
    auto vert = [&](int32_t i) { return D3{vertices[3 * i], vertices[3 * i + 1], vertices[3 * i + 2]}; };
    std::vector<D3> fn(nt), vn(nv, D3{0, 0, 0});
    // edges by their two vertices, numbered through an open-addressed table that is at most half full
    size_t cap = 16;
    while (cap < 6 * (size_t)nt) cap *= 2;
    std::vector<uint32_t> table(cap, ~0u);
    std::vector<uint64_t> edge_key;
    std::vector<D3> edge_sum;
    edge_key.reserve(3 * (size_t)nt / 2 + 1);
    edge_sum.reserve(3 * (size_t)nt / 2 + 1);
    std::vector<uint32_t> edge_of(3 * (size_t)nt);
    std::vector<double> longest(nt);
    for (int32_t t = 0; t < nt; t++) {
        const int32_t* T = triangles + 3 * t;
        for (int q = 0; q < 3; q++)
            if (T[q] < 0 || T[q] >= nv) return bake_fail(KAMI_ERR_INVALID_ARGUMENT, "triangle index out of range");
        const D3 p[3] = {vert(T[0]), vert(T[1]), vert(T[2])};
        D3 n = crossd(sub(p[1], p[0]), sub(p[2], p[0]));
        const double ln = lend(n);
        if (!(ln > 0) || !std::isfinite(ln))
            return bake_fail(KAMI_ERR_GEOMETRY, "triangle " + std::to_string(t) + " has zero area");
        n = mul(1.0 / ln, n);
        fn[t] = n;
        const double len[3] = {lend(sub(p[1], p[0])), lend(sub(p[2], p[1])), lend(sub(p[0], p[2]))};
        longest[t] = std::max({len[0], len[1], len[2]});
        for (int q = 0; q < 3; q++) {
            const D3 e1 = sub(p[(q + 1) % 3], p[q]), e2 = sub(p[(q + 2) % 3], p[q]);
            const double c = dotd(e1, e2) / (len[q] * len[(q + 2) % 3]);
            vn[T[q]] = add(vn[T[q]], mul(std::acos(std::max(-1.0, std::min(1.0, c))), n));
            const int32_t i0 = T[q], i1 = T[(q + 1) % 3];
            const uint64_t key = (uint64_t)(uint32_t)std::min(i0, i1) << 32 | (uint32_t)std::max(i0, i1);
            uint64_t at = key * 0x9E3779B97F4A7C15ull;
            at = (at ^ at >> 32) & (cap - 1);
            while (table[at] != ~0u && edge_key[table[at]] != key) at = (at + 1) & (cap - 1);
            if (table[at] == ~0u) {
                table[at] = (uint32_t)edge_key.size();
                edge_key.push_back(key);
                edge_sum.push_back(n);
            } else {
                edge_sum[table[at]] = add(edge_sum[table[at]], n);
            }
            edge_of[3 * (size_t)t + q] = table[at];
        }
    }
    // Clusters: triangles by the Morton code of their centroids (10 bits an axis of the mesh's box)
    float mlo[3] = {INFINITY, INFINITY, INFINITY}, mhi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t q = 0; q < 3LL * nv; q++) {
        mlo[q % 3] = std::min(mlo[q % 3], vertices[q]);
        mhi[q % 3] = std::max(mhi[q % 3], vertices[q]);
    }
    std::vector<uint64_t> code(nt);
    for (int32_t t = 0; t < nt; t++) {
        uint64_t m = 0;
        for (int a = 0; a < 3; a++) {
            const double c = ((double)vertices[3 * triangles[3 * t] + a] + vertices[3 * triangles[3 * t + 1] + a] +
                              vertices[3 * triangles[3 * t + 2] + a]) / 3.0;
            const double w = (double)mhi[a] - mlo[a];
            uint32_t v = w > 0 ? (uint32_t)std::max(0.0, std::min(1023.0, 1024.0 * ((c - mlo[a]) / w))) : 0;
            v = (v | v << 16) & 0x030000FF;
            v = (v | v << 8) & 0x0300F00F;
            v = (v | v << 4) & 0x030C30C3;
            v = (v | v << 2) & 0x09249249;
            m |= (uint64_t)v << a;
        }
        code[t] = m << 32 | (uint32_t)t;
    }
    {  // by code, equal codes in the mesh's order: three passes over 10 bits each
        std::vector<uint64_t> other(nt);
        for (int pass = 0; pass < 3; pass++) {
            const int shift = 32 + 10 * pass;
            uint32_t at[1024] = {};
            for (uint64_t c : code) at[c >> shift & 1023]++;
            uint32_t sum = 0;
            for (uint32_t& a : at) {
                const uint32_t n = a;
                a = sum;
                sum += n;
            }
            for (uint64_t c : code) other[at[c >> shift & 1023]++] = c;
            code.swap(other);
        }
    }
    const int nc = (nt + BAKE_CLUSTER - 1) / BAKE_CLUSTER;
    // one upload: normals first (16-byte elements), then boxes, corners and indices
    const size_t o_e = sizeof(float4) * (size_t)nt, o_v = o_e + sizeof(float4) * 3 * (size_t)nt,
                 o_c = o_v + sizeof(float4) * (size_t)nv, o_tv = o_c + sizeof(BakeCluster) * (size_t)nc,
                 o_o = o_tv + sizeof(float) * 9 * (size_t)nt, o_t = o_o + sizeof(int32_t) * (size_t)nt,
                 o_end = (o_t + sizeof(int32_t) * 3 * (size_t)nt + 15) / 16 * 16;
    std::vector<char> up(o_end);
    float4 *hf = (float4*)up.data(), *he = (float4*)(up.data() + o_e), *hv = (float4*)(up.data() + o_v);
    BakeCluster* hc = (BakeCluster*)(up.data() + o_c);
    float* tv = (float*)(up.data() + o_tv);
    int32_t* ho = (int32_t*)(up.data() + o_o);
    std::memcpy(up.data() + o_t, triangles, sizeof(int32_t) * 3 * (size_t)nt);
    constexpr double kU = 5.9604644775390625e-8;  // unit roundoff
    for (int32_t c = 0; c < nc; c++) {
        BakeCluster& C = hc[c];
        for (int a = 0; a < 3; a++) {
            C.lo[a] = INFINITY;
            C.hi[a] = -INFINITY;
        }
        double e1 = 0, e2 = 0;
        for (int32_t q = c * BAKE_CLUSTER; q < std::min(nt, (c + 1) * BAKE_CLUSTER); q++) {
            const int32_t t = (int32_t)(uint32_t)code[q];
            const int32_t* T = triangles + 3 * (int64_t)t;
            ho[q] = t;
            for (int a = 0; a < 9; a++) {
                const float v = vertices[3 * (int64_t)T[a / 3] + a % 3];
                tv[9 * (int64_t)q + a] = v;
                C.lo[a % 3] = std::min(C.lo[a % 3], v);
                C.hi[a % 3] = std::max(C.hi[a % 3], v);
            }
            const D3 a = vert(T[0]), b = vert(T[1]), d = vert(T[2]);
            const D3 n = crossd(sub(b, a), sub(d, a));
            const double L = longest[t], A4 = dotd(n, n);
            const double E = A4 > 1e-30 ? 72 * kU * L * L / A4 : INFINITY;  // below: products may underflow
            e1 = std::max(e1, E);
            e2 = std::max(e2, 8 * E * L);
        }
        C.e1 = (float)(1.001 * e1);
        C.e2 = (float)(1.001 * e2);
    }
    std::vector<float4> edge_n(edge_sum.size());  // .w != 0: the sum vanishes, each face takes its own normal
    for (size_t k = 0; k < edge_n.size(); k++) {
        const double le = lend(edge_sum[k]);
        const D3 e = le > 0 ? mul(1.0 / le, edge_sum[k]) : D3{0, 0, 0};
        edge_n[k] = make_float4((float)e.x, (float)e.y, (float)e.z, le > 0 ? 0.f : 1.f);
    }
    for (int32_t t = 0; t < nt; t++) {
        hf[t] = make_float4((float)fn[t].x, (float)fn[t].y, (float)fn[t].z, 0.f);
        for (int q = 0; q < 3; q++) {
            const float4 e = edge_n[edge_of[3 * (size_t)t + q]];
            he[3 * t + q] = e.w == 0.f ? e : hf[t];
        }
    }
    for (int32_t i = 0; i < nv; i++) {
        const double l = lend(vn[i]);
        const D3 n = l > 0 ? mul(1.0 / l, vn[i]) : D3{0, 0, 0};
        hv[i] = make_float4((float)n.x, (float)n.y, (float)n.z, 0.f);
    }

    if (device >= 0) {
        cudaError_t e = cudaSetDevice(device);
        if (e != cudaSuccess) return bake_fail(KAMI_ERR_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(e));
    }
    char* d = nullptr;  // the upload, then the outputs that go to host memory: one allocation
    const size_t out_bytes = memory == KAMI_MEMORY_HOST ? sizeof(float) * 4 * (size_t)total : 0;
    cudaError_t e = cudaMalloc((void**)&d, o_end + out_bytes);
    if (e == cudaSuccess) e = cudaMemcpy(d, up.data(), o_end, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        float* out_phi = memory == KAMI_MEMORY_HOST ? (float*)(d + o_end) : phi;
        float* out_grad = memory == KAMI_MEMORY_HOST ? out_phi + total : grad;
        const float3 lo = f3(grid_min[0], grid_min[1], grid_min[2]);
        // node spacing and grid centre as SDFBodyCollisionSolver / StoreSDFQueries compute them
        const float3 ds = f3((grid_max[0] - grid_min[0]) / (1.f * dims[0]), (grid_max[1] - grid_min[1]) / (1.f * dims[1]),
                             (grid_max[2] - grid_min[2]) / (1.f * dims[2]));
        const float3 centre = f3((grid_max[0] + grid_min[0]) / 2.f, (grid_max[1] + grid_min[1]) / 2.f,
                                 (grid_max[2] + grid_min[2]) / 2.f);
        // rounding of a closest point's coordinates: a few units in the last place of the largest
        float big = 0.f;
        for (int a = 0; a < 3; a++)
            big = std::max({big, std::fabs(mlo[a]), std::fabs(mhi[a]), std::fabs(grid_min[a]), std::fabs(grid_max[a])});
        const float slack = 32.f * (float)kU * big;
        const int64_t bricks = (int64_t)((dims[0] + BX - 1) / BX) * ((dims[1] + BY - 1) / BY) * ((dims[2] + BZ - 1) / BZ);
        const unsigned blocks = (unsigned)std::min<int64_t>(bricks, 1 << 30);
        sdf_bake_kernel<<<blocks, BAKE_THREADS>>>((const float*)(d + o_tv), nt, (const int32_t*)(d + o_o),
                                                  (const BakeCluster*)(d + o_c), nc, (const int32_t*)(d + o_t),
                                                  (const float4*)d, (const float4*)(d + o_e), (const float4*)(d + o_v),
                                                  dims[0], dims[1], dims[2], lo, ds, centre, slack, out_phi, out_grad);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
        if (e == cudaSuccess && memory == KAMI_MEMORY_HOST) {
            e = cudaMemcpy(phi, out_phi, sizeof(float) * total, cudaMemcpyDeviceToHost);
            if (e == cudaSuccess) e = cudaMemcpy(grad, out_grad, sizeof(float) * 3 * total, cudaMemcpyDeviceToHost);
        }
    }
    if (d) cudaFree(d);
    if (e != cudaSuccess)
        return bake_fail(e == cudaErrorMemoryAllocation ? KAMI_ERR_OUT_OF_MEMORY : KAMI_ERR_CUDA,
                         std::string("SDF bake: ") + cudaGetErrorString(e));
    return KAMI_OK;
}
