// F3D2 (reg_f3d2, reg-lib/_reg_f3d2.cpp) on the device: the stationary velocity field of a
// cubic B-spline grid exponentiated by scaling and squaring, composition of deformation fields,
// the "Dartel-like" gradient exponentiation and the symmetrisation of the forward and backward
// velocity grids.
//
// This file is compiled with -fmad=false: every float expression below rounds each product and
// each sum on its own, in the order written, which is the reference's (its SSE build has no
// fused multiply-add), so the arithmetic is the reference's and not a contraction of it.
//
// Fields that stay inside an exponentiation (the flow, the squarings, the intermediate fields and
// gradients) are held as pairs (x, y) followed by a plane of z, in the 3 * n floats of a planar
// field: a tap is then one 8-byte and one 4-byte load instead of three, its pair feeds the packed
// products as it arrives, and no byte is added. Fields that a caller sees are planar x | y | z (the
// NIfTI vector layout). Gathers hit L1/L2 because neighbouring threads read neighbouring voxels.

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "nrb_common.cuh"
#include "nrb_packed.cuh"

namespace nrb {

namespace {

// a dense field over an image grid: dims, voxel -> mm and mm -> voxel (first three rows)
struct FieldGeom {
    int nx, ny, nz;
    Mat34 xyz, ijk;
};

FieldGeom field_geom(const int32_t dim[3], const float xyz[16], const float ijk[16]) {
    FieldGeom f;
    f.nx = dim[0];
    f.ny = dim[1];
    f.nz = dim[2];
    f.xyz = to_mat34(xyz);
    f.ijk = to_mat34(ijk);
    return f;
}

// m0 * x + m1 * y + m2 * z + m3, left to right: the voxel -> mm conversions of
// reg_getDeformationFromDisplacement (reg-lib/cpu/_reg_tools.cpp:2107-2150) and the mm -> voxel
// conversions of the composition (reg-lib/cpu/_reg_localTrans.cpp:2380-2395)
__device__ __forceinline__ float row(const float *m, float x, float y, float z) {
    return m[0] * x + m[1] * y + m[2] * z + m[3];
}

__device__ __forceinline__ int floor_int(float v) {
    // Floor<int> of the reference, clamped so that a position far outside (or NaN) stays a
    // defined integer; the sliding clamp below keeps every read inside the field
    float f = floorf(v);
    f = f != f ? 0.f : fminf(fmaxf(f, -1073741824.f), 1073741824.f);
    return (int)f;
}
__device__ __forceinline__ int ceil_int(float v) {
    float f = ceilf(v);
    f = f != f ? 0.f : fminf(fmaxf(f, -1073741824.f), 1073741824.f);
    return (int)f;
}

// a / 6 correctly rounded, from the rounded reciprocal and one residual step (P. Markstein, IBM J.
// Res. Dev. 34, 1990): three FP64 operations. a is 0 or of normal size here (sums of cubes of
// floats), so no step underflows.
__device__ __forceinline__ double sixth(double a) {
    const double inv = 1.0 / 6.0, q = a * inv;
    return __fma_rn(__fma_rn(-6.0, q, a), inv, q);
}

// get_BSplineBasisValues (reg-lib/cpu/_reg_splineBasis.cpp:17-26): the cube and the polynomial
// sums in double, as the reference writes them
__device__ __forceinline__ void bspline_basis_f64(float b, float v[4]) {
    const float ff = b * b, fff = ff * b;
    const float mf = (float)(1.0 - (double)b);
    v[0] = (float)sixth((double)(mf * mf * mf));
    v[1] = (float)sixth(3.0 * (double)fff - 6.0 * (double)ff + 4.0);
    v[2] = (float)sixth(-3.0 * (double)fff + 3.0 * (double)ff + 3.0 * (double)b + 1.0);
    v[3] = (float)sixth((double)fff);
}

// A vector field of n voxels in one of the two layouts
template <bool kPairs>
struct VecField {
    const float *p;
    long long n;
    __device__ __forceinline__ void load(long long i, float& x, float& y, float& z) const {
        if (kPairs) {
            const float2 q = __ldg(reinterpret_cast<const float2 *>(p) + i);
            x = q.x;
            y = q.y;
            z = __ldg(p + 2 * n + i);
        } else {
            x = __ldg(p + i);
            y = __ldg(p + n + i);
            z = __ldg(p + 2 * n + i);
        }
    }
};
template <bool kPairs>
__device__ __forceinline__ void store_vec(float *p, long long n, long long i, float x, float y, float z) {
    if (kPairs) {
        reinterpret_cast<float2 *>(p)[i] = make_float2(x, y);
    } else {
        p[i] = x;
        p[n + i] = y;
    }
    p[2 * n + i] = z;
}

// get_SlidedValues (reg-lib/cpu/_reg_splineBasis.cpp:497-550) for a field of positions: the
// value at the clamped index, shifted by the voxel -> mm columns times the clamped distance
template <typename Field>
__device__ __forceinline__ void slided(const Field& F, int x, int y, int z, int nx, int ny, int nz,
                                       const Mat34& xyz, float& vx, float& vy, float& vz) {
    const int cx = x < 0 ? 0 : (x >= nx ? nx - 1 : x);
    const int cy = y < 0 ? 0 : (y >= ny ? ny - 1 : y);
    const int cz = z < 0 ? 0 : (z >= nz ? nz - 1 : z);
    const float sx = (float)(x - cx), sy = (float)(y - cy), sz = (float)(z - cz);
    const long long i = ((long long)cz * ny + cy) * nx + cx;
    F.load(i, vx, vy, vz);
    vx = vx + (sx * xyz.m[0] + sy * xyz.m[1] + sz * xyz.m[2]);
    vy = vy + (sx * xyz.m[4] + sy * xyz.m[5] + sz * xyz.m[6]);
    vz = vz + (sx * xyz.m[8] + sy * xyz.m[9] + sz * xyz.m[10]);
}

// order-preserving float <-> unsigned for atomic min / max
__device__ __forceinline__ unsigned fkey(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
float fkey_inv(unsigned k) {
    const unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    memcpy(&f, &u, 4);
    return f;
}

// reg_spline_getFlowFieldFromVelocityGrid (reg-lib/cpu/_reg_localTrans.cpp:3465-3491) followed by
// the displacement conversion of reg_defField_getDeformationFieldFromFlowField (:3497-3511): the
// velocity grid evaluated (cubic B-spline, composition path :903-1079) at the identity position
// of every voxel, minus that position. The 64 taps are summed as the SSE build sums them: four
// x-lanes accumulated over (z, y), then the lanes added in order. Also the extrema of all three
// components (the squaring-number rule, :3514-3521).
// One axis of the flow's sampling when the field's voxel -> mm and the grid's mm -> voxel
// matrices are both diagonal: then the identity coordinate, the grid coordinate and so the node
// index and the four basis values along an axis depend on that axis's voxel index alone (every
// off-diagonal product is an exact zero and adds nothing), and are the same floats as the
// per-voxel evaluation gives.
struct AxisEntry {
    float w[4];
    float r;  // identity coordinate (mm)
    int pre;  // first node
};

// the three axes' tables (blockIdx.y = axis) end to end, and the cleared extrema of the flow that
// follows
__global__ void k_axis_table(FieldGeom f, Mat34 gijk, AxisEntry *__restrict__ out, unsigned *__restrict__ minmax) {
    const int axis = blockIdx.y, n = axis == 0 ? f.nx : (axis == 1 ? f.ny : f.nz);
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (minmax && axis == 0 && t == 0) {
        minmax[0] = 0xffffffffu;
        minmax[1] = 0u;
    }
    if (t >= n) return;
    const float fx = axis == 0 ? (float)t : 0.f, fy = axis == 1 ? (float)t : 0.f, fz = axis == 2 ? (float)t : 0.f;
    const float rx = row(f.xyz.m, fx, fy, fz), ry = row(f.xyz.m + 4, fx, fy, fz), rz = row(f.xyz.m + 8, fx, fy, fz);
    const float v = row(gijk.m + 4 * axis, rx, ry, rz);
    const int p = floor_int(v);
    const float b = v - (float)p;
    AxisEntry e;
    bspline_basis_f64(b < 0 ? 0.f : b, e.w);
    e.r = axis == 0 ? rx : (axis == 1 ? ry : rz);
    e.pre = p - 1;
    out[(axis > 0 ? f.nx : 0) + (axis > 1 ? f.ny : 0) + t] = e;
}

// What the flow kernels write per voxel: the displacement, with its extrema over all components
// (kExtrema; the squaring number follows from them), or the scaled deformation the squarings start
// from (reg_defField_getDeformationFieldFromFlowField, :3537-3547; scale = 2^-N, exact, as the
// reference's double division by 2^N is). Pairs layout.
template <bool kExtrema>
__device__ __forceinline__ void flow_out(float *out, long long n, long long i, float ox, float oy, float oz, float rx,
                                         float ry, float rz, float scale, float& lo, float& hi) {
    const float dx = ox - rx, dy = oy - ry, dz = oz - rz;
    if (kExtrema) {
        store_vec<true>(out, n, i, dx, dy, dz);
        lo = fminf(lo, fminf(fminf(dx, dy), dz));
        hi = fmaxf(hi, fmaxf(fmaxf(dx, dy), dz));
    } else {
        store_vec<true>(out, n, i, dx * scale + rx, dy * scale + ry, dz * scale + rz);
    }
}

// the block's extrema, then one pair of atomics per block (one per warp serialised in L2)
__device__ __forceinline__ void flow_extrema(float lo, float hi, unsigned *minmax) {
    __shared__ float slo[8], shi[8];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((tid & 31) == 0) {
        slo[tid >> 5] = lo;
        shi[tid >> 5] = hi;
    }
    __syncthreads();
    if (tid != 0) return;
#pragma unroll
    for (int w = 1; w < 8; ++w) {
        lo = fminf(lo, slo[w]);
        hi = fmaxf(hi, shi[w]);
    }
    if (lo <= hi) {
        atomicMin(minmax, fkey(lo));
        atomicMax(minmax + 1, fkey(hi));
    }
}

// sums of the four x-lanes of a voxel's 64 taps, lanes in pairs (0, 1) and (2, 3)
struct FlowSums {
    F2 x01, x23, y01, y23, z01, z23;
};
__device__ __forceinline__ void flow_clear(FlowSums& t) { t.x01 = t.x23 = t.y01 = t.y23 = t.z01 = t.z23 = f2(0.f); }
// one row of four taps (values v[component][lane pair]) with the row weight yz = By * Bz
__device__ __forceinline__ void flow_row(FlowSums& t, const F2 v[3][2], float yz, F2 xb01, F2 xb23) {
    const F2 w = f2(yz), w01 = mul2(w, xb01), w23 = mul2(w, xb23);
    t.x01 = add2(mul2(w01, v[0][0]), t.x01);
    t.x23 = add2(mul2(w23, v[0][1]), t.x23);
    t.y01 = add2(mul2(w01, v[1][0]), t.y01);
    t.y23 = add2(mul2(w23, v[1][1]), t.y23);
    t.z01 = add2(mul2(w01, v[2][0]), t.z01);
    t.z23 = add2(mul2(w23, v[2][1]), t.z23);
}
__device__ __forceinline__ float flow_lanes(F2 a, F2 b) {
    float v0, v1, v2, v3;
    split(a, v0, v1);
    split(b, v2, v3);
    return v0 + v1 + v2 + v3;
}
__device__ __forceinline__ void flow_load_row(const float *__restrict__ q, long long gn, F2 v[3][2]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        v[k][0] = f2(__ldg(q + k * gn), __ldg(q + k * gn + 1));
        v[k][1] = f2(__ldg(q + k * gn + 2), __ldg(q + k * gn + 3));
    }
}

// w0, w1, w2, w3 <- w1, w2, w3, w0: the next weight of a rolled loop without a register array index
__device__ __forceinline__ void rotate4(float w[4]) {
    const float t = w[0];
    w[0] = w[1];
    w[1] = w[2];
    w[2] = w[3];
    w[3] = t;
}

// a voxel with a tap outside the grid: sliding values, the taps in the same order
__device__ __forceinline__ void flow_border(const VecField<false>& vel, int gx, int gy, int gz, const Mat34& gxyz, int xp,
                                            int yp, int zp, const float xb[4], const float yb[4], const float zb[4],
                                            float& ox, float& oy, float& oz) {
    float tx[4] = { 0.f, 0.f, 0.f, 0.f }, ty[4] = { 0.f, 0.f, 0.f, 0.f }, tz[4] = { 0.f, 0.f, 0.f, 0.f };
    float wy[4] = { yb[0], yb[1], yb[2], yb[3] }, wz[4] = { zb[0], zb[1], zb[2], zb[3] };
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
#pragma unroll 1
        for (int bb = 0; bb < 4; ++bb) {
            const float yz = wy[0] * wz[0];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const float w = yz * xb[a];
                float px, py, pz;
                slided(vel, xp + a, yp + bb, zp + c, gx, gy, gz, gxyz, px, py, pz);
                tx[a] = w * px + tx[a];
                ty[a] = w * py + ty[a];
                tz[a] = w * pz + tz[a];
            }
            rotate4(wy);
        }
        rotate4(wz);
    }
    ox = tx[0] + tx[1] + tx[2] + tx[3];
    oy = ty[0] + ty[1] + ty[2] + ty[3];
    oz = tz[0] + tz[1] + tz[2] + tz[3];
}

// The flow with the axis tables. A thread takes kFlowVox consecutive slices of its column: they
// share most node planes (a plane spans the grid spacing, five voxels as a rule), so the twelve
// values of a node row are loaded once for all slices that use its plane. The slices of a block are
// the same for all its threads, so which slice uses a plane is a uniform test. Every voxel's taps
// keep their order (z, then y, four x-lanes).
//
// Bound by the FP32 lanes: 464 products and sums per voxel, none fusable (92 us for 182x218x182 at
// the lane rate). One voxel per thread took 362 us (1280 warp instructions per 32 voxels, 192 of
// them loads).
constexpr int kFlowVox = 5;

template <bool kExtrema>
__global__ void __launch_bounds__(256, 2) k_velocity_flow_table(const float *__restrict__ vel, int gx, int gy, int gz,
                                                            Mat34 gxyz, FieldGeom f, const AxisEntry *__restrict__ tab,
                                                            float *__restrict__ out, float scale,
                                                            unsigned *__restrict__ minmax) {
    const int x = blockIdx.x * 32 + threadIdx.x;
    const AxisEntry *tz = tab + f.nx + f.ny;
    const long long n = (long long)f.nx * f.ny * f.nz, gn = (long long)gx * gy * gz;
    float lo = INFINITY, hi = -INFINITY;
    const int groups = (f.nz + kFlowVox - 1) / kFlowVox;
    for (int y = blockIdx.y * 8 + threadIdx.y; y < f.ny && x < f.nx; y += gridDim.y * 8)
    for (int group = blockIdx.z; group < groups; group += gridDim.z) {
        const int z0 = group * kFlowVox;
        const AxisEntry ex = tab[x], ey = tab[f.nx + y];
        const int nv = min(kFlowVox, f.nz - z0);
        int pre[kFlowVox];
#pragma unroll
        for (int v = 0; v < kFlowVox; ++v) pre[v] = tz[z0 + min(v, nv - 1)].pre;
        // node planes ascend or descend with z (the sign of the matrices); either way these bound them
        int c0 = pre[0], c1 = pre[0];
#pragma unroll
        for (int v = 1; v < kFlowVox; ++v) {
            c0 = min(c0, pre[v]);
            c1 = max(c1, pre[v]);
        }
        c1 += 3;
        const long long i0 = ((long long)z0 * f.ny + y) * f.nx + x, plane = (long long)f.nx * f.ny;
        if (ex.pre >= 0 && ex.pre + 3 < gx && ey.pre >= 0 && ey.pre + 3 < gy && c0 >= 0 && c1 < gz) {
            const F2 xb01 = f2(ex.w[0], ex.w[1]), xb23 = f2(ex.w[2], ex.w[3]);
            FlowSums t[kFlowVox];
#pragma unroll
            for (int v = 0; v < kFlowVox; ++v) flow_clear(t[v]);
            const float *p = vel + ((long long)c0 * gy + ey.pre) * gx + ex.pre;
            for (int c = c0; c <= c1; ++c, p += (long long)gx * gy) {
                float zw[kFlowVox];
                bool use[kFlowVox], any = false;
#pragma unroll
                for (int v = 0; v < kFlowVox; ++v) {
                    use[v] = (unsigned)(c - pre[v]) < 4u;
                    any = any || use[v];
                    zw[v] = use[v] ? tz[z0 + min(v, nv - 1)].w[c - pre[v]] : 0.f;
                }
                if (!any) continue;
                const float *q = p;
#pragma unroll
                for (int bb = 0; bb < 4; ++bb, q += gx) {
                    F2 r[3][2];
                    flow_load_row(q, gn, r);
#pragma unroll
                    for (int v = 0; v < kFlowVox; ++v)
                        if (use[v]) flow_row(t[v], r, ey.w[bb] * zw[v], xb01, xb23);
                }
            }
#pragma unroll
            for (int v = 0; v < kFlowVox; ++v)
                if (v < nv)
                    flow_out<kExtrema>(out, n, i0 + v * plane, flow_lanes(t[v].x01, t[v].x23), flow_lanes(t[v].y01, t[v].y23),
                                       flow_lanes(t[v].z01, t[v].z23), ex.r, ey.r, tz[z0 + v].r, scale, lo, hi);
        } else {
            const VecField<false> F{ vel, gn };
#pragma unroll 1
            for (int v = 0; v < nv; ++v) {
                const AxisEntry ez = tz[z0 + v];
                float ox, oy, oz;
                flow_border(F, gx, gy, gz, gxyz, ex.pre, ey.pre, ez.pre, ex.w, ey.w, ez.w, ox, oy, oz);
                flow_out<kExtrema>(out, n, i0 + v * plane, ox, oy, oz, ex.r, ey.r, ez.r, scale, lo, hi);
            }
        }
    }
    if (kExtrema) flow_extrema(lo, hi, minmax);
}

// The flow of a field in any orientation: one voxel per thread, its basis evaluated in full. 64
// registers for four blocks per SM: an exponentiation of an oblique 160x192x160 field takes 603 us,
// 613 at 80 registers (2.2 ms before the pairs layout and the pool).
template <bool kExtrema>
__global__ void __launch_bounds__(256, 4) k_velocity_flow(const float *__restrict__ vel, int gx, int gy, int gz,
                                                      Mat34 gxyz, Mat34 gijk, FieldGeom f, float *__restrict__ out,
                                                      float scale, unsigned *__restrict__ minmax) {
    const long long n = (long long)f.nx * f.ny * f.nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float lo = INFINITY, hi = -INFINITY;
    if (i < n) {
        const int x = (int)(i % f.nx), y = (int)((i / f.nx) % f.ny), z = (int)(i / ((long long)f.nx * f.ny));
        const float fx = (float)x, fy = (float)y, fz = (float)z;
        const float rx = row(f.xyz.m, fx, fy, fz), ry = row(f.xyz.m + 4, fx, fy, fz), rz = row(f.xyz.m + 8, fx, fy, fz);
        const float vx = row(gijk.m, rx, ry, rz), vy = row(gijk.m + 4, rx, ry, rz), vz = row(gijk.m + 8, rx, ry, rz);
        int xp = floor_int(vx), yp = floor_int(vy), zp = floor_int(vz);
        float xb[4], yb[4], zb[4];
        float b = vx - (float)xp;
        bspline_basis_f64(b < 0 ? 0.f : b, xb);
        b = vy - (float)yp;
        bspline_basis_f64(b < 0 ? 0.f : b, yb);
        b = vz - (float)zp;
        bspline_basis_f64(b < 0 ? 0.f : b, zb);
        --xp;
        --yp;
        --zp;
        const long long gn = (long long)gx * gy * gz;
        float ox, oy, oz;
        if (xp >= 0 && xp + 3 < gx && yp >= 0 && yp + 3 < gy && zp >= 0 && zp + 3 < gz) {
            // every tap inside the grid: one row pointer stepped through the rows
            const F2 xb01 = f2(xb[0], xb[1]), xb23 = f2(xb[2], xb[3]);
            FlowSums t;
            flow_clear(t);
            const float *q = vel + ((long long)zp * gy + yp) * gx + xp;
#pragma unroll
            for (int c = 0; c < 4; ++c, q += (long long)gx * (gy - 4)) {
#pragma unroll
                for (int bb = 0; bb < 4; ++bb, q += gx) {
                    F2 r[3][2];
                    flow_load_row(q, gn, r);
                    flow_row(t, r, yb[bb] * zb[c], xb01, xb23);
                }
            }
            ox = flow_lanes(t.x01, t.x23);
            oy = flow_lanes(t.y01, t.y23);
            oz = flow_lanes(t.z01, t.z23);
        } else {
            flow_border(VecField<false>{ vel, gn }, gx, gy, gz, gxyz, xp, yp, zp, xb, yb, zb, ox, oy, oz);
        }
        flow_out<kExtrema>(out, n, i, ox, oy, oz, rx, ry, rz, scale, lo, hi);
    }
    if (kExtrema) flow_extrema(lo, hi, minmax);
}

__global__ void k_minmax_init(unsigned *minmax) {
    minmax[0] = 0xffffffffu;
    minmax[1] = 0u;
}

// displacement / 2^N back to a deformation (reg_defField_getDeformationFieldFromFlowField,
// :3537-3547) once N is known from the extrema: scale is 2^-N. Pairs layout; out may be d.
__global__ void __launch_bounds__(256) k_flow_scale(const float *d, float *out, float scale, FieldGeom f) {
    const int x = blockIdx.x * 64 + threadIdx.x % 64;
    if (x >= f.nx) return;
    const long long n = (long long)f.nx * f.ny * f.nz, plane = (long long)f.nx * f.ny;
    for (int y = blockIdx.y * 4 + threadIdx.x / 64; y < f.ny; y += gridDim.y * 4)
    for (int z = blockIdx.z; z < f.nz; z += gridDim.z) {
        const float fx = (float)x, fy = (float)y;
        const long long i = z * plane + (long long)y * f.nx + x;
        const float2 q = reinterpret_cast<const float2 *>(d)[i];
        const float w = d[2 * n + i], fz = (float)z;
        store_vec<true>(out, n, i, q.x * scale + row(f.xyz.m, fx, fy, fz), q.y * scale + row(f.xyz.m + 4, fx, fy, fz),
                        w * scale + row(f.xyz.m + 8, fx, fy, fz));
    }
}

// reg_defField_compose3D (reg-lib/cpu/_reg_localTrans.cpp:2334-2458): out(x) = apply(pos(x)),
// trilinear in the apply field's voxel space, sliding (linear extrapolation of the positions)
// outside it. out may alias pos (each voxel reads only its own position), never apply.
// kPairs: apply and pos are in the pairs layout (a squaring applies a field to itself); kOutPairs:
// so is out. I: an index type that holds 3 * n.
//
// Bound by the L1 data stage (a gather of 32 neighbours touches three to four lines: 89 wavefronts
// per 32 voxels, whatever the layout) and by latency, so the registers are cut to the full 64 warps
// per SM: a squaring of 182x218x182 takes 93 us at 32 registers, 104 at 48, 116 at 64 (four voxels
// per thread in the planar layout at 80: 142). Blocks of 32x8, 32x4x2 or 64x4 voxels instead of
// runs of 256 measured 3 to 7% slower. Planar fields come from a caller and may leave the volume
// anywhere: their border path is unrolled, at 48 registers (smooth fields take the same time; a field
// composed with itself until it has left 256x256x256 594 us, 666 like the pairs).
template <bool kPairs, bool kOutPairs, typename I>
__global__ void __launch_bounds__(256, kPairs ? 8 : 5) k_compose(const float *__restrict__ apply, const float *pos, float *out,
                                                FieldGeom f) {
    const I n = (I)f.nx * f.ny * f.nz;
    const I i = (I)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const VecField<kPairs> A{ apply, n };
    float px, py, pz;
    if (kPairs) {
        const float2 q = reinterpret_cast<const float2 *>(pos)[i];
        px = q.x;
        py = q.y;
    } else {
        px = pos[i];
        py = pos[n + i];
    }
    pz = pos[2 * n + i];
    const float vx = row(f.ijk.m, px, py, pz), vy = row(f.ijk.m + 4, px, py, pz), vz = row(f.ijk.m + 8, px, py, pz);
    const int x0 = floor_int(vx), y0 = floor_int(vy), z0 = floor_int(vz);
    float rx[2], ry[2], rz[2];
    rx[1] = vx - (float)x0;
    rx[0] = 1.f - rx[1];
    ry[1] = vy - (float)y0;
    ry[0] = 1.f - ry[1];
    rz[1] = vz - (float)z0;
    rz[0] = 1.f - rz[1];
    F2 oxy = f2(0.f);
    float oz = 0.f;
    if (x0 >= 0 && x0 + 1 < f.nx && y0 >= 0 && y0 + 1 < f.ny && z0 >= 0 && z0 + 1 < f.nz) {
        // every tap inside the field: offsets from one base, the taps in the same order
        const I j0 = ((I)z0 * f.ny + y0) * f.nx + x0;
        const I sy = f.nx, sz = (I)f.nx * f.ny;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const I j = j0 + c * sz + b * sy;
                const float tb = ry[b] * rz[c];
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const float w = rx[a] * tb;
                    float vx_, vy_, vz_;
                    A.load(j + a, vx_, vy_, vz_);
                    oxy = add2(oxy, mul2(f2(vx_, vy_), f2(w)));
                    oz = oz + vz_ * w;
                }
            }
        }
    } else {
#pragma unroll(kPairs ? 1 : 2)
        for (int c = 0; c < 2; ++c) {
            const int z = z0 + c;
#pragma unroll(kPairs ? 1 : 2)
            for (int b = 0; b < 2; ++b) {
                const int y = y0 + b;
                const float tb = (b ? ry[1] : ry[0]) * (c ? rz[1] : rz[0]);
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const int x = x0 + a;
                    float dx, dy, dz;
                    if (x > -1 && x < f.nx && y > -1 && y < f.ny && z > -1 && z < f.nz)
                        A.load(((I)z * f.ny + y) * f.nx + x, dx, dy, dz);
                    else
                        slided(A, x, y, z, f.nx, f.ny, f.nz, f.xyz, dx, dy, dz);
                    const float w = rx[a] * tb;
                    oxy = add2(oxy, mul2(f2(dx, dy), f2(w)));
                    oz = oz + dz * w;
                }
            }
        }
    }
    float ox, oy;
    split(oxy, ox, oy);
    store_vec<kOutPairs>(out, n, i, ox, oy, oz);
}

struct Mat33f {
    float m[9];
};

// One step of Compute::ExponentiateGradient (reg-lib/Compute.cpp:288-330):
//   out = (J * trilinear(g, def(x)) + g(x)) * scale
// reg_trilinearResampleGradient (reg-lib/cpu/_reg_resampling.cpp:1537-1766) with padding 0: the
// vector image g (on the field's own grid) sampled at def(x), reoriented by the finite-difference
// Jacobian of def (forward differences, backward at the last index, where the other axes'
// differences are taken one slice back as the reference's weights select), premultiplied by
// `reorient` and divided by the real spacing per column; then reg_tools_addImageToImage, and on
// the last step the division by 2^N (scale = 2^-N, exact).
// def is in the pairs layout, g in it when kInPairs, out when kOutPairs. A division by the spacing
// is a product where the spacing is a power of two (the same float). Waits on its gathers: 40
// registers for six blocks per SM; a transport of 160x192x160 (N = 6, the squarings included) takes
// 1154 us, 1240 at 64 registers, 3.9 ms or more planar with the buffers mapped by each call.
template <bool kInPairs, bool kOutPairs, typename I>
__global__ void __launch_bounds__(256, 6) k_gradient_exp_step(const float *__restrict__ g, const float *__restrict__ def,
                                                          float *__restrict__ out, FieldGeom f, Mat33f R, float spx,
                                                          float spy, float spz, int unit, float scale) {
    const I n = (I)f.nx * f.ny * f.nz;
    const I i = (I)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int x = (int)(i % f.nx), y = (int)((i / f.nx) % f.ny), z = (int)(i / ((I)f.nx * f.ny));
    const VecField<true> D{ def, n };
    const VecField<kInPairs> G{ g, n };
    // sampling position in the gradient image's voxels
    float px, py, pz;
    D.load(i, px, py, pz);
    const float cx = row(f.ijk.m, px, py, pz), cy = row(f.ijk.m + 4, px, py, pz), cz = row(f.ijk.m + 8, px, py, pz);
    int ax[2], ay[2], az[2];
    ax[0] = floor_int(cx);
    ax[1] = ceil_int(cx);
    ay[0] = floor_int(cy);
    ay[1] = ceil_int(cy);
    az[0] = floor_int(cz);
    az[1] = ceil_int(cz);
    float bx[2], by[2], bz[2];
    bx[1] = fabsf(cx - (float)ax[0]);
    by[1] = fabsf(cy - (float)ay[0]);
    bz[1] = fabsf(cz - (float)az[0]);
    bx[0] = 1.f - bx[1];
    by[0] = 1.f - by[1];
    bz[0] = 1.f - bz[1];
    F2 vxy = f2(0.f);
    float vz = 0.f;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const bool in = (unsigned)az[c] < (unsigned)f.nz && (unsigned)ay[b] < (unsigned)f.ny;
            const I j = ((I)az[c] * f.ny + ay[b]) * f.nx;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                const float w = bx[a] * by[b] * bz[c];
                if (in && (unsigned)ax[a] < (unsigned)f.nx) {
                    float gx, gy, gz;
                    G.load(j + ax[a], gx, gy, gz);
                    vxy = add2(vxy, mul2(f2(gx, gy), f2(w)));
                    vz = vz + gz * w;
                }
                // a tap outside adds padding (0) * weight: nothing
            }
        }
    }
    float vx, vy;
    split(vxy, vx, vy);
    // Jacobian of the deformation by finite differences
    const int bxi = x == f.nx - 1 ? x - 1 : x, byi = y == f.ny - 1 ? y - 1 : y, bzi = z == f.nz - 1 ? z - 1 : z;
    const I base = ((I)bzi * f.ny + byi) * f.nx + bxi;
    float o[3], e[3][3];
    D.load(base, o[0], o[1], o[2]);
    D.load(base + 1, e[0][0], e[0][1], e[0][2]);
    D.load(base + f.nx, e[1][0], e[1][1], e[1][2]);
    D.load(base + (I)f.nx * f.ny, e[2][0], e[2][1], e[2][2]);
    float J[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int col = 0; col < 3; ++col) J[3 * r + col] = e[col][r] - o[r];
    // nifti_mat33_mul(reorient, J), then the division by the real spacing per column
    float M[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int col = 0; col < 3; ++col)
            M[3 * r + col] = R.m[3 * r] * J[col] + R.m[3 * r + 1] * J[3 + col] + R.m[3 * r + 2] * J[6 + col];
    if (unit) {  // spx, spy, spz hold the reciprocals
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            M[3 * r] = M[3 * r] * spx;
            M[3 * r + 1] = M[3 * r + 1] * spy;
            M[3 * r + 2] = M[3 * r + 2] * spz;
        }
    } else {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            M[3 * r] = M[3 * r] / spx;
            M[3 * r + 1] = M[3 * r + 1] / spy;
            M[3 * r + 2] = M[3 * r + 2] / spz;
        }
    }
    const float tx = M[0] * vx + M[1] * vy + M[2] * vz;
    const float ty = M[3] * vx + M[4] * vy + M[5] * vz;
    const float tz = M[6] * vx + M[7] * vy + M[8] * vz;
    float gx, gy, gz;
    G.load(i, gx, gy, gz);
    store_vec<kOutPairs>(out, n, i, (tx + gx) * scale, (ty + gy) * scale, (tz + gz) * scale);
}

// Compute::SymmetriseVelocityFields (reg-lib/Compute.cpp:356-392): both grids as displacements,
// forward = (fw - bw) / 2, backward = (bw - fw) / 2, back to positions. Both grids share dims.
__global__ void __launch_bounds__(256) k_symmetrise(float *__restrict__ fw, float *__restrict__ bw, int nx, int ny,
                                                   int nz, Mat34 fxyz, Mat34 bxyz) {
    const long long n = (long long)nx * ny * nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int x = (int)(i % nx), y = (int)((i / nx) % ny), z = (int)(i / ((long long)nx * ny));
    const float fx = (float)x, fy = (float)y, fz = (float)z;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float idf = row(fxyz.m + 4 * k, fx, fy, fz), idb = row(bxyz.m + 4 * k, fx, fy, fz);
        const float df = fw[k * n + i] - idf, db = bw[k * n + i] - idb;
        fw[k * n + i] = (df - db) * 0.5f + idf;
        bw[k * n + i] = (db - df) * 0.5f + idb;
    }
}

// reg_voxelCentricToNodeCentric (reg-lib/cpu/_reg_localTrans.cpp:1540-1685) for a grid in any
// orientation relative to the image: each node mapped into the image's voxels (T = image ijk x
// grid xyz, Mat44Mul in double), the convolved voxel gradient sampled trilinearly (0 outside),
// reoriented by the transpose of R and scaled by the weight. One thread per node.
__global__ void k_voxel_to_node_general(const float *__restrict__ vox, int nx, int ny, int nz, Mat34 T, Mat33f R,
                                        float weight, int cx, int cy, int cz, float *__restrict__ node) {
    const long long nc = (long long)cx * cy * cz, nv = (long long)nx * ny * nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc) return;
    const double gx = (double)(i % cx), gy = (double)((i / cx) % cy), gz = (double)(i / ((long long)cx * cy));
    float v[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
        v[r] = (float)((double)T.m[4 * r] * gx + (double)T.m[4 * r + 1] * gy + (double)T.m[4 * r + 2] * gz +
                       (double)T.m[4 * r + 3]);
    int pre[3];
    float b[3][2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        pre[k] = floor_int(v[k]);
        b[k][1] = v[k] - (float)pre[k];
        b[k][0] = 1.f - b[k][1];
    }
    float iv0 = 0.f, iv1 = 0.f, iv2 = 0.f;
    for (int c = 0; c < 2; ++c) {
        const int Z = pre[2] + c;
        if (Z <= -1 || Z >= nz) continue;
        for (int bb = 0; bb < 2; ++bb) {
            const int Y = pre[1] + bb;
            if (Y <= -1 || Y >= ny) continue;
            for (int a = 0; a < 2; ++a) {
                const int X = pre[0] + a;
                if (X <= -1 || X >= nx) continue;
                const long long j = ((long long)Z * ny + Y) * nx + X;
                float lw = b[0][a] * b[1][bb];
                lw = lw * b[2][c];
                iv0 = iv0 + lw * __ldg(vox + j);
                iv1 = iv1 + lw * __ldg(vox + nv + j);
                iv2 = iv2 + lw * __ldg(vox + 2 * nv + j);
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float ro = R.m[d] * iv0 + R.m[3 + d] * iv1 + R.m[6 + d] * iv2;
        node[d * nc + i] = ro * weight;
    }
}

inline unsigned blocks_for(long long n) { return (unsigned)((n + 255) / 256); }
// whether 3 * n fits the 32-bit index arithmetic of the gathers
inline bool small_field(long long n) { return n < (1LL << 29); }

// The pairs layout needs 8-byte alignment. A caller's buffer that lacks it is not used as one: a
// temporary takes its place between the steps (the step that writes the caller's planar result
// stores single floats).
inline bool holds_pairs(const float *p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; }
struct PairBuffer {
    float *p = nullptr;
    float *own = nullptr;
    cudaStream_t st;
    explicit PairBuffer(cudaStream_t s): st(s) {}
    nrb_status set(float *buffer, long long n) {
        p = buffer;
        if (!buffer || holds_pairs(buffer)) return NRB_OK;
        NRB_CUDA(tmp_alloc(&own, 3 * n * sizeof(float), st));
        p = own;
        return NRB_OK;
    }
    ~PairBuffer() {
        if (own) cudaFreeAsync(own, st);
    }
};

// algorithmic bytes of one composition per voxel: its position read, the applied field read once
// and the result written, 3 x 4 bytes each; a squaring step applies the field to itself, so the
// positions and the applied field are one read
constexpr double kComposeBytes = 36.0, kSquaringBytes = 24.0;

}  // namespace

// floats from one intermediate field to the next (every field starts 16-byte aligned)
int64_t velocity_field_stride(int64_t nvox) { return (3 * nvox + 3) & ~int64_t(3); }

// The squaring-number rule of reg_defField_getDeformationFieldFromFlowField (:3514-3526): the
// smallest N with max|displacement| / 2^N < 0.28 (3D), at least 6.
int velocity_squaring_steps(float vmin, float vmax) {
    float extrema = std::max(std::fabs(vmin), vmax);
    int steps = 1;
    while (extrema / static_cast<float>(std::pow(2, steps)) >= 0.28f) ++steps;
    return std::max(steps, 6);
}

// reg_spline_getDefFieldFromVelocityGrid (reg-lib/cpu/_reg_localTrans.cpp:3583-3613) and
// reg_spline_getIntermediateDefFieldFromVelGrid (:3616-3681) on the field grid g->ref_* from the
// velocity grid g->cpp_*. *steps is the grid's squaring number (its intent_p2); with update it is
// first recomputed from this flow (a host read of the extrema). def (optional) receives the
// exponentiated field (planar); fields (optional) the fields after 0..N-1 squarings in the pairs
// layout, velocity_field_stride(nvox) floats apart. scratch: 3 * nvox floats, 8-byte aligned;
// minmax: 2 unsigned on the device.
nrb_status velocity_to_deformation(const nrb_geometry *g, const float *vel, bool update, int *steps, float *def,
                                   float *fields, float *scratch, unsigned *minmax, cudaStream_t st) {
    const FieldGeom f = field_geom(g->ref_dim, g->ref_xyz, g->ref_ijk);
    const long long n = nvox(g->ref_dim);
    if (!def && !fields) return fail(NRB_ERR_INVALID, "velocity exponentiation: no output");
    KernelTimer stage(TK_F2_VELOCITY, 0.0, st);
    int N = *steps;
    // the flow lands where the squarings start: the first intermediate field, or the buffer from
    // which N ping-pong squarings end in def
    PairBuffer ping(st);
    if (!fields) NRB_TRY(ping.set(def, n));
    const int64_t fs = velocity_field_stride(n);
    float *first = fields ? fields : (N % 2 == 0 ? ping.p : scratch);
    auto diagonal = [](const float *m) {
        return m[1] == 0.f && m[2] == 0.f && m[4] == 0.f && m[6] == 0.f && m[8] == 0.f && m[9] == 0.f;
    };
    const float scale = update ? 1.f : std::ldexp(1.f, -N);
    const Mat34 gxyz = to_mat34(g->cpp_xyz), gijk = to_mat34(g->cpp_ijk);
    const int32_t *gd = g->cpp_dim;
    if (diagonal(g->ref_xyz) && diagonal(g->cpp_ijk)) {
        AxisEntry *tab = nullptr;
        NRB_CUDA(tmp_alloc(&tab, ((size_t)f.nx + f.ny + f.nz) * sizeof(AxisEntry), st));
        const int longest = std::max(f.nx, std::max(f.ny, f.nz));
        k_axis_table<<<dim3((longest + 127) / 128, 3), 128, 0, st>>>(f, gijk, tab, update ? minmax : nullptr);
        NRB_LAUNCHED("k_axis_table");
        const dim3 grid((f.nx + 31) / 32, std::min((f.ny + 7) / 8, 65535), std::min((f.nz + kFlowVox - 1) / kFlowVox, 65535));
        auto kernel = update ? k_velocity_flow_table<true> : k_velocity_flow_table<false>;
        kernel<<<grid, dim3(32, 8), 0, st>>>(vel, gd[0], gd[1], gd[2], gxyz, f, tab, first, scale, minmax);
        NRB_LAUNCHED("k_velocity_flow_table");
        NRB_CUDA(cudaFreeAsync(tab, st));
    } else {
        if (update) {
            k_minmax_init<<<1, 1, 0, st>>>(minmax);
            NRB_LAUNCHED("k_minmax_init");
        }
        auto kernel = update ? k_velocity_flow<true> : k_velocity_flow<false>;
        kernel<<<blocks_for(n), 256, 0, st>>>(vel, gd[0], gd[1], gd[2], gxyz, gijk, f, first, scale, minmax);
        NRB_LAUNCHED("k_velocity_flow");
    }
    if (update) {
        unsigned mm[2];
        NRB_TRY(read_back(mm, minmax, sizeof(mm), st));
        N = velocity_squaring_steps(fkey_inv(mm[0]), fkey_inv(mm[1]));
        *steps = N;
        // scaled into the buffer an even or odd chain starts from (another one when the parity of N
        // changed)
        float *want = fields ? first : (N % 2 == 0 ? ping.p : scratch);
        const dim3 grid((f.nx + 63) / 64, std::min((f.ny + 3) / 4, 65535), std::min(f.nz, 65535));
        k_flow_scale<<<grid, 256, 0, st>>>(first, want, std::ldexp(1.f, -N), f);
        NRB_LAUNCHED("k_flow_scale");
        first = want;
    }
    auto squaring = [&](const float *in, float *out, bool planar) -> nrb_status {
        KernelTimer kt(TK_F2_COMPOSE, kSquaringBytes * n, st);
        if (small_field(n)) {
            if (planar) k_compose<true, false, int><<<blocks_for(n), 256, 0, st>>>(in, in, out, f);
            else k_compose<true, true, int><<<blocks_for(n), 256, 0, st>>>(in, in, out, f);
        } else {
            if (planar) k_compose<true, false, long long><<<blocks_for(n), 256, 0, st>>>(in, in, out, f);
            else k_compose<true, true, long long><<<blocks_for(n), 256, 0, st>>>(in, in, out, f);
        }
        NRB_LAUNCHED("k_compose");
        return NRB_OK;
    };
    if (fields) {
        // keep every intermediate field; the last squaring only when def is wanted
        for (int k = 1; k < N; ++k) NRB_TRY(squaring(fields + (k - 1) * fs, fields + k * fs, false));
        return def ? squaring(fields + (N - 1) * fs, def, true) : NRB_OK;
    }
    float *a = first, *b = first == ping.p ? scratch : ping.p;
    for (int k = 0; k < N; ++k) {
        NRB_TRY(squaring(a, k == N - 1 ? def : b, k == N - 1));
        std::swap(a, b);
    }
    return NRB_OK;  // the last squaring read scratch and wrote def
}

nrb_status compose_fields(const int32_t dim[3], const float xyz[16], const float ijk[16], const float *apply,
                          float *update, cudaStream_t st) {
    const FieldGeom f = field_geom(dim, xyz, ijk);
    KernelTimer kt(TK_F2_COMPOSE, kComposeBytes * nvox(dim), st);
    if (small_field(nvox(dim))) k_compose<false, false, int><<<blocks_for(nvox(dim)), 256, 0, st>>>(apply, update, update, f);
    else k_compose<false, false, long long><<<blocks_for(nvox(dim)), 256, 0, st>>>(apply, update, update, f);
    NRB_LAUNCHED("k_compose");
    return NRB_OK;
}

// nifti_mat33_polar's role (the orthogonal factor of a 3x3 matrix) by Higham's scaled Newton
// iteration, in double
static void polar_factor(const double A[3][3], double Q[3][3]) {
    double X[3][3];
    memcpy(X, A, sizeof(X));
    for (int it = 0; it < 100; ++it) {
        const double det = X[0][0] * (X[1][1] * X[2][2] - X[1][2] * X[2][1]) -
                           X[0][1] * (X[1][0] * X[2][2] - X[1][2] * X[2][0]) +
                           X[0][2] * (X[1][0] * X[2][1] - X[1][1] * X[2][0]);
        if (det == 0.0) break;
        double Y[3][3];  // inverse transpose
        Y[0][0] = (X[1][1] * X[2][2] - X[1][2] * X[2][1]) / det;
        Y[0][1] = (X[1][2] * X[2][0] - X[1][0] * X[2][2]) / det;
        Y[0][2] = (X[1][0] * X[2][1] - X[1][1] * X[2][0]) / det;
        Y[1][0] = (X[0][2] * X[2][1] - X[0][1] * X[2][2]) / det;
        Y[1][1] = (X[0][0] * X[2][2] - X[0][2] * X[2][0]) / det;
        Y[1][2] = (X[0][1] * X[2][0] - X[0][0] * X[2][1]) / det;
        Y[2][0] = (X[0][1] * X[1][2] - X[0][2] * X[1][1]) / det;
        Y[2][1] = (X[0][2] * X[1][0] - X[0][0] * X[1][2]) / det;
        Y[2][2] = (X[0][0] * X[1][1] - X[0][1] * X[1][0]) / det;
        double nx = 0, ny = 0;
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) {
                nx += X[r][c] * X[r][c];
                ny += Y[r][c] * Y[r][c];
            }
        const double gam = std::sqrt(std::sqrt(ny / nx));
        double d = 0;
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) {
                const double v = 0.5 * (gam * X[r][c] + Y[r][c] / gam);
                d += std::fabs(v - X[r][c]);
                X[r][c] = v;
            }
        if (d < 1e-15) break;
    }
    memcpy(Q, X, sizeof(X));
}

// reg_getRealImageSpacing (reg-lib/cpu/_reg_tools.cpp:253-273): the distance in mm between voxel
// 0 and its neighbour along each axis, through Mat44Mul (double, rounded to float)
static void real_spacing(const float xyz[16], float sp[3]) {
    float o[3];
    for (int r = 0; r < 3; ++r) o[r] = (float)((double)xyz[4 * r + 3]);
    for (int c = 0; c < 3; ++c) {
        float p[3];
        for (int r = 0; r < 3; ++r) p[r] = (float)((double)xyz[4 * r + c] + (double)xyz[4 * r + 3]);
        const float a = o[0] - p[0], b = o[1] - p[1], d = o[2] - p[2];
        sp[c] = std::sqrt(a * a + b * b + d * d);
    }
}

// Compute::ExponentiateGradient (reg-lib/Compute.cpp:288-330) for the voxel-based gradient
// `vgrad` on g->ref_* and the opposite transformation's velocity grid g->cpp_*: the intermediate
// fields of that grid (N squarings), then N gradient resampling steps, then the division by 2^N.
// fields: fields_n floats, of which N * velocity_field_stride(nvox) are used (refused when there are
// fewer), scratch: 3 * nvox floats, both 8-byte aligned.
nrb_status exponentiate_gradient(const nrb_geometry *g, const float *vel_other, int steps, float *vgrad,
                                 float *fields, int64_t fields_n, float *scratch, unsigned *minmax, cudaStream_t st) {
    if (steps < 1) return fail(NRB_ERR_INVALID, "gradient exponentiation: the squaring number must be >= 1");
    if (steps * velocity_field_stride(nvox(g->ref_dim)) > fields_n)
        return fail(NRB_ERR_INVALID, "gradient exponentiation: the intermediate fields exceed their buffer");
    KernelTimer stage(TK_F2_GRADIENT_EXP, 0.0, st);
    int N = steps;
    NRB_TRY(velocity_to_deformation(g, vel_other, false, &N, nullptr, fields, scratch, minmax, st));
    const FieldGeom f = field_geom(g->ref_dim, g->ref_xyz, g->ref_ijk);
    const long long n = nvox(g->ref_dim);
    // reorient = inverse(polar(rotation-scaling part of voxel -> mm))
    double A[3][3], Q[3][3];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) A[r][c] = g->ref_xyz[4 * r + c];
    polar_factor(A, Q);
    Mat33f R;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) R.m[3 * r + c] = (float)Q[c][r];  // inverse of an orthogonal matrix
    float sp[3];
    real_spacing(g->ref_xyz, sp);
    int exponent, unit = 1;
    for (int i = 0; i < 3; ++i) unit = unit && std::frexp(sp[i], &exponent) == 0.5f && sp[i] > 1e-3f && sp[i] < 1e3f;
    if (unit)
        for (int i = 0; i < 3; ++i) sp[i] = 1.f / sp[i];
    PairBuffer ping(st);
    NRB_TRY(ping.set(vgrad, n));
    const int64_t fs = velocity_field_stride(n);
    // vgrad -> scratch -> ping (vgrad's memory when aligned) -> scratch ... ; the last step of an
    // even chain writes vgrad itself
    float *a = vgrad, *b = scratch;
    for (int k = 0; k < N; ++k) {
        const float scale = k == N - 1 ? std::ldexp(1.f, -N) : 1.f;
        // the caller's gradient goes in and comes out planar
        const bool in_pairs = k > 0, out_pairs = k < N - 1;
        auto step = [&](auto kernel) {
            kernel<<<blocks_for(n), 256, 0, st>>>(a, fields + k * fs, b, f, R, sp[0], sp[1], sp[2], unit, scale);
        };
        if (small_field(n)) {
            if (in_pairs) out_pairs ? step(k_gradient_exp_step<true, true, int>) : step(k_gradient_exp_step<true, false, int>);
            else out_pairs ? step(k_gradient_exp_step<false, true, int>) : step(k_gradient_exp_step<false, false, int>);
        } else {
            if (in_pairs) out_pairs ? step(k_gradient_exp_step<true, true, long long>) : step(k_gradient_exp_step<true, false, long long>);
            else out_pairs ? step(k_gradient_exp_step<false, true, long long>) : step(k_gradient_exp_step<false, false, long long>);
        }
        NRB_LAUNCHED("k_gradient_exp_step");
        a = b;
        b = a == scratch ? (k + 2 == N ? vgrad : ping.p) : scratch;
    }
    if (a != vgrad) NRB_CUDA(cudaMemcpyAsync(vgrad, a, 3 * n * sizeof(float), cudaMemcpyDeviceToDevice, st));
    return NRB_OK;
}

// The voxel -> node step for a grid not aligned with the image (the F3D2 grids of rotated
// images): `vox` holds the voxel gradient already convolved along the image axes.
nrb_status voxel_to_node_general(const float *vox, const nrb_geometry *g, float weight, float *node,
                                 cudaStream_t st) {
    float T[16];
    for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c) {
            double acc = 0;
            for (int k = 0; k < 4; ++k) acc += (double)g->ref_ijk[4 * r + k] * (double)g->cpp_xyz[4 * k + c];
            T[4 * r + c] = (float)acc;  // mat44 product, each entry rounded to float
        }
    for (int r = 0; r < 3; ++r) {
        const float a = g->cpp_xyz[4 * r], b = g->cpp_xyz[4 * r + 1], c = g->cpp_xyz[4 * r + 2];
        float ratio = std::sqrt(a * a + b * b + c * c);
        ratio = ratio / g->ref_pixdim[r];
        weight = weight * ratio;
    }
    Mat33f R;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) R.m[3 * r + c] = g->flo_ijk[4 * r + c];
    const long long nc = nvox(g->cpp_dim);
    k_voxel_to_node_general<<<blocks_for(nc), 256, 0, st>>>(vox, g->ref_dim[0], g->ref_dim[1], g->ref_dim[2],
                                                           to_mat34(T), R, weight, g->cpp_dim[0], g->cpp_dim[1],
                                                           g->cpp_dim[2], node);
    NRB_LAUNCHED("k_voxel_to_node_general");
    return NRB_OK;
}

nrb_status symmetrise_velocity(const int32_t cdim[3], const float fw_xyz[16], float *fw, const float bw_xyz[16],
                               float *bw, cudaStream_t st) {
    k_symmetrise<<<blocks_for(nvox(cdim)), 256, 0, st>>>(fw, bw, cdim[0], cdim[1], cdim[2], to_mat34(fw_xyz),
                                                         to_mat34(bw_xyz));
    NRB_LAUNCHED("k_symmetrise");
    return NRB_OK;
}

}  // namespace nrb

using namespace nrb;

static nrb_status check_field_geometry(const nrb_geometry *g, const char *what) {
    for (int i = 0; i < 3; ++i)
        if (g->ref_dim[i] < 1 || g->cpp_dim[i] < 1) return fail(NRB_ERR_INVALID, std::string(what) + ": empty grid");
    if (nvox(g->ref_dim) >= (1LL << 40) || nvox(g->cpp_dim) >= (1LL << 40))
        return fail(NRB_ERR_UNSUPPORTED, std::string(what) + ": grid too large");
    return NRB_OK;
}

// Scratch buffers of one call, `call_bytes` in all. From the library's pool and freed in stream order on
// any stream (the default stream's cudaMalloc and cudaFree cost 1.3 ms of a 2.6 ms call at
// 182x218x182). On the default stream a call that needs more than the pool keeps mapped allocates
// plainly: the pool would map and unmap the rest around every call (a gradient of 160x192x160
// through seven squarings, 470 MB: 21 ms against 4.3).
struct Scratch {
    float *p = nullptr;
    unsigned *mm = nullptr;
    cudaStream_t st;
    const bool plain;
    Scratch(cudaStream_t s, size_t call_bytes): st(s), plain(!s && call_bytes > kLibPoolFloor) {}
    template <typename T>
    nrb_status alloc(T **out, size_t bytes) {
        NRB_CUDA(plain ? dev_alloc(out, bytes, nullptr) : tmp_alloc(out, bytes, st));
        return NRB_OK;
    }
    void give_back(void *q) {
        if (plain) dev_free(q, nullptr);
        else if (q) cudaFreeAsync(q, st);
    }
    ~Scratch() {
        give_back(p);
        give_back(mm);
    }
};

extern "C" nrb_status nrb_get_def_field_from_velocity_grid(const nrb_geometry *g, const float *vel,
                                                          int update_step_number, int32_t *steps, float *def,
                                                          void *stream) {
    if (!g || !vel || !steps || !def) return fail(NRB_ERR_INVALID, "nrb_get_def_field_from_velocity_grid: null pointer");
    NRB_TRY(check_field_geometry(g, "nrb_get_def_field_from_velocity_grid"));
    if (*steps < 1 && !update_step_number)
        return fail(NRB_ERR_INVALID, "nrb_get_def_field_from_velocity_grid: the squaring number must be >= 1");
    cudaStream_t st = as_stream(stream);
    const size_t field = 3 * nvox(g->ref_dim) * sizeof(float);
    Scratch s(st, field);
    NRB_TRY(s.alloc(&s.p, field));
    NRB_TRY(s.alloc(&s.mm, 2 * sizeof(unsigned)));
    int N = *steps < 1 ? 6 : *steps;
    NRB_TRY(velocity_to_deformation(g, vel, update_step_number != 0 || *steps == 0, &N, def, nullptr, s.p, s.mm, st));
    *steps = N;
    return NRB_OK;
}

extern "C" nrb_status nrb_def_field_compose(const int32_t dim[3], const float xyz[16], const float ijk[16],
                                           const float *apply, float *update, void *stream) {
    if (!dim || !xyz || !ijk || !apply || !update) return fail(NRB_ERR_INVALID, "nrb_def_field_compose: null pointer");
    if (apply == update) return fail(NRB_ERR_INVALID, "nrb_def_field_compose: the two fields must not alias");
    for (int i = 0; i < 3; ++i)
        if (dim[i] < 1) return fail(NRB_ERR_INVALID, "nrb_def_field_compose: empty field");
    return compose_fields(dim, xyz, ijk, apply, update, as_stream(stream));
}

extern "C" nrb_status nrb_exponentiate_gradient(const nrb_geometry *g, const float *vel_other, int32_t steps,
                                               float *vgrad, void *stream) {
    if (!g || !vel_other || !vgrad) return fail(NRB_ERR_INVALID, "nrb_exponentiate_gradient: null pointer");
    NRB_TRY(check_field_geometry(g, "nrb_exponentiate_gradient"));
    for (int i = 0; i < 3; ++i)  // the Jacobian's finite differences need two voxels per axis
        if (g->ref_dim[i] < 2) return fail(NRB_ERR_INVALID, "nrb_exponentiate_gradient: 3D fields of >= 2 voxels per axis");
    if (steps < 1 || steps > 30) return fail(NRB_ERR_INVALID, "nrb_exponentiate_gradient: squaring number in [1, 30]");
    cudaStream_t st = as_stream(stream);
    const long long n = nvox(g->ref_dim);
    const int64_t fields_n = steps * velocity_field_stride(n);
    const size_t field = 3 * n * sizeof(float), all = field + fields_n * sizeof(float);
    Scratch s(st, all), fields(st, all);
    NRB_TRY(s.alloc(&s.p, field));
    NRB_TRY(s.alloc(&s.mm, 2 * sizeof(unsigned)));
    NRB_TRY(fields.alloc(&fields.p, fields_n * sizeof(float)));
    return exponentiate_gradient(g, vel_other, steps, vgrad, fields.p, fields_n, s.p, s.mm, st);
}

extern "C" nrb_status nrb_symmetrise_velocity_fields(const nrb_geometry *g_fw, float *fw, const nrb_geometry *g_bw,
                                                    float *bw, void *stream) {
    if (!g_fw || !fw || !g_bw || !bw) return fail(NRB_ERR_INVALID, "nrb_symmetrise_velocity_fields: null pointer");
    for (int i = 0; i < 3; ++i)
        if (g_fw->cpp_dim[i] != g_bw->cpp_dim[i] || g_fw->cpp_dim[i] < 1)
            return fail(NRB_ERR_INVALID, "nrb_symmetrise_velocity_fields: the two grids must have the same dims");
    if (fw == bw) return fail(NRB_ERR_INVALID, "nrb_symmetrise_velocity_fields: the two grids must not alias");
    return symmetrise_velocity(g_fw->cpp_dim, g_fw->cpp_xyz, fw, g_bw->cpp_xyz, bw, as_stream(stream));
}
