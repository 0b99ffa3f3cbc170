// Node-grid and reduction kernels of the F3D gradient path, the voxel->node convolution, the
// image pyramid and the workspace that sizes their scratch buffers.
//
// Every reduction writes a fixed number of per-block partials and combines them in a fixed
// order, so each result is identical from run to run whatever the device's SM count.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include <cuda_pipeline.h>

#include "nrb_state.cuh"

namespace nrb {

// ---------------------------------------------------------------------------------------------
// bending energy
// ---------------------------------------------------------------------------------------------
// Second-derivative stencils at the nodes in the 27-point (c, b, a) order of
// set_second_order_bspline_basis_values (reg-lib/cpu/_reg_splineBasis.cpp:291-455). The
// reference tabulates the exact values rounded to 6 decimals; the same rounding is applied
// here to B(+-1) = 1/6, B(0) = 2/3, B'(+-1) = +-1/2, B'(0) = 0, B''(+-1) = 1, B''(0) = -2.
static BeBasis make_be_basis() {
    const double B[3] = { 1.0 / 6.0, 2.0 / 3.0, 1.0 / 6.0 };
    const double D[3] = { -0.5, 0.0, 0.5 };
    const double S[3] = { 1.0, -2.0, 1.0 };
    auto r6 = [](double x) { return (float)(std::round(x * 1e6) / 1e6); };
    BeBasis b;
    int i = 0;
    for (int c = 0; c < 3; ++c)
        for (int bb = 0; bb < 3; ++bb)
            for (int a = 0; a < 3; ++a, ++i) {
                b.v[0][i] = r6(S[a] * B[bb] * B[c]);
                b.v[1][i] = r6(B[a] * S[bb] * B[c]);
                b.v[2][i] = r6(B[a] * B[bb] * S[c]);
                b.v[3][i] = r6(D[a] * D[bb] * B[c]);
                b.v[4][i] = r6(B[a] * D[bb] * D[c]);
                b.v[5][i] = r6(D[a] * B[bb] * D[c]);
            }
    return b;
}

static const BeBasis& be_basis() {
    static const BeBasis b = make_be_basis();
    return b;
}

__device__ double block_sum_d(double v, double *red) {
    const int tid = threadIdx.x;
    red[tid] = v;
    __syncthreads();
    for (int s = NRB_RED_THREADS / 2; s > 0; s >>= 1) {
        if (tid < s) red[tid] += red[tid + s];
        __syncthreads();
    }
    return red[0];
}

// reg_spline_approxBendingEnergyValue3D (reg-lib/cpu/_reg_localTrans_regul.cpp:72-153): per
// interior node the 6 second derivatives of each component from 27-point stencils of the
// positions, summed squares (cross terms doubled) accumulated in double. The stencil sums use
// the reference's order without contraction: each node's terms are bit-identical to the CPU's.
// grad/step (optional): the positions are the line search's trial values cpp - cur_len * grad
//
// Three threads per node, one per component (threads k * NRB_RED_THREADS + j of a block), so 27
// loads per thread are in flight and three times as many warps hide their latency. Node lane j
// (component 0) adds the other components' terms in the reference's order and accumulates its
// nodes in the grid-stride order of a one-thread-per-node loop; the block sum is the same tree
// as block_sum_d over the NRB_RED_THREADS node lanes, so every partial is unchanged bit for bit.
__global__ void __launch_bounds__(3 * NRB_RED_THREADS, 2)
k_be_value(int cx, int cy, int cz, const float *__restrict__ cpp, BeBasis B,
           double *__restrict__ partials, const float *__restrict__ grad, const OptState *__restrict__ step) {
    __shared__ double red[NRB_RED_THREADS];
    __shared__ BeTerms other[2][NRB_RED_THREADS];  // components 1 and 2 of the lane's node
    const float scale = grad ? -step->cur_len : 0.f;
    const int j = threadIdx.x % NRB_RED_THREADS, k = threadIdx.x / NRB_RED_THREADS;
    const int ix = cx - 2, iy = cy - 2, iz = cz - 2;
    const long long ni = (ix > 0 && iy > 0 && iz > 0) ? (long long)ix * iy * iz : 0;
    double acc = 0;
    for (long long base = blockIdx.x * (long long)NRB_RED_THREADS; base < ni; base += (long long)gridDim.x * NRB_RED_THREADS) {
        const long long n = base + j;
        BeTerms t{ 0.f, 0.f, 0.f, 0.f };
        if (n < ni) t = be_node_component<true>(cx, cy, cz, ix, iy, cpp, B, grad, scale, n, k);
        if (k > 0) other[k - 1][j] = t;
        __syncthreads();
        if (k == 0 && n < ni) {
            double s = be_add_component(0.0, t, 0);
            s = be_add_component(s, other[0][j], 1);
            acc += be_add_component(s, other[1][j], 2);
        }
        __syncthreads();  // `other` is rewritten by the next round
    }
    if (k == 0) red[j] = acc;
    __syncthreads();
    for (int s = NRB_RED_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partials[blockIdx.x] = red[0];
}

__global__ void k_be_sum(const double *__restrict__ partials, int n, double norm,
                         nrb_objective *__restrict__ obj) {
    __shared__ double red[NRB_RED_THREADS];
    double a = 0;
    for (int i = threadIdx.x; i < n; i += NRB_RED_THREADS) a += partials[i];
    const double s = block_sum_d(a, red);
    if (threadIdx.x == 0) obj->be = s / norm;
}

// Node position on the identity grid, float arithmetic in the reference's order
// (reg_getDisplacementFromDeformation_3D, reg-lib/cpu/_reg_tools.cpp:2011-2022).
__device__ __forceinline__ float identity_pos(const Mat34& M, int k, int x, int y, int z) {
    const float *m = M.m + 4 * k;
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], (float)x), __fmul_rn(m[1], (float)y)),
                               __fmul_rn(m[2], (float)z)), m[3]);
}

// reg_spline_approxBendingEnergyGradient3D (reg-lib/cpu/_reg_localTrans_regul.cpp:286-451),
// first half: the 6 derivative values of component k of node n from zero-padded stencils of the
// displacements, cross terms doubled. Layout der[(3 * t + k) * BePad::size + BePad node]: every derivative
// plane has a ring of zeros around the grid (cleared when the workspace is made and never written),
// so that the second half reads all 27 neighbours of any node without a test; a zero adds nothing.
struct BePad {
    int sy, sz;
    long long size;
    __host__ __device__ __forceinline__ BePad(int cx, int cy, int cz)
        : sy(cx + 2), sz((cx + 2) * (cy + 2)), size((long long)(cx + 2) * (cy + 2) * (cz + 2)) {}
    __device__ __forceinline__ long long node(int x, int y, int z) const { return (long long)(z + 1) * sz + (y + 1) * sy + x + 1; }
};

__device__ __forceinline__ void be_node_derivatives_k(int cx, int cy, int cz, const Mat34& M,
                                                      const float *__restrict__ cpp, const BeBasis& B,
                                                      float *__restrict__ der, long long n, int k) {
    const long long nc = (long long)cx * cy * cz;
    // node indices fit 32 bits (a grid has fewer than 2^31 / 3 nodes)
    const int i32 = (int)n, row = i32 / cx, x = i32 - row * cx, z = row / cy, y = row - z * cy;
    // row k of the grid matrix picked by selects (a runtime index into the parameter would copy
    // the matrix to local memory)
    float m[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = k == 0 ? M.m[q] : (k == 1 ? M.m[4 + q] : M.m[8 + q]);
    float d[6];
#pragma unroll
    for (int t = 0; t < 6; ++t) d[t] = 0.f;
#pragma unroll
    for (int c = -1; c < 2; ++c)
#pragma unroll
        for (int b = -1; b < 2; ++b)
#pragma unroll
            for (int a = -1; a < 2; ++a) {
                const int i = 9 * (c + 1) + 3 * (b + 1) + (a + 1);
                const int X = x + a, Y = y + b, Z = z + c;
                if (X < 0 || Y < 0 || Z < 0 || X >= cx || Y >= cy || Z >= cz) continue;
                const long long idx = ((long long)Z * cy + Y) * cx + X;
                const float id = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], (float)X), __fmul_rn(m[1], (float)Y)),
                                                     __fmul_rn(m[2], (float)Z)), m[3]);  // identity_pos
                const float v = __fsub_rn(__ldg(&cpp[k * nc + idx]), id);
#pragma unroll
                for (int t = 0; t < 6; ++t) d[t] = __fadd_rn(d[t], __fmul_rn(B.v[t][i], v));
            }
    const BePad pad(cx, cy, cz);
    float *q = der + k * pad.size + pad.node(x, y, z);
#pragma unroll
    for (int t = 0; t < 3; ++t) q[3 * t * pad.size] = d[t];
#pragma unroll
    for (int t = 3; t < 6; ++t) q[3 * t * pad.size] = (float)(2.0 * (double)d[t]);
}

// one thread per (node, component): component k = blockIdx.y
__global__ void k_be_derivatives(int cx, int cy, int cz, Mat34 M, const float *__restrict__ cpp,
                                 BeBasis B, float *__restrict__ der) {
    const long long nc = (long long)cx * cy * cz;
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < nc;
         n += (long long)gridDim.x * blockDim.x)
        be_node_derivatives_k(cx, cy, cz, M, cpp, B, der, n, (int)blockIdx.y);
}

// second half: the same stencils applied to the derivative values of the 27 neighbours,
// grad += weight / #nodes * sum, for component k of node n: the sum runs over the neighbours
// in (z, y, x) order and the 6 derivative kinds within each, as for all components at once.
__device__ __forceinline__ void be_node_accumulate_k(int cx, int cy, int cz, const float *__restrict__ der,
                                                     const BeBasis& B, float ratio, float *__restrict__ grad,
                                                     long long n, int k) {
    const long long nc = (long long)cx * cy * cz;
    // node indices fit 32 bits (a grid has fewer than 2^31 / 3 nodes)
    const int i32 = (int)n, row = i32 / cx, x = i32 - row * cx, z = row / cy, y = row - z * cy;
    const BePad pad(cx, cy, cz);
    const float *p = der + k * pad.size + pad.node(x, y, z);
    float g = 0.f;
#pragma unroll
    for (int c = -1; c < 2; ++c)
#pragma unroll
        for (int b = -1; b < 2; ++b) {
            const float *r = p + (c * pad.sz + b * pad.sy);
#pragma unroll
            for (int e = -1; e < 2; ++e) {
                const int a = 9 * (c + 1) + 3 * (b + 1) + (e + 1);
#pragma unroll
                for (int t = 0; t < 6; ++t) g = __fadd_rn(g, __fmul_rn(__ldg(r + 3 * t * pad.size + e), B.v[t][a]));
            }
        }
    grad[k * nc + n] = __fadd_rn(grad[k * nc + n], __fmul_rn(ratio, g));
}

// one thread per (node, component): component k = blockIdx.y
__global__ void k_be_accumulate(int cx, int cy, int cz, const float *__restrict__ der, BeBasis B,
                                float ratio, float *__restrict__ grad) {
    const long long nc = (long long)cx * cy * cz;
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < nc;
         n += (long long)gridDim.x * blockDim.x)
        be_node_accumulate_k(cx, cy, cz, der, B, ratio, grad, n, (int)blockIdx.y);
}

// ---------------------------------------------------------------------------------------------
// voxel -> node: cubic convolution evaluated only at the sampled voxels
// ---------------------------------------------------------------------------------------------
// Normalised convolution of one line at one sample: density = finite(value) (the reference's
// mask is all-active here), NaN at the sample itself stays NaN (_reg_tools.cpp:863-867, :1105).
template <typename Load>
__device__ __forceinline__ float conv_at(int s, int n, int R, const float *__restrict__ K, Load ld) {
    const float centre = ld(s);
    if (centre != centre) return centre;
    float num = 0.f, den = 0.f;
    const int k0 = max(0, s - R), k1 = min(n - 1, s + R);
    for (int k = k0; k <= k1; ++k) {
        const float v = ld(k);
        const float w = K[k - s + R];
        if (v == v) {
            num = fmaf(w, v, num);
            den += w;
        }
    }
    return num / den;
}

// Four consecutive sampled outputs of one line, the taps of each in ascending order and every weight
// read once for the four. ld reads 0 for the R positions beyond either end (a tap there adds
// weight * 0 and changes no sum). The sum assumes no NaN (its density is then dens[j], the in-line weights
// summed in the same order); a NaN shows in it, and that output is taken again with conv_at.
template <typename Samples, typename Load>
__device__ __forceinline__ void conv_outputs4(int n, int R, const float *w, const float *dens, Samples samples, int ns,
                                              int j0, Load ld, float out[4]) {
    const int last = min(4, ns - j0) - 1;
    int s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = samples[j0 + min(u, last)];
    float num[4] = { 0.f, 0.f, 0.f, 0.f };
    const int taps = 2 * R + 1;
    int t = 0;
    for (; t + 4 <= taps; t += 4) {
        const float4 q = *reinterpret_cast<const float4 *>(w + t);
        const float wt[4] = { q.x, q.y, q.z, q.w };
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int u = 0; u < 4; ++u) num[u] = fmaf(wt[e], ld(s[u] - R + t + e), num[u]);
    }
#pragma unroll 1
    for (; t < taps; ++t) {
        const float wt = w[t];
#pragma unroll
        for (int u = 0; u < 4; ++u) num[u] = fmaf(wt, ld(s[u] - R + t), num[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) out[u] = num[u] / dens[j0 + min(u, last)];
#pragma unroll 1
    for (int u = 0; u <= last; ++u) {
        const float v = u < 2 ? (u == 0 ? num[0] : num[1]) : (u == 2 ? num[2] : num[3]);
        if (v == v) continue;
        const float r = conv_at(samples[j0 + u], n, R, w, ld);
        if (u == 0) out[0] = r;
        else if (u == 1) out[1] = r;
        else if (u == 2) out[2] = r;
        else out[3] = r;
    }
}

// weights (16-byte aligned, padded to fours) and densities of one axis in a block's shared memory;
// ends with a barrier
__host__ __device__ inline int conv_weight_floats(int R, int ns) { return ((2 * R + 4) & ~3) + ((ns + 3) & ~3); }
template <typename Samples>
__device__ __forceinline__ void conv_weights(int n, int R, const float *__restrict__ K, Samples samples, int ns, float *w,
                                             float *&dens) {
    dens = w + ((2 * R + 4) & ~3);
    for (int i = threadIdx.x; i < 2 * R + 1; i += blockDim.x) w[i] = K[i];
    __syncthreads();
    for (int j = threadIdx.x; j < ns; j += blockDim.x) {
        const int sj = samples[j];
        const int k0 = max(0, sj - R), k1 = min(n - 1, sj + R);
        float den = 0.f;
        for (int k = k0; k <= k1; ++k) den += w[k - sj + R];
        dens[j] = den;
    }
    __syncthreads();
}

// Above 48 KB a block's shared memory, static arrays included, is opted into: the batched passes hold
// a BatchList beside their tile. The opt-in belongs to the function, not to the launch, and other
// host threads launch it too, so it is one constant and never this launch's size.
constexpr size_t CONV_STATIC_BYTES = 2048, CONV_SHARED_MAX = 227 * 1024 - CONV_STATIC_BYTES;
static_assert(sizeof(BatchList) + 128 <= CONV_STATIC_BYTES, "static shared memory of the batched convolution passes");

// Pass along x. A block takes kRows consecutive rows of one component, transposes them into shared
// memory (column stride kRows + 1: no bank conflict either way; R columns of zeros on either side),
// and each lane convolves one row; its warps share the outputs, four at a time. The outputs go out
// through shared memory as one contiguous run. 32 rows while the tile stays small enough for
// several blocks per SM; long rows take 16 or 8 (4 when the window is as long as the row, too), the
// warp's other lanes then working on other outputs of the same rows.
//
// One load and a quarter of a weight load per multiply-add, rows copied asynchronously: 182x218x182
// with a 5-voxel grid (37 samples, 21 taps) takes 55 us (37.7 M warp instructions, issue-bound); it
// took 64 us (47.6 M) when a thread stepped through the outputs of several rows with a weight, a
// value and a bounds check per tap. The y pass went from 22 to 18 us.
constexpr int CONV_X_THREADS = 128;
__host__ __device__ inline size_t conv_x_bytes(int rows, int nx, int R, int ns) {
    return 4 * ((size_t)conv_weight_floats(R, ns) + (size_t)(nx + 2 * R) * (rows + 1) + (size_t)rows * (ns | 1));
}
inline int conv_x_rows(int nx, int R, int ns) {
    for (int rows : { 32, 16 })
        if (conv_x_bytes(rows, nx, R, ns) <= 48 * 1024) return rows;
    return conv_x_bytes(8, nx, R, ns) <= CONV_SHARED_MAX ? 8 : 4;
}
__host__ __device__ inline long long conv_x_units(int rows, int ny, int nz) {
    return 3 * (((long long)ny * nz + rows - 1) / rows);
}

// unit = (component, group of rows); conv_weights has filled w and dens
template <int kRows>
__device__ __forceinline__ void conv_x_unit(int nx, int ny, int nz, const float *__restrict__ vg,
                                            const int *__restrict__ samples, int ns, int R, float *__restrict__ out,
                                            long long unit, const float *w, const float *dens, float *tile) {
    constexpr int kStride = kRows + 1, kSub = 32 / kRows, kWarps = CONV_X_THREADS / 32;
    float *res = tile + (size_t)(nx + 2 * R) * kStride;
    const int rstride = ns | 1;
    const long long nrow = (long long)ny * nz, groups = (nrow + kRows - 1) / kRows;
    const int c = (int)(unit / groups);
    const long long r0 = (unit - c * groups) * kRows;
    const int nr = (int)min((long long)kRows, nrow - r0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *body = tile + R * kStride;
    for (int r = warp; r < nr; r += kWarps) {
        const float *src = vg + (c * nrow + r0 + r) * nx;
#pragma unroll 4
        for (int x = lane; x < nx; x += 32) __pipeline_memcpy_async(body + x * kStride + r, src + x, 4);
    }
    __pipeline_commit();
    for (int i = threadIdx.x; i < R * kStride; i += CONV_X_THREADS) tile[i] = body[nx * kStride + i] = 0.f;
    __pipeline_wait_prior(0);
    __syncthreads();
    const int lrow = lane % kRows;
    const float *col = body + lrow;
    for (int q = warp * kSub + lane / kRows; 4 * q < ns; q += kWarps * kSub) {
        if (lrow >= nr) continue;
        float v[4];
        conv_outputs4(nx, R, w, dens, samples, ns, 4 * q, [&](int k) { return col[k * kStride]; }, v);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (4 * q + u < ns) res[lrow * rstride + 4 * q + u] = v[u];
    }
    __syncthreads();
    float *dst = out + (c * nrow + r0) * ns;
    for (int r = warp; r < nr; r += kWarps)
#pragma unroll 2
        for (int j = lane; j < ns; j += 32) dst[r * ns + j] = res[r * rstride + j];
}

template <int kRows>
__global__ void __launch_bounds__(CONV_X_THREADS)
k_conv_x(int nx, int ny, int nz, const float *__restrict__ vg, const int *__restrict__ samples, int ns,
         const float *__restrict__ K, int R, float *__restrict__ out) {
    extern __shared__ __align__(16) float conv_sm[];
    float *dens;
    conv_weights(nx, R, K, samples, ns, conv_sm, dens);
    conv_x_unit<kRows>(nx, ny, nz, vg, samples, ns, R, out, blockIdx.x, conv_sm, dens, conv_sm + conv_weight_floats(R, ns));
}

// Pass along y of a [3][nz][ny][inner] array: a block takes one (component, z) slice, or an even share
// of its columns, in shared memory (R rows of zeros above and below), a thread four outputs of a
// column.
constexpr int CONV_Y_THREADS = 256;
struct ConvY {
    int width, chunks;  // columns of a block, blocks of a slice
    __host__ __device__ ConvY(int ny, int inner, int R) {
        const int most = 12 * 1024 / (ny + 2 * R);
        chunks = most < 1 ? inner : (inner + most - 1) / most;
        width = (inner + chunks - 1) / chunks;
    }
};
__host__ __device__ inline size_t conv_y_bytes(int ny, int inner, int R, int ns) {
    return 4 * ((size_t)conv_weight_floats(R, ns) + (size_t)(ny + 2 * R) * ConvY(ny, inner, R).width);
}
// A block pays for its staging where it has a warp's worth of outputs and, when a thread takes more
// than one, where there is a block for every SM; other volumes go through conv_strided_element. All
// passes, with the tile and without: 182x218x182 with a 5-voxel grid 74 and 79 us, 512x512x320 with 3
// voxels 1024 and 1216; 3x4x1900 (three columns a slice) 39 and 20, 100x101x3 with 1 voxel (nine
// slices) 33 and 24. Even shares: 256x256x256 with 5 voxels 158 us, 169 with as many columns as fit.
inline bool conv_y_tile(int ny, int inner, int R, int ns, long long slices) {
    const ConvY C(ny, inner, R);
    const int quads = (ns + 3) / 4 * C.width;
    return quads >= 32 && (C.chunks == 1 || C.width >= 16) && (quads <= CONV_Y_THREADS || slices * C.chunks >= sm_count());
}

__device__ __forceinline__ void conv_y_unit(int ny, int inner, const float *__restrict__ in,
                                            const int *__restrict__ samples, int ns, int R, float *__restrict__ out,
                                            long long unit, const float *w, const float *dens, float *tile) {
    const ConvY C(ny, inner, R);
    const long long slice = unit / C.chunks;  // component * nz + z
    const int i0 = (int)(unit - slice * C.chunks) * C.width, wd = min(C.width, inner - i0);
    if (wd <= 0) return;
    const float *src = in + slice * ny * inner + i0;
    float *body = tile + R * wd;
    if (wd == inner) {
#pragma unroll 4
        for (int i = threadIdx.x; i < ny * inner; i += CONV_Y_THREADS) __pipeline_memcpy_async(body + i, src + i, 4);
    } else {
        for (int i = threadIdx.x; i < ny * wd; i += CONV_Y_THREADS) {
            const int y = i / wd;
            __pipeline_memcpy_async(body + i, src + (long long)y * inner + (i - y * wd), 4);
        }
    }
    __pipeline_commit();
    for (int i = threadIdx.x; i < R * wd; i += CONV_Y_THREADS) tile[i] = body[ny * wd + i] = 0.f;
    __pipeline_wait_prior(0);
    __syncthreads();
    float *dst = out + slice * ns * inner + i0;
    for (int e = threadIdx.x; e < (ns + 3) / 4 * wd; e += CONV_Y_THREADS) {
        const int q = e / wd, ii = e - q * wd;
        const float *col = body + ii;
        float v[4];
        conv_outputs4(ny, R, w, dens, samples, ns, 4 * q, [&](int k) { return col[k * wd]; }, v);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (4 * q + u < ns) dst[(long long)(4 * q + u) * inner + ii] = v[u];
    }
}

__global__ void __launch_bounds__(CONV_Y_THREADS)
k_conv_y(int ny, int inner, const float *__restrict__ in, const int *__restrict__ samples, int ns,
         const float *__restrict__ K, int R, float *__restrict__ out) {
    extern __shared__ __align__(16) float conv_sm[];
    float *dens;
    conv_weights(ny, R, K, samples, ns, conv_sm, dens);
    conv_y_unit(ny, inner, in, samples, ns, R, out, blockIdx.x, conv_sm, dens, conv_sm + conv_weight_floats(R, ns));
}

// Pass along the middle axis of an [outer][len][inner] array, one output per thread, element =
// (outer, sample, column): reads are coalesced over the columns and shared by a column's samples in
// L1. The z pass (its array is small, y and x being sampled: four outputs per thread left too few
// warps and staged weights cost more than they saved, 14 and 12 us against 9), and the y pass of
// the volumes that conv_y_tile leaves.
__device__ __forceinline__ void conv_strided_element(int len, int inner, const float *__restrict__ in,
                                                     const int *__restrict__ samples, int ns,
                                                     const float *__restrict__ K, int R, float *__restrict__ out,
                                                     long long e) {
    const int i32 = (int)e, rest = i32 / inner, ii = i32 - rest * inner;  // < 3 x voxels, below 2^31
    const int c = rest / ns, s = __ldg(&samples[rest - c * ns]);
    const float *col = in + (long long)c * len * inner + ii;
    const int k0 = max(0, s - R), k1 = min(len - 1, s + R);
    const float *p = col + (long long)k0 * inner, *q = K + (k0 - s + R);
    float num = 0.f, den = 0.f;
#pragma unroll 8
    for (int k = k0; k <= k1; ++k, p += inner, ++q) {
        const float w = __ldg(q);
        num = fmaf(w, __ldg(p), num);
        den += w;
    }
    float v = num / den;
    if (num != num) v = conv_at(s, len, R, K, [&](int k) { return __ldg(col + (long long)k * inner); });
    out[e] = v;
}

__global__ void __launch_bounds__(256)
k_conv_strided(long long elements, int len, int inner, const float *__restrict__ in, const int *__restrict__ samples, int ns,
               const float *__restrict__ K, int R, float *__restrict__ out) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e < elements) conv_strided_element(len, inner, in, samples, ns, K, R, out, e);
}

// reg_voxelCentricToNodeCentric (reg-lib/cpu/_reg_localTrans.cpp:1616-1683): trilinear sample
// of the convolved gradient (taps outside the volume skipped), reorientation by the transpose
// of the floating ijk 3x3, weighting; overwrites the node gradient.
__device__ __forceinline__ void node_at(int cx, int cy, int cz, int nsx, int nsy, int nsz,
                                        const float *__restrict__ conv, const int *__restrict__ tsx,
                                        const float *__restrict__ wsx, const int *__restrict__ tsy,
                                        const float *__restrict__ wsy, const int *__restrict__ tsz,
                                        const float *__restrict__ wsz, const Mat34& R, float weight,
                                        float *__restrict__ node, long long n) {
    const long long nc = (long long)cx * cy * cz;
    const long long cs = (long long)nsz * nsy * nsx;
    {
        const int x = (int)(n % cx);
        const int y = (int)((n / cx) % cy);
        const int z = (int)(n / ((long long)cx * cy));
        float iv[3] = { 0.f, 0.f, 0.f };
        for (int c = 0; c < 2; ++c) {
            const int sz = tsz[2 * z + c];
            if (sz < 0) continue;
            const float wz = wsz[2 * z + c];
            for (int b = 0; b < 2; ++b) {
                const int sy = tsy[2 * y + b];
                if (sy < 0) continue;
                const float wy = wsy[2 * y + b];
                for (int a = 0; a < 2; ++a) {
                    const int sx = tsx[2 * x + a];
                    if (sx < 0) continue;
                    const float lw = __fmul_rn(__fmul_rn(wsx[2 * x + a], wy), wz);
                    const long long idx = ((long long)sz * nsy + sy) * nsx + sx;
                    iv[0] = fmaf(lw, conv[idx], iv[0]);
                    iv[1] = fmaf(lw, conv[cs + idx], iv[1]);
                    iv[2] = fmaf(lw, conv[2 * cs + idx], iv[2]);
                }
            }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float ro = R.m[0 * 4 + d] * iv[0] + R.m[1 * 4 + d] * iv[1] + R.m[2 * 4 + d] * iv[2];
            node[d * nc + n] = ro * weight;
        }
    }
}

__global__ void k_nodes(int cx, int cy, int cz, int nsx, int nsy, int nsz,
                        const float *__restrict__ conv, const int *__restrict__ tsx,
                        const float *__restrict__ wsx, const int *__restrict__ tsy,
                        const float *__restrict__ wsy, const int *__restrict__ tsz,
                        const float *__restrict__ wsz, Mat34 R, float weight,
                        float *__restrict__ node) {
    const long long nc = (long long)cx * cy * cz;
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < nc;
         n += (long long)gridDim.x * blockDim.x)
        node_at(cx, cy, cz, nsx, nsy, nsz, conv, tsx, wsx, tsy, wsy, tsz, wsz, R, weight, node, n);
}

// ---------------------------------------------------------------------------------------------
// batched levels: the node-grid and node-convolution stages of every pair that needs them, with
// each pair's elements computed exactly as the plain kernels compute them
// ---------------------------------------------------------------------------------------------
// bending-energy value partials of every pair in INIT or LINE: work unit = one block of the plain
// k_be_value (same node range, three threads per node, same shared-memory tree), persistent
// blocks of 3 * NRB_RED_THREADS
__global__ void __launch_bounds__(3 * NRB_RED_THREADS, 2)
k_b_be_value(const BatchPair *__restrict__ pairs, const OptState *__restrict__ states, int npairs, BeBasis B) {
    __shared__ BatchList L;
    __shared__ double red[NRB_RED_THREADS];
    __shared__ BeTerms other[2][NRB_RED_THREADS];
    const int j = threadIdx.x % NRB_RED_THREADS, kc = threadIdx.x / NRB_RED_THREADS;
    batch_list_build(states, npairs, (1u << PH_INIT) | (1u << PH_LINE),
                     [&](int q, int& u, int& w) {
                         const BatchPair& b = pairs[q];
                         u = b.be_w > 0 ? b.n_be : 0;
                         w = 1;
                     }, L);
    int k = 0;
    for (long long u = blockIdx.x; u < L.total; u += gridDim.x) {
        while (L.pref[k + 1] <= u) ++k;
        const int p = L.pair[k], v = (int)(u - L.pref[k]);
        const BatchPair& P = pairs[p];
        const bool line = states[p].phase == PH_LINE;
        const float *grad = line ? P.grad : nullptr;
        const float scale = line ? -states[p].cur_len : 0.f;
        const int cx = P.cdim[0], cy = P.cdim[1], cz = P.cdim[2];
        const int ix = cx - 2, iy = cy - 2, iz = cz - 2;
        const long long ni = (ix > 0 && iy > 0 && iz > 0) ? (long long)ix * iy * iz : 0;
        double acc = 0;
        // the unit's bounds are the same for every thread of the block (one pair per unit)
        for (long long base = (long long)v * NRB_RED_THREADS; base < ni; base += (long long)P.n_be * NRB_RED_THREADS) {
            const long long n = base + j;
            BeTerms t{ 0.f, 0.f, 0.f, 0.f };
            if (n < ni) t = be_node_component<true>(cx, cy, cz, ix, iy, P.best, B, grad, scale, n, kc);
            if (kc > 0) other[kc - 1][j] = t;
            __syncthreads();
            if (kc == 0 && n < ni) {
                double s = be_add_component(0.0, t, 0);
                s = be_add_component(s, other[0][j], 1);
                acc += be_add_component(s, other[1][j], 2);
            }
            __syncthreads();
        }
        if (kc == 0) red[j] = acc;
        __syncthreads();
        for (int s = NRB_RED_THREADS / 2; s > 0; s >>= 1) {
            if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
            __syncthreads();
        }
        if (threadIdx.x == 0) P.be_partials[v] = red[0];
        __syncthreads();  // red is reused by the next unit
    }
}

__global__ void k_b_be_derivatives(const BatchPair *__restrict__ pairs, const OptState *__restrict__ states,
                                   int npairs, BeBasis B) {
    __shared__ BatchList L;
    batch_list_build(states, npairs, 1u << PH_GRAD,
                     [&](int q, int& u, int& w) {
                         const BatchPair& b = pairs[q];
                         u = b.be_w > 0 ? (int)(3 * b.nnode) : 0;  // one element per (component, node)
                         w = 1;
                     }, L);
    batch_elements(L, [&](int p, long long e) {
        const BatchPair& P = pairs[p];
        const int k = (int)(e / P.nnode);
        const long long n = e - k * P.nnode;
        be_node_derivatives_k(P.cdim[0], P.cdim[1], P.cdim[2], P.grid_xyz, P.best, B, P.be_der, n, k);
    });
}

__global__ void k_b_be_accumulate(const BatchPair *__restrict__ pairs, const OptState *__restrict__ states,
                                  int npairs, BeBasis B) {
    __shared__ BatchList L;
    batch_list_build(states, npairs, 1u << PH_GRAD,
                     [&](int q, int& u, int& w) {
                         const BatchPair& b = pairs[q];
                         u = b.be_w > 0 ? (int)(3 * b.nnode) : 0;  // one element per (component, node)
                         w = 1;
                     }, L);
    batch_elements(L, [&](int p, long long e) {
        const BatchPair& P = pairs[p];
        const int k = (int)(e / P.nnode);
        const long long n = e - k * P.nnode;
        be_node_accumulate_k(P.cdim[0], P.cdim[1], P.cdim[2], P.be_der, B, P.be_ratio, P.grad, n, k);
    });
}

// Passes of the node convolution: work unit = one block of the plain k_conv_x and k_conv_y; or one
// element. A block fills its weights when it comes to a pair's first unit.
template <int kRows>
__global__ void __launch_bounds__(CONV_X_THREADS)
k_b_conv_x(const BatchPair *__restrict__ pairs, const OptState *__restrict__ states, int npairs) {
    extern __shared__ __align__(16) float conv_sm[];
    __shared__ BatchList L;
    batch_list_build(states, npairs, 1u << PH_GRAD,
                     [&](int q, int& u, int& w) {
                         const BatchPair& b = pairs[q];
                         u = (int)conv_x_units(kRows, b.rdim[1], b.rdim[2]);
                         w = 1;
                     }, L);
    int k = 0, have = -1;
    float *dens = nullptr;
    for (long long u = blockIdx.x; u < L.total; u += gridDim.x) {
        while (L.pref[k + 1] <= u) ++k;
        const BatchPair& P = pairs[L.pair[k]];
        if (have != k) {
            conv_weights(P.rdim[0], P.radius[0], P.kernel[0], P.samples[0], P.ns[0], conv_sm, dens);
            have = k;
        }
        conv_x_unit<kRows>(P.rdim[0], P.rdim[1], P.rdim[2], P.vgrad, P.samples[0], P.ns[0], P.radius[0], P.conv1,
                           u - L.pref[k], conv_sm, dens, conv_sm + conv_weight_floats(P.radius[0], P.ns[0]));
        __syncthreads();  // the tile is reused by the next unit
    }
}

__global__ void __launch_bounds__(CONV_Y_THREADS)
k_b_conv_y(const BatchPair *__restrict__ pairs, const OptState *__restrict__ states, int npairs) {
    extern __shared__ __align__(16) float conv_sm[];
    __shared__ BatchList L;
    batch_list_build(states, npairs, 1u << PH_GRAD,
                     [&](int q, int& u, int& w) {
                         const BatchPair& b = pairs[q];
                         u = 3 * b.rdim[2] * ConvY(b.rdim[1], b.ns[0], b.radius[1]).chunks;
                         w = 1;
                     }, L);
    int k = 0, have = -1;
    float *dens = nullptr;
    for (long long u = blockIdx.x; u < L.total; u += gridDim.x) {
        while (L.pref[k + 1] <= u) ++k;
        const BatchPair& P = pairs[L.pair[k]];
        if (have != k) {
            conv_weights(P.rdim[1], P.radius[1], P.kernel[1], P.samples[1], P.ns[1], conv_sm, dens);
            have = k;
        }
        conv_y_unit(P.rdim[1], P.ns[0], P.conv1, P.samples[1], P.ns[1], P.radius[1], P.conv2, u - L.pref[k], conv_sm, dens,
                    conv_sm + conv_weight_floats(P.radius[1], P.ns[1]));
        __syncthreads();
    }
}

// along y (kAxis 1) or z (kAxis 2), element-wise
template <int kAxis>
__global__ void k_b_conv_strided(const BatchPair *__restrict__ pairs, const OptState *__restrict__ states, int npairs) {
    __shared__ BatchList L;
    batch_list_build(states, npairs, 1u << PH_GRAD,
                     [&](int q, int& u, int& w) {
                         const BatchPair& b = pairs[q];
                         u = 3 * (kAxis == 1 ? b.rdim[2] : b.ns[2]) * b.ns[1] * b.ns[0];
                         w = 1;
                     }, L);
    batch_elements(L, [&](int p, long long e) {
        const BatchPair& P = pairs[p];
        if (kAxis == 1)
            conv_strided_element(P.rdim[1], P.ns[0], P.conv1, P.samples[1], P.ns[1], P.kernel[1], P.radius[1], P.conv2, e);
        else
            conv_strided_element(P.rdim[2], P.ns[1] * P.ns[0], P.conv2, P.samples[2], P.ns[2], P.kernel[2], P.radius[2],
                                 P.conv1, e);
    });
}

// node sampling, reorientation and weighting (overwrites the node gradient)
__global__ void k_b_nodes(const BatchPair *__restrict__ pairs, const OptState *__restrict__ states, int npairs) {
    __shared__ BatchList L;
    batch_list_build(states, npairs, 1u << PH_GRAD,
                     [&](int q, int& u, int& w) {
                         const BatchPair& b = pairs[q];
                         u = (int)b.nnode;
                         w = 1;
                     }, L);
    batch_elements(L, [&](int p, long long n) {
        const BatchPair& P = pairs[p];
        node_at(P.cdim[0], P.cdim[1], P.cdim[2], P.ns[0], P.ns[1], P.ns[2], P.conv1, P.tap_slot[0], P.tap_weight[0],
                P.tap_slot[1], P.tap_weight[1], P.tap_slot[2], P.tap_weight[2], P.flo_ijk, P.node_weight, P.grad, n);
    });
}

// ---------------------------------------------------------------------------------------------
// full-volume one-axis normalised convolution (value, density) pairs
// ---------------------------------------------------------------------------------------------
// din == nullptr: density = finite(vin) and NaN values count as 0 (first axis of a call).
__global__ void k_conv_axis(int nx, int ny, int nz, int axis, const float *__restrict__ vin,
                            const float *__restrict__ din, const float *__restrict__ K, int R,
                            float *__restrict__ vout, float *__restrict__ dout) {
    const long long nv = (long long)nx * ny * nz;
    const int n = axis == 0 ? nx : axis == 1 ? ny : nz;
    const long long stride = axis == 0 ? 1 : axis == 1 ? nx : (long long)nx * ny;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv;
         i += (long long)gridDim.x * blockDim.x) {
        const int p = axis == 0 ? (int)(i % nx) : axis == 1 ? (int)((i / nx) % ny) : (int)(i / ((long long)nx * ny));
        const long long base = i - (long long)p * stride;
        const int k0 = max(0, p - R), k1 = min(n - 1, p + R);
        float num = 0.f, den = 0.f;
        for (int k = k0; k <= k1; ++k) {
            const float w = K[k - p + R];
            float v = __ldg(&vin[base + k * stride]);
            float d;
            if (din) {
                d = __ldg(&din[base + k * stride]);
            } else {
                d = (v == v) ? 1.f : 0.f;
                if (v != v) v = 0.f;
            }
            num = fmaf(w, v, num);
            den = fmaf(w, d, den);
        }
        vout[i] = num;
        dout[i] = den;
    }
}

// The same convolution of whole lines, normalised, in place: a block holds kCols lines of one volume
// in shared memory (zeros at both ends, lines side by side so that neighbouring lanes read
// neighbouring banks), convolves them with conv_outputs4 and writes them back. Each value crosses HBM
// twice; the separate passes moved 28 bytes per voxel and read the taps, the line and its finite
// flags from global memory tap by tap (182x218x182, 21 taps: 190 us per volume and axis;
// 512x512x160 along z, 81 taps: 7.6 ms, 0.92 like this; 1024x1024x2 along y, 241 taps: 731 us, 185).
// Taps travel as a kernel argument.
struct ConvTaps {
    float k[NRB_STATIC_CONV_MAX_TAPS];
};
struct EverySample {
    __device__ __forceinline__ int operator[](int j) const { return j; }
};
constexpr int CONV_LINE_THREADS = 256;
constexpr size_t CONV_LINE_SHARED_MAX = 200 * 1024;
// Floats from one position of `cols` lines to the next. A warp works on quads 4 positions apart, 32 /
// cols of them: with 10 and 20 floats for 8 and 16 lines they read different banks (packed lines
// read the same ones four and two at a time). Along x lines are transposed as they are copied, for
// which an odd stride has no conflict either.
__host__ __device__ constexpr int conv_line_stride(int cols, bool along_x) {
    return along_x ? cols + 1 : cols == 8 ? 10 : cols == 16 ? 20 : cols;
}
// shared bytes of a block of `cols` lines
inline size_t conv_line_bytes(int cols, int n, int R, bool along_x) {
    return 4 * ((size_t)conv_weight_floats(R, n) + (size_t)(n + 2 * R) * conv_line_stride(cols, along_x));
}
inline int conv_line_cols(int n, int R, bool along_x) {
    for (int cols : { 32, 16, 8 })
        if (conv_line_bytes(cols, n, R, along_x) <= (cols == 8 ? CONV_LINE_SHARED_MAX : 64 * 1024)) return cols;
    return 0;
}

// [outer][n][inner] lines along n. kAlongX: inner = 1 (a line is contiguous). Groups of kCols lines:
// of consecutive inner positions, or along x of consecutive rows.
template <int kCols, bool kAlongX>
__global__ void __launch_bounds__(CONV_LINE_THREADS)
k_conv_lines(float *__restrict__ img, long long outer, int n, int inner, const __grid_constant__ ConvTaps K, int R) {
    extern __shared__ __align__(16) float conv_sm[];
    constexpr int kStride = conv_line_stride(kCols, kAlongX), kWarps = CONV_LINE_THREADS / 32, kSub = 32 / kCols;
    float *dens, *w = conv_sm;
    conv_weights(n, R, K.k, EverySample{}, n, w, dens);
    float *body = conv_sm + conv_weight_floats(R, n) + R * kStride;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *base;
    int cols;
    if (kAlongX) {
        const long long row = (long long)blockIdx.x * kCols;
        cols = (int)min((long long)kCols, outer - row);
        base = img + row * n;
        for (int r = warp; r < cols; r += kWarps)
#pragma unroll 4
            for (int x = lane; x < n; x += 32) body[x * kStride + r] = base[(long long)r * n + x];
    } else {
        const int groups = (inner + kCols - 1) / kCols;
        const long long o = blockIdx.x / groups;
        const int i0 = (int)(blockIdx.x - o * groups) * kCols;
        cols = min(kCols, inner - i0);
        base = img + o * n * inner + i0;
#pragma unroll 4
        for (int p = warp * kSub + lane / kCols; p < n; p += kWarps * kSub)
            if (lane % kCols < cols) body[p * kStride + lane % kCols] = base[(long long)p * inner + lane % kCols];
    }
    for (int i = threadIdx.x; i < R * kStride; i += CONV_LINE_THREADS) (body - R * kStride)[i] = body[n * kStride + i] = 0.f;
    __syncthreads();
    // the lines are in shared memory whole, so outputs go straight to the image
    const int col = lane % kCols;
    const float *line = body + col;
    const int quads = (n + 3) / 4, step = kWarps * kSub;
    for (int q0 = 0; q0 < quads; q0 += step) {
        const int q = q0 + warp * kSub + lane / kCols;
        if (q >= quads || col >= cols) continue;
        float v[4];
        conv_outputs4(n, R, w, dens, EverySample{}, n, 4 * q, [&](int k) { return line[k * kStride]; }, v);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (4 * q + u < n) base[kAlongX ? (long long)col * n + 4 * q + u : (long long)(4 * q + u) * inner + col] = v[u];
    }
}

// Whether the whole-line pass of `blocks` blocks beats the separate ones. It does where it fills the
// device, unless that takes thousands of blocks of a few positions each, whose set-up then costs more
// than their voxels (1024x512 lines of 4, 7 and 12 positions along y or z: 74, 80 and 98 us against
// 47, 75 and 130; along x of 4, 10 and 12: 91, 108 and 111 against 47, 100 and 136). With fewer blocks its time is a block's own: the taps of a warp's quads one after the other,
// and along y and z the positions that it copies (0.075 us a tap, eight taps a position). The
// separate passes take 9 us more per volume and run their taps in every voxel at once (0.056 us a tap
// and volume, 8e5 taps a us). All in taps of the first kind; 3x4x1900 along z, 481 taps: 54 us
// separate, 572 whole; 10x1000x9 along y, 161: 37, 124; 64x64x64, 21: 27, 20; 129x65x33 along x,
// 161: 55, 36; three volumes of 100x101x3 along y, 201: 87, 59.
static bool conv_lines_pay(int n, int R, int cols, bool along_x, int nvol, long long nvox, long long blocks) {
    if (blocks >= sm_count()) return blocks <= 4096 || n >= (along_x ? 11 : 8);
    const int slots = CONV_LINE_THREADS / cols;  // positions of a line that a block works on at once
    const double taps = 2.0 * R + 1, quads = (n + 3) / 4;
    const double chain = std::ceil(quads / slots) * taps + (along_x ? 0.0 : 8 * std::ceil((double)n / slots));
    return chain <= 27 + nvol * (120 + 0.75 * taps + nvox * taps / 6e4);
}

// whole-volume convolution of nvol volumes along an axis in place; false when a line and its taps do
// not fit a block or do not pay (the caller then runs the separate passes)
static bool conv_lines(float *img, int nvol, const int32_t dim[3], int axis, const ConvTaps& taps, int radius,
                       cudaStream_t st, nrb_status *status) {
    if ((long long)dim[0] * dim[1] >= (1LL << 31)) return false;  // a slice is addressed with an int
    // taps further out than a line is long meet no voxel
    const int n = dim[axis], R = std::min(radius, n - 1);
    const int cols = conv_line_cols(n, R, axis == 0);
    if (cols == 0) return false;
    const int inner = axis == 0 ? 1 : axis == 1 ? dim[0] : dim[0] * dim[1];
    const long long lines = (long long)nvol * dim[0] * dim[1] * dim[2] / n, outer = lines / inner;
    const long long blocks = axis == 0 ? (lines + cols - 1) / cols : outer * ((inner + cols - 1LL) / cols);
    if (blocks >= (1LL << 31) ||
        !conv_lines_pay(n, R, cols, axis == 0, nvol, (long long)dim[0] * dim[1] * dim[2], blocks)) return false;
    ConvTaps K;
    std::copy(taps.k + (radius - R), taps.k + (radius + R + 1), K.k);
    const size_t smem = conv_line_bytes(cols, n, R, axis == 0);
    auto go = [&](auto kernel) -> nrb_status {
        // one constant: the opt-in is the function's, and other host threads launch it too
        NRB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CONV_LINE_SHARED_MAX));
        kernel<<<(unsigned)blocks, CONV_LINE_THREADS, smem, st>>>(img, outer, n, inner, K, R);
        NRB_LAUNCHED("k_conv_lines");
        return NRB_OK;
    };
    if (axis == 0)
        *status = cols == 32 ? go(k_conv_lines<32, true>) : cols == 16 ? go(k_conv_lines<16, true>) : go(k_conv_lines<8, true>);
    else
        *status = cols == 32 ? go(k_conv_lines<32, false>) : cols == 16 ? go(k_conv_lines<16, false>) : go(k_conv_lines<8, false>);
    return true;
}

// value / density, NaN where the original value was NaN (_reg_tools.cpp:1100-1110)
__global__ void k_conv_normalise(long long nv, const float *orig, const float *__restrict__ v,
                                 const float *__restrict__ d, float *out) {  // out may alias orig
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv;
         i += (long long)gridDim.x * blockDim.x) {
        const float o = orig[i];
        out[i] = (o != o) ? o : v[i] / d[i];
    }
}

// float affine map in the reference's evaluation order, no contraction
__device__ __forceinline__ float affine_row_rn(const float *m, float x, float y, float z) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, m[0]), __fmul_rn(y, m[1])), __fmul_rn(z, m[2])), m[3]);
}

// Round<int> of reg-lib/cpu/Maths.hpp:83-85
__device__ __forceinline__ int round_ref(float x) { return (int)__fadd_rn(x, x >= 0.f ? 0.5f : -0.5f); }

// nearest-neighbour downsampling (reg_downsampleImage, reg-lib/cpu/_reg_tools.cpp:1343-1440):
// new voxel -> mm with the new qform, mm -> old voxel with the old one, rounded; NaN outside.
__global__ void k_downsample(int nx, int ny, int nz, int ox, int oy, int oz, Mat34 new_xyz,
                             Mat34 old_ijk, const float *__restrict__ in, float *__restrict__ out) {
    const long long nv = (long long)nx * ny * nz;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv;
         i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % nx), y = (int)((i / nx) % ny), z = (int)(i / ((long long)nx * ny));
        const float rx = affine_row_rn(new_xyz.m, (float)x, (float)y, (float)z);
        const float ry = affine_row_rn(new_xyz.m + 4, (float)x, (float)y, (float)z);
        const float rz = affine_row_rn(new_xyz.m + 8, (float)x, (float)y, (float)z);
        const float px = affine_row_rn(old_ijk.m, rx, ry, rz);
        const float py = affine_row_rn(old_ijk.m + 4, rx, ry, rz);
        const float pz = affine_row_rn(old_ijk.m + 8, rx, ry, rz);
        const int X = round_ref(px), Y = round_ref(py), Z = oz == 1 ? 0 : round_ref(pz);
        float v = __int_as_float(0x7fffffff);
        if (X > -1 && X < ox && Y > -1 && Y < oy && Z > -1 && Z < oz) v = in[((long long)Z * oy + Y) * ox + X];
        out[i] = v;
    }
}

// The smoothing, normalisation and downsampling of one pyramid level in one pass. A block of
// 32 x 8 threads owns 32 x 8 output columns over a run of output slices: it walks the input slices
// they need, convolves each along x at the sampled columns and along y at the sampled rows in
// shared memory (only the values a sampled output reads), and every thread keeps the last
// 2 * SMOOTH_R + 1 results of its column in registers for the z pass, whose output it divides and
// stores. Sums are k_conv_axis's, tap for tap; a tap outside the volume adds weight * 0. While no
// value is NaN the density of an output depends on its indices alone (three short sums); a block
// that meets a NaN starts its run over with (value, density) pairs.
//
// One read of the input and one write of the output, where the three axis passes, the normalisation
// and the sampling moved 60 bytes per input voxel (and 16 bytes per voxel of temporaries were
// mapped for each call). Bound by instruction issue now (72% active, 38% of the copy bandwidth):
// 512x512x320 -> 256x256x160 takes 193 us, the separate passes took about 4 ms. Tiles of 32 x 8
// outputs: the rows' halo is 6% and the columns' 25%, read from L2, and 256 threads with 64
// registers keep four blocks per SM in flight across the two barriers of a slice.
constexpr int SMOOTH_R = 2, SMOOTH_TAPS = 2 * SMOOTH_R + 1, SMOOTH_X = 32, SMOOTH_Y = 8;
constexpr int SMOOTH_IN_X = 2 * SMOOTH_X + 2 * SMOOTH_R, SMOOTH_IN_Y = 2 * SMOOTH_Y + 2 * SMOOTH_R;
constexpr int SMOOTH_THREADS = SMOOTH_X * SMOOTH_Y;
constexpr int SMOOTH_LOADS = (SMOOTH_IN_X * SMOOTH_IN_Y + SMOOTH_THREADS - 1) / SMOOTH_THREADS;

struct SmoothParams {
    int n[3], o[3], s[3];    // input dims, output dims, shift per axis (0 or 1): output i samples i << s
    int zrun;                // output slices per block
    float k[SMOOTH_TAPS];
};

// sum of the weights of the taps of position p inside [0, n), each times d (a pass over densities)
__device__ __forceinline__ float smooth_density(const float *k, int p, int n, float d) {
    float s = 0.f;
#pragma unroll
    for (int t = 0; t < SMOOTH_TAPS; ++t)
        if ((unsigned)(p + t - SMOOTH_R) < (unsigned)n) s = fmaf(k[t], d, s);
    return s;
}

// One block's run; returns false (with nothing final written) when !kNan and an input value is NaN
template <bool kNan, bool kHalve>
__device__ __forceinline__ bool smooth_run(const SmoothParams& P, const float *__restrict__ in, float *__restrict__ out,
                                           float (*tile)[SMOOTH_IN_Y * SMOOTH_IN_X], float (*xs)[SMOOTH_IN_Y * SMOOTH_X]) {
    const int tid = threadIdx.x, lx = tid % SMOOTH_X, ly = tid / SMOOTH_X;
    const int ox0 = blockIdx.x * SMOOTH_X, oy0 = blockIdx.y * SMOOTH_Y, oz0 = blockIdx.z * P.zrun;
    const int oz1 = min(oz0 + P.zrun, P.o[2]);
    const int sx = kHalve ? 1 : P.s[0], sy = kHalve ? 1 : P.s[1], sz = kHalve ? 1 : P.s[2];
    const int ix0 = (ox0 << sx) - SMOOTH_R, iy0 = (oy0 << sy) - SMOOTH_R;
    const int wx = ((SMOOTH_X - 1) << sx) + SMOOTH_TAPS, wy = ((SMOOTH_Y - 1) << sy) + SMOOTH_TAPS;
    const int x = ox0 + lx, y = oy0 + ly;
    const bool mine = x < P.o[0] && y < P.o[1];
    const long long plane = (long long)P.n[0] * P.n[1];
    // the elements of a slice's tile this thread loads: offset in the slice, and byte offset in the
    // tile (-1: outside the volume or the tile, never written, so the zero stored here stays)
    int src[SMOOTH_LOADS], dst[SMOOTH_LOADS];
#pragma unroll
    for (int l = 0; l < SMOOTH_LOADS; ++l) {
        const int e = tid + l * SMOOTH_THREADS;
        const int r = e / wx, c = e - r * wx;
        const int gx = ix0 + c, gy = iy0 + r;
        const bool inside = r < wy && (unsigned)gx < (unsigned)P.n[0] && (unsigned)gy < (unsigned)P.n[1];
        src[l] = inside ? gy * P.n[0] + gx : 0;
        dst[l] = inside ? 4 * (r * SMOOTH_IN_X + c) : -1;
        asm volatile("" : "+r"(src[l]), "+r"(dst[l]));  // kept in registers, not recomputed per slice
    }
    for (int e = tid; e < SMOOTH_IN_Y * SMOOTH_IN_X; e += SMOOTH_THREADS) tile[0][e] = tile[1][e] = 0.f;
    __syncthreads();
    // the density over x and y, and that of a column whose z taps are all inside
    const float dxy = kNan ? 0.f : smooth_density(P.k, y << sy, P.n[1], smooth_density(P.k, x << sx, P.n[0], 1.f));
    const float dmid = kNan ? 0.f : smooth_density(P.k, SMOOTH_R, SMOOTH_TAPS, dxy);
    float v[SMOOTH_TAPS], d[SMOOTH_TAPS];
#pragma unroll
    for (int t = 0; t < SMOOTH_TAPS; ++t) v[t] = d[t] = 0.f;
    const int z0 = (oz0 << sz) - SMOOTH_R, z1 = ((oz1 - 1) << sz) + SMOOTH_R;
    float next[SMOOTH_LOADS];
    auto fetch = [&](int z) {
        if ((unsigned)z >= (unsigned)P.n[2]) return;
        const float *p = in + z * plane;
#pragma unroll
        for (int l = 0; l < SMOOTH_LOADS; ++l)
            if (dst[l] >= 0) next[l] = __ldg(p + src[l]);
    };
    auto slot = [&](int q, int l) -> float& { return *reinterpret_cast<float *>(reinterpret_cast<char *>(tile[q]) + dst[l]); };
#pragma unroll
    for (int l = 0; l < SMOOTH_LOADS; ++l) next[l] = 0.f;
    fetch(z0);
    int nan = 0;
    for (int z = z0; z <= z1; ++z) {
        const bool inz = (unsigned)z < (unsigned)P.n[2];
#pragma unroll
        for (int l = 0; l < SMOOTH_LOADS; ++l) {
            if (dst[l] < 0) continue;
            const bool use = inz && (!kNan || next[l] == next[l]);
            slot(0, l) = use ? next[l] : 0.f;
            if (kNan) slot(1, l) = use ? 1.f : 0.f;
        }
        if (z < z1) fetch(z + 1);  // in flight while this slice is convolved
        // a NaN shows in the sums of the slice it is in (the check of a slice is read one later)
        if (kNan) __syncthreads();
        else if (__syncthreads_or(nan)) return false;
        // along x at the sampled columns of every row of the tile
#pragma unroll
        for (int u = 0; u < (SMOOTH_IN_Y + SMOOTH_Y - 1) / SMOOTH_Y; ++u) {
            const int r = ly + u * SMOOTH_Y;
            if (r >= wy) break;
#pragma unroll
            for (int q = 0; q < (kNan ? 2 : 1); ++q) {
                const float *row = tile[q] + r * SMOOTH_IN_X + (lx << sx);
                float in5[SMOOTH_TAPS + 1];
                if (kHalve) {  // 8-byte aligned: three loads without a bank conflict for the five taps
#pragma unroll
                    for (int t = 0; t < SMOOTH_TAPS + 1; t += 2) {
                        const float2 w = *reinterpret_cast<const float2 *>(row + t);
                        in5[t] = w.x;
                        in5[t + 1] = w.y;
                    }
                } else {
#pragma unroll
                    for (int t = 0; t < SMOOTH_TAPS; ++t) in5[t] = row[t];
                }
                float s = 0.f;
#pragma unroll
                for (int t = 0; t < SMOOTH_TAPS; ++t) s = fmaf(P.k[t], in5[t], s);
                xs[q][r * SMOOTH_X + lx] = s;
            }
        }
        __syncthreads();
        // along y at the sampled rows, into the column's window
#pragma unroll
        for (int t = 0; t + 1 < SMOOTH_TAPS; ++t) {
            v[t] = v[t + 1];
            if (kNan) d[t] = d[t + 1];
        }
#pragma unroll
        for (int q = 0; q < (kNan ? 2 : 1); ++q) {
            const float *col = xs[q] + (ly << sy) * SMOOTH_X + lx;
            float s = 0.f;
#pragma unroll
            for (int t = 0; t < SMOOTH_TAPS; ++t) s = fmaf(P.k[t], col[t * SMOOTH_X], s);
            (q == 0 ? v : d)[SMOOTH_TAPS - 1] = s;
            nan |= s != s;
        }
        // along z: the window is centred on slice z - SMOOTH_R
        const int zc = z - SMOOTH_R;
        if (zc < (oz0 << sz) || (zc & sz) != 0 || !mine) continue;
        float num = 0.f, den = 0.f;
#pragma unroll
        for (int t = 0; t < SMOOTH_TAPS; ++t) {
            num = fmaf(P.k[t], v[t], num);
            if (kNan) den = fmaf(P.k[t], d[t], den);
        }
        if (!kNan) den = zc >= SMOOTH_R && zc + SMOOTH_R < P.n[2] ? dmid : smooth_density(P.k, zc, P.n[2], dxy);
        float r = num / den;
        if (kNan) {
            const float o = __ldg(in + zc * plane + (long long)(y << sy) * P.n[0] + (x << sx));
            if (o != o) r = o;  // _reg_tools.cpp:1100-1110
        }
        out[((long long)(zc >> sz) * P.o[1] + y) * P.o[0] + x] = r;
    }
    if (!kNan && __syncthreads_or(nan)) return false;
    return true;
}

template <bool kHalve>
__global__ void __launch_bounds__(SMOOTH_THREADS, 4)
k_smooth_downsample(const __grid_constant__ SmoothParams P, const float *__restrict__ in, float *__restrict__ out) {
    __shared__ __align__(16) float tile[2][SMOOTH_IN_Y * SMOOTH_IN_X];
    __shared__ float xs[2][SMOOTH_IN_Y * SMOOTH_X];
    if (smooth_run<false, kHalve>(P, in, out, tile, xs)) return;
    __syncthreads();
    smooth_run<true, kHalve>(P, in, out, tile, xs);
}

// ---------------------------------------------------------------------------------------------
// reductions and element-wise updates
// ---------------------------------------------------------------------------------------------
// [0, n) of `img` as `head` elements before its first 16-byte boundary, `nvec` whole float4s and a
// tail of at most three.
struct VecSpan {
    long long head, nvec, n;
    __device__ __forceinline__ VecSpan(const float *img, long long count): n(count) {
        head = min(count, (long long)((16 - (reinterpret_cast<uintptr_t>(img) & 15)) & 15) / 4);
        nvec = (count - head) / 4;
    }
};

// min and max are exact in any order, so the split is free: it is chosen to keep loads in flight
__global__ void __launch_bounds__(2 * NRB_RED_THREADS, 4)
k_minmax(long long n, const float *__restrict__ img, float *__restrict__ pmin, float *__restrict__ pmax) {
    __shared__ float smin[2 * NRB_RED_THREADS / 32], smax[2 * NRB_RED_THREADS / 32];
    const VecSpan S(img, n);
    const long long gtid = blockIdx.x * (long long)blockDim.x + threadIdx.x, gs = (long long)gridDim.x * blockDim.x;
    float mn = FLT_MAX, mx = -FLT_MAX;
    auto take = [&](float v) {
        if (v == v) {
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
        }
    };
    const float4 *vec = reinterpret_cast<const float4 *>(img + S.head);
    long long i = gtid;
    for (; i + gs < S.nvec; i += 2 * gs) {
        float4 q[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) q[u] = __ldg(vec + i + u * gs);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            take(q[u].x);
            take(q[u].y);
            take(q[u].z);
            take(q[u].w);
        }
    }
    for (; i < S.nvec; i += gs) {
        const float4 q = __ldg(vec + i);
        take(q.x);
        take(q.y);
        take(q.z);
        take(q.w);
    }
    if (gtid < S.head) take(img[gtid]);
    const long long tail = S.head + 4 * S.nvec + gtid;
    if (tail < n) take(img[tail]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        smin[threadIdx.x >> 5] = mn;
        smax[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)blockDim.x / 32; ++w) {
            mn = fminf(mn, smin[w]);
            mx = fmaxf(mx, smax[w]);
        }
        pmin[blockIdx.x] = mn;
        pmax[blockIdx.x] = mx;
    }
}

// reg_intensityRescale_core (reg-lib/cpu/_reg_tools.cpp:92-174): double-precision rescale of
// the finite values; every block combines the min/max partials itself.
//
// The quotient by the range is the correctly rounded one from the rounded reciprocal and one
// residual step (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990): three FP64 operations per voxel instead of a division.
// It needs a finite, normal range and quotient; other ranges (infinite values, a constant image)
// are divided. Four floats per load and store. 512x512x320: min/max 54 us, rescale 140 us (74% of
// the copy bandwidth; FP64 division and single floats before).
__global__ void __launch_bounds__(256)
k_rescale(long long n, float *__restrict__ img, const float *__restrict__ pmin, const float *__restrict__ pmax, int np,
          float new_min, float new_max) {
    __shared__ float smin[8], smax[8];
    float mn = FLT_MAX, mx = -FLT_MAX;
    for (int i = threadIdx.x; i < np; i += blockDim.x) {
        mn = fminf(mn, pmin[i]);
        mx = fmaxf(mx, pmax[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        smin[threadIdx.x >> 5] = mn;
        smax[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    mn = smin[0];
    mx = smax[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) {
        mn = fminf(mn, smin[w]);
        mx = fmaxf(mx, smax[w]);
    }
    const double cur = (double)(mx - mn), nd = (double)(new_max - new_min), lo = (double)mn;
    const bool by_reciprocal = cur > 1e-30 && cur < 1e38;
    const double inv = 1.0 / cur;
    auto one = [&](float f) {
        double v = (double)f;
        if (v == v) {
            const double a = v - lo;
            if (by_reciprocal) {
                const double q = a * inv;
                v = fma(fma(-cur, q, a), inv, q);
            } else {
                v = a / cur;
            }
            v = fma(v, nd, (double)new_min);
        }
        return (float)v;
    };
    const VecSpan S(img, n);
    const long long gtid = blockIdx.x * (long long)blockDim.x + threadIdx.x, gs = (long long)gridDim.x * blockDim.x;
    float4 *vec = reinterpret_cast<float4 *>(img + S.head);
    for (long long i = gtid; i < S.nvec; i += gs) {
        float4 q = vec[i];
        q.x = one(q.x);
        q.y = one(q.y);
        q.z = one(q.z);
        q.w = one(q.w);
        vec[i] = q;
    }
    if (gtid < S.head) img[gtid] = one(img[gtid]);
    const long long tail = S.head + 4 * S.nvec + gtid;
    if (tail < n) img[tail] = one(img[tail]);
}

// reg_getMaximalLength (reg-lib/cpu/_reg_tools.cpp:335-355): float lengths, max is exact in any
// order.
__global__ void __launch_bounds__(NRB_RED_THREADS)
k_maxlen(long long nnode, const float *__restrict__ g, float *__restrict__ pmax) {
    __shared__ float s[NRB_RED_THREADS];
    float mx = 0.f;
    for (long long i = blockIdx.x * (long long)NRB_RED_THREADS + threadIdx.x; i < nnode;
         i += (long long)gridDim.x * NRB_RED_THREADS) {
        const float x = g[i], y = g[nnode + i], z = g[2 * nnode + i];
        const float l = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
        mx = fmaxf(mx, l);
    }
    s[threadIdx.x] = mx;
    __syncthreads();
    for (int k = NRB_RED_THREADS / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) s[threadIdx.x] = fmaxf(s[threadIdx.x], s[threadIdx.x + k]);
        __syncthreads();
    }
    if (threadIdx.x == 0) pmax[blockIdx.x] = s[0];
}

// one thread per partial (a max is exact in any order; a single thread's chain of loads took 9 us)
__global__ void __launch_bounds__(NRB_RED_BLOCKS)
k_maxlen_finish(const float *__restrict__ pmax, int np, nrb_objective *__restrict__ obj, double *__restrict__ out) {
    __shared__ float s[NRB_RED_BLOCKS / 32];
    float mx = threadIdx.x < np ? pmax[threadIdx.x] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 0; w < NRB_RED_BLOCKS / 32; ++w) mx = fmaxf(mx, s[w]);
        if (obj) obj->max_grad_len = (double)mx;
        if (out) *out = (double)mx;
    }
}

// Compute::NormaliseGradient (reg-lib/Compute.cpp:148-176)
__global__ void k_normalise(long long n, float *__restrict__ g, const nrb_objective *__restrict__ obj,
                            double len) {
    const double l = len >= 0 ? len : obj->max_grad_len;
    if (l == 0) return;
    const double inv = 1.0 / l;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        g[i] = (float)((double)g[i] * inv);
}

// Compute::UpdateControlPointPosition (reg-lib/Compute.cpp:103-106)
__global__ void k_update(long long n, float *__restrict__ cur, const float *__restrict__ best,
                         const float *__restrict__ grad, float scale) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        cur[i] = __fadd_rn(best[i], __fmul_rn(scale, grad[i]));
}

// ConjugateGradient::UpdateGradientValues (reg-lib/Optimiser.cpp:231-317)
__global__ void k_cg_init(long long n, const float *__restrict__ g, float *__restrict__ g1, float *__restrict__ g2) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float v = -g[i];
        g1[i] = v;
        g2[i] = v;
    }
}

__global__ void __launch_bounds__(NRB_RED_THREADS)
k_cg_dots(long long n, const float *__restrict__ g, const float *__restrict__ g1,
          const float *__restrict__ g2, double *__restrict__ partials) {
    __shared__ double red[NRB_RED_THREADS];
    double gg = 0, dgg = 0;
    for (long long i = blockIdx.x * (long long)NRB_RED_THREADS + threadIdx.x; i < n;
         i += (long long)gridDim.x * NRB_RED_THREADS) {
        gg += (double)__fmul_rn(g2[i], g1[i]);
        dgg += (double)__fmul_rn(__fadd_rn(g[i], g1[i]), g[i]);
    }
    const double a = block_sum_d(gg, red);
    __syncthreads();
    const double b = block_sum_d(dgg, red);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = a;
        partials[2 * blockIdx.x + 1] = b;
    }
}

// first_call (optional, device flag): when set, the first-call initialisation g1 = g2 = -g
// runs instead, so one captured launch serves both branches of UpdateGradientValues.
__global__ void k_cg_update(long long n, float *__restrict__ g, float *__restrict__ g1,
                            float *__restrict__ g2, const double *__restrict__ partials, int np,
                            const int *__restrict__ first_call) {
    if (first_call && *first_call) {
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
             i += (long long)gridDim.x * blockDim.x) {
            const float v = -g[i];
            g1[i] = v;
            g2[i] = v;
        }
        return;
    }
    // the partials are copied to shared memory by the whole block, then summed in index order by
    // two threads (gg and dgg side by side), instead of one thread's chain of global loads
    __shared__ double sp[2 * NRB_RED_BLOCKS];
    __shared__ double sgg, sdgg;
    for (int i = threadIdx.x; i < 2 * np; i += blockDim.x) sp[i] = partials[i];
    __syncthreads();
    if (threadIdx.x == 0 || threadIdx.x == 32) {
        const int q = threadIdx.x == 0 ? 0 : 1;
        double sum = 0;
        for (int i = 0; i < np; ++i) sum += sp[2 * i + q];
        if (q == 0) sgg = sum;
        else sdgg = sum;
    }
    __syncthreads();
    const double gm = sdgg / sgg;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float a1 = -g[i];
        const float a2 = (float)((double)a1 + gm * (double)g2[i]);
        g1[i] = a1;
        g2[i] = a2;
        g[i] = -a2;
    }
}

// ---------------------------------------------------------------------------------------------
// control-point grid construction and refinement
// ---------------------------------------------------------------------------------------------
// reg_createControlPointGrid's identity initialisation (reg_getDeformationFromDisplacement)
__global__ void k_grid_identity(int cx, int cy, int cz, Mat34 M, float *__restrict__ cpp) {
    const long long nc = (long long)cx * cy * cz;
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < nc;
         n += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(n % cx), y = (int)((n / cx) % cy), z = (int)(n / ((long long)cx * cy));
        for (int k = 0; k < 3; ++k) cpp[k * nc + n] = identity_pos(M, k, x, y, z);
    }
}

// reg_spline_refineControlPointGrid3D (reg-lib/cpu/_reg_localTrans.cpp:1809-2119): new node
// 2x-1 takes the (1,6,1)/8 mask around old node x, new node 2x the (1,1)/2 mask of x, x+1,
// per axis; old nodes outside the grid read as 0; new nodes past 2*old-2 are never written
// by the reference and stay 0.
__device__ __forceinline__ int refine_taps(int X, int oldn, int idx[3], int w[3]) {
    if ((X + 1) % 2 == 0) {
        const int x = (X + 1) / 2;
        if (x >= oldn) return 0;
        idx[0] = x - 1; idx[1] = x; idx[2] = x + 1;
        w[0] = 1; w[1] = 6; w[2] = 1;
        return 3;
    }
    const int x = X / 2;
    if (x >= oldn) return 0;
    idx[0] = x; idx[1] = x + 1;
    w[0] = 1; w[1] = 1;
    return 2;
}

__global__ void k_grid_refine(int ox, int oy, int oz, int nx, int ny, int nz, const float *__restrict__ old,
                              float *__restrict__ out) {
    const long long onc = (long long)ox * oy * oz, nnc = (long long)nx * ny * nz;
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < nnc;
         n += (long long)gridDim.x * blockDim.x) {
        const int X = (int)(n % nx), Y = (int)((n / nx) % ny), Z = (int)(n / ((long long)nx * ny));
        int ix[3], iy[3], iz[3], wx[3], wy[3], wz[3];
        const int ax = refine_taps(X, ox, ix, wx), ay = refine_taps(Y, oy, iy, wy), az = refine_taps(Z, oz, iz, wz);
        const float den = (float)((ax == 3 ? 8 : 2) * (ay == 3 ? 8 : 2) * (az == 3 ? 8 : 2));
        for (int k = 0; k < 3; ++k) {
            float v = 0.f;
            if (ax && ay && az) {
                // weight classes summed separately as the reference groups them
                float s1 = 0.f, s6 = 0.f, s36 = 0.f, s216 = 0.f;
                for (int c = 0; c < az; ++c)
                    for (int b = 0; b < ay; ++b)
                        for (int a = 0; a < ax; ++a) {
                            const int x = ix[a], y = iy[b], z = iz[c];
                            float val = 0.f;
                            if (x >= 0 && x < ox && y >= 0 && y < oy && z >= 0 && z < oz)
                                val = old[k * onc + ((long long)z * oy + y) * ox + x];
                            const int w = wx[a] * wy[b] * wz[c];
                            if (w == 1) s1 += val;
                            else if (w == 6) s6 += val;
                            else if (w == 36) s36 += val;
                            else s216 += val;
                        }
                v = (s1 + 6.f * s6 + 36.f * s36 + 216.f * s216) / den;
            }
            out[k * nnc + n] = v;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
static int grid_for(long long n, int threads, int max_blocks_per_sm = 16) {
    const long long want = (n + threads - 1) / threads;
    return (int)std::max<long long>(1, std::min<long long>(want, (long long)max_blocks_per_sm * sm_count()));
}

// Kernel width of reg_tools_kernelConvolution (_reg_tools.cpp:882-884): the spacing in mm over
// the voxel size, or |spacing| voxels when the spacing is negative; radius = int(2 * width).
// Refuses spacings and voxel sizes for which that is undefined (NaN, infinite, a voxel size that
// is not > 0 with a spacing in mm) and radii above 2^20 voxels.
static nrb_status cubic_extent(const char *who, float spacing_mm, float pixdim, double& temp, int& radius) {
    if (!std::isfinite(spacing_mm) || (spacing_mm > 0 && !(std::isfinite(pixdim) && pixdim > 0.f)))
        return fail(NRB_ERR_INVALID, std::string(who) + ": the spacing must be finite and, when given in mm, the "
                                                        "voxel size finite and > 0");
    temp = spacing_mm > 0 ? (double)(spacing_mm / pixdim) : std::fabs((double)spacing_mm);
    if (!(temp * 2.0 < (double)(1 << 20)))
        return fail(NRB_ERR_UNSUPPORTED, std::string(who) + ": kernel radius above 2^20 voxels");
    radius = (int)(temp * 2.0f);
    return NRB_OK;
}

// the 2 * radius + 1 cubic B-spline taps of reg_tools_kernelConvolution (_reg_tools.cpp:893-904)
static void cubic_taps(double temp, int radius, float *out) {
    for (int i = -radius; i <= radius; ++i) {
        const double rel = std::fabs(i / temp);
        float v;
        if (rel < 1.0) v = (float)(2.0 / 3.0 - rel * rel + 0.5 * rel * rel * rel);
        else if (rel < 2.0) v = (float)(-(rel - 2.0) * (rel - 2.0) * (rel - 2.0) / 6.0);
        else v = 0.f;
        out[i + radius] = v;
    }
}

// cubic B-spline convolution kernel of a geometry the workspace has already validated
static std::vector<float> cubic_kernel(float spacing_mm, float pixdim, int& radius) {
    const double temp = spacing_mm > 0 ? (double)(spacing_mm / pixdim) : std::fabs((double)spacing_mm);
    radius = (int)(temp * 2.0f);
    std::vector<float> k(2 * radius + 1);
    cubic_taps(temp, radius, k.data());
    return k;
}

// ref_ijk * cpp_xyz (mat44 product, entries rounded to float): the grid's node -> reference
// voxel map; aligned when its 3x3 part is diagonal (to 1e-6 relative), as every grid built by
// reg_createControlPointGrid / refinement is for its reference
static void node_to_voxel(const nrb_geometry *g, double T[3][4]) {
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 4; ++j) {
            double s = 0;
            for (int k = 0; k < 4; ++k) s += (double)g->ref_ijk[4 * i + k] * (double)g->cpp_xyz[4 * k + j];
            T[i][j] = (float)s;
        }
}
static bool grid_aligned(const nrb_geometry *g) {
    double T[3][4];
    node_to_voxel(g, T);
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            if (i != j && std::fabs(T[i][j]) > 1e-6 * std::fabs(T[i][i])) return false;
    return true;
}

nrb_status validate_geometry(const nrb_geometry *g) {
    // voxel and node indices are 32-bit in the kernels
    if (nvox(g->ref_dim) >= (1LL << 31) / 3 || nvox(g->flo_dim) >= (1LL << 31) || nvox(g->cpp_dim) >= (1LL << 31) / 3)
        return fail(NRB_ERR_UNSUPPORTED, "geometry: volume too large for 32-bit indexing");
    for (int d = 0; d < 3; ++d) {
        if (g->ref_dim[d] <= 0 || g->flo_dim[d] <= 0 || g->cpp_dim[d] <= 0)
            return fail(NRB_ERR_INVALID, "geometry: non-positive dimension");
        if (!(g->ref_pixdim[d] > 0) || !(g->cpp_pixdim[d] > 0))
            return fail(NRB_ERR_INVALID, "geometry: non-positive voxel size");
        if (g->ref_dim[d] > 2048) return fail(NRB_ERR_UNSUPPORTED, "geometry: dimension above 2048");
        const float gs = g->cpp_pixdim[d] / g->ref_pixdim[d];
        if (gs < 1.f) return fail(NRB_ERR_UNSUPPORTED, "geometry: control spacing below one voxel");
        const int last = (int)((float)(g->ref_dim[d] - 1) / gs);
        // the aligned passes address nodes from voxel indices; an unaligned grid is sampled
        // through its full matrix (0 outside), so only an aligned grid must cover the reference
        if (last + 3 >= g->cpp_dim[d] && grid_aligned(g))
            return fail(NRB_ERR_UNSUPPORTED, "geometry: control-point grid does not cover the reference");
    }
    return NRB_OK;
}

static int tile_span(int n, int tile, float gs) {
    int span = 0;
    for (int v0 = 0; v0 < n; v0 += tile) {
        const int v1 = std::min(v0 + tile - 1, n - 1);
        span = std::max(span, (int)((float)v1 / gs) + 4 - (int)((float)v0 / gs));
    }
    return span;
}

// Node -> reference voxel sampling per axis (reg_voxelCentricToNodeCentric,
// _reg_localTrans.cpp:1572-1631): requires ref_ijk * cpp_xyz to be axis-aligned, which holds
// for every grid built by reg_createControlPointGrid / refinement.
static nrb_status make_sampling(const nrb_geometry *g, AxisSampling ax[3]) {
    double T[3][4];
    node_to_voxel(g, T);  // mat44 operator* rounds each entry to float
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            if (i != j && std::fabs(T[i][j]) > 1e-6 * std::fabs(T[i][i]))
                return fail(NRB_ERR_UNSUPPORTED, "voxel->node: grid not axis-aligned with the reference");
    for (int d = 0; d < 3; ++d) {
        AxisSampling& a = ax[d];
        const int n = g->ref_dim[d], cn = g->cpp_dim[d];
        std::vector<int> pre(cn);
        std::vector<float> w1(cn);
        std::vector<int> used;
        for (int i = 0; i < cn; ++i) {
            const float v = (float)(T[d][d] * (double)i + T[d][3]);
            pre[i] = (int)std::floor(v);
            w1[i] = v - (float)pre[i];
            if (pre[i] >= 0 && pre[i] < n) used.push_back(pre[i]);
            if (w1[i] != 0.f && pre[i] + 1 >= 0 && pre[i] + 1 < n) used.push_back(pre[i] + 1);
        }
        std::sort(used.begin(), used.end());
        used.erase(std::unique(used.begin(), used.end()), used.end());
        if (used.empty()) used.push_back(0);  // keep buffers non-empty; no node reads it
        a.samples = used;
        a.nsamples = (int)used.size();
        a.tap_slot.assign(2 * cn, -1);
        a.tap_weight.assign(2 * cn, 0.f);
        for (int i = 0; i < cn; ++i) {
            const float w0 = 1.f - w1[i];
            if (pre[i] >= 0 && pre[i] < n) {
                a.tap_slot[2 * i] = (int)(std::lower_bound(used.begin(), used.end(), pre[i]) - used.begin());
                a.tap_weight[2 * i] = w0;
            }
            if (w1[i] != 0.f && pre[i] + 1 >= 0 && pre[i] + 1 < n) {
                a.tap_slot[2 * i + 1] = (int)(std::lower_bound(used.begin(), used.end(), pre[i] + 1) - used.begin());
                a.tap_weight[2 * i + 1] = w1[i];
            }
        }
        a.kernel = cubic_kernel(g->cpp_pixdim[d], g->ref_pixdim[d], a.radius);
    }
    return NRB_OK;
}

// A workspace's memory: on its owner's stream when it has one; otherwise from the library's pool as
// well, usable on any stream once the creator has synchronised, and given back only after the device
// has finished with it, as cudaFree would wait (mapping and unmapping fresh memory took most of a
// creation). Parts beyond what the pool keeps mapped are allocated plainly: from the pool, an oblique
// 512x512x160 workspace took 3.3 ms instead of 2.8.
static bool ws_plain(size_t bytes, cudaStream_t st) { return !st && bytes > kLibPoolFloor; }
template <typename T>
static cudaError_t ws_alloc(T **p, size_t bytes, cudaStream_t st) {
    return st || ws_plain(bytes, st) ? dev_alloc(p, bytes, st) : tmp_alloc(p, bytes, nullptr);
}

// Consecutive 256-byte aligned parts of one allocation
struct Arena {
    size_t bytes = 0;
    size_t add(size_t n) {
        const size_t at = bytes;
        bytes += (std::max<size_t>(1, n) + 255) & ~size_t(255);
        return at;
    }
};

// Items of the voxel walk. The persistent grid holds slots_for(shared bytes) co-resident blocks
// and every block walks ceil(items / slots) items, so the z-chunk count is chosen to minimise a
// block's walk: rounds x (slices per chunk + the item's fixed cost, `overhead` slices: staging,
// the x rows, the column set-up), over chunk counts that keep chunks at least `min_chunk`
// slices long (the staged control points are reused along z). Small volumes, whose few long
// items would leave most blocks idle, get shorter chunks spread over more blocks.
WalkPlan plan_walk(const nrb_geometry *g, int ty, long long (*slots_for)(size_t smem), size_t extra_smem,
                   int min_chunk, int overhead) {
    WalkPlan p;
    p.ty = ty;
    const int nx = g->ref_dim[0], ny = g->ref_dim[1], nz = g->ref_dim[2];
    const float gs[3] = { g->cpp_pixdim[0] / g->ref_pixdim[0], g->cpp_pixdim[1] / g->ref_pixdim[1],
                          g->cpp_pixdim[2] / g->ref_pixdim[2] };
    p.tiles_x = (nx + COL_X - 1) / COL_X;
    p.tiles_y = (ny + ty - 1) / ty;
    const long long xy = (long long)p.tiles_x * p.tiles_y;
    p.sa = tile_span(nx, COL_X, gs[0]);
    p.sb = tile_span(ny, ty, gs[1]);
    long long best_cost = LLONG_MAX;
    WalkPlan best = p;
    int last_chunk = -1;
    for (int c = 1; c <= std::max(1, nz / min_chunk); ++c) {
        WalkPlan q = p;
        q.zchunk = (nz + c - 1) / c;
        if (q.zchunk == last_chunk) continue;  // the same plan again (an occupancy query each)
        last_chunk = q.zchunk;
        q.nchunks = (nz + q.zchunk - 1) / q.zchunk;
        q.nitems = (int)(xy * q.nchunks);
        q.sc = tile_span(nz, q.zchunk, gs[2]);
        q.cp_floats = 3 * q.sa * q.sb * q.sc;
        const long long slots = std::max(1LL, slots_for(walk_smem_bytes(q) + extra_smem));
        const long long rounds = (q.nitems + slots - 1) / slots;
        const long long cost = rounds * (q.zchunk + overhead);
        if (cost < best_cost) {
            best_cost = cost;
            best = q;
        }
    }
    return best;
}

std::vector<WalkPlan> plan_walk_candidates(const nrb_geometry *g, int ty, long long (*slots_for)(size_t smem),
                                           size_t extra_smem, int min_chunk, int overhead, int count) {
    const int nx = g->ref_dim[0], ny = g->ref_dim[1], nz = g->ref_dim[2];
    const float gs[3] = { g->cpp_pixdim[0] / g->ref_pixdim[0], g->cpp_pixdim[1] / g->ref_pixdim[1],
                          g->cpp_pixdim[2] / g->ref_pixdim[2] };
    WalkPlan p;
    p.ty = ty;
    p.tiles_x = (nx + COL_X - 1) / COL_X;
    p.tiles_y = (ny + ty - 1) / ty;
    p.sa = tile_span(nx, COL_X, gs[0]);
    p.sb = tile_span(ny, ty, gs[1]);
    const long long xy = (long long)p.tiles_x * p.tiles_y;
    std::vector<std::pair<long long, WalkPlan>> all;
    int last_chunk = -1;
    for (int c = 1; c <= std::max(1, nz / min_chunk); ++c) {
        WalkPlan q = p;
        q.zchunk = (nz + c - 1) / c;
        if (q.zchunk == last_chunk) continue;
        last_chunk = q.zchunk;
        q.nchunks = (nz + q.zchunk - 1) / q.zchunk;
        q.nitems = (int)(xy * q.nchunks);
        q.sc = tile_span(nz, q.zchunk, gs[2]);
        q.cp_floats = 3 * q.sa * q.sb * q.sc;
        const long long slots = std::max(1LL, slots_for(walk_smem_bytes(q) + extra_smem));
        const long long rounds = (q.nitems + slots - 1) / slots;
        all.emplace_back(rounds * (q.zchunk + overhead), q);
    }
    std::stable_sort(all.begin(), all.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
    std::vector<WalkPlan> out;
    for (size_t i = 0; i < all.size() && (int)out.size() < count; ++i) out.push_back(all[i].second);
    return out;
}

nrb_status workspace_init(nrb_workspace *ws, const nrb_geometry *g) {
    ws->g = *g;
    // shared memory beyond the walk: the 64-bin joint histogram / FP32 log table (the plan is
    // made before the bin count is known; other bin counts shift occupancy little)
    ws->walk_obj = plan_walk(g, TY_OBJECTIVE, objective_slots, OBJ_PLAN_EXTRA, 4, 6);
    ws->walk_grad = plan_walk(g, TY_GRADIENT, gradient_slots, GRAD_PLAN_EXTRA, 4, 4);
    return NRB_OK;
}

static nrb_status workspace_alloc(nrb_workspace *ws) {
    const nrb_geometry *g = &ws->g;
    NRB_CUDA(cudaGetDevice(&ws->device));
    size_t bytes = 0;
    if (!grid_aligned(g)) {
        // the whole-volume convolution and per-node sampling replace the separable passes
        ws->general = true;
        const size_t vb = (size_t)3 * nvox(g->ref_dim) * 4;
        ws->vox_bytes = vb;
        if (ws_alloc(&ws->general_vox, vb, ws->st) != cudaSuccess) {
            cudaGetLastError();
            return fail(NRB_ERR_OOM, "workspace allocation failed");
        }
        bytes += vb;
        for (int d = 0; d < 3; ++d) {
            ws->ax[d] = AxisSampling{};
            ws->ax[d].samples.assign(1, 0);
            ws->ax[d].nsamples = 1;
        }
    } else {
        NRB_TRY(make_sampling(g, ws->ax));
    }
    cudaStream_t st = ws->st;
    // the sampling tables: one allocation and one copy (its host image lives as long as the
    // workspace, so the stream-ordered copy may finish later)
    Arena t;
    size_t at[3][4];
    for (int d = 0; d < 3; ++d) {
        const AxisSampling& x = ws->ax[d];
        at[d][0] = t.add(x.samples.size() * sizeof(int));
        at[d][1] = t.add(x.tap_slot.size() * sizeof(int));
        at[d][2] = t.add(x.tap_weight.size() * sizeof(float));
        at[d][3] = t.add(x.kernel.size() * sizeof(float));
    }
    ws->table_host.assign(t.bytes, 0);
    // scratch: one allocation
    const long long ny = g->ref_dim[1], nz = g->ref_dim[2];
    const long long c1 = 3LL * nz * ny * ws->ax[0].nsamples;
    const long long c2 = 3LL * nz * ws->ax[1].nsamples * ws->ax[0].nsamples;
    const long long c3 = 3LL * ws->ax[2].nsamples * ws->ax[1].nsamples * ws->ax[0].nsamples;
    const size_t be_bytes = (size_t)18 * BePad(g->cpp_dim[0], g->cpp_dim[1], g->cpp_dim[2]).size * 4;
    Arena m;
    const size_t o_conv1 = m.add((size_t)std::max(c1, c3) * 4), o_conv2 = m.add((size_t)c2 * 4), o_be = m.add(be_bytes);
    const size_t o_red = m.add(2 * NRB_RED_BLOCKS * sizeof(double)), o_bep = m.add(NRB_RED_BLOCKS * sizeof(double));
    const size_t o_fred = m.add(2 * NRB_RED_BLOCKS * sizeof(float));
    ws->scratch_bytes = m.bytes;
    if (ws_alloc(&ws->tables, t.bytes, st) != cudaSuccess || ws_alloc(&ws->scratch, m.bytes, st) != cudaSuccess) {
        cudaGetLastError();
        return fail(NRB_ERR_OOM, "workspace allocation failed");
    }
    for (int d = 0; d < 3; ++d) {
        const AxisSampling& x = ws->ax[d];
        char *h = ws->table_host.data();
        auto put = [&](size_t off, const void *src, size_t n) {
            if (n) memcpy(h + off, src, n);
        };
        put(at[d][0], x.samples.data(), x.samples.size() * sizeof(int));
        put(at[d][1], x.tap_slot.data(), x.tap_slot.size() * sizeof(int));
        put(at[d][2], x.tap_weight.data(), x.tap_weight.size() * sizeof(float));
        put(at[d][3], x.kernel.data(), x.kernel.size() * sizeof(float));
        ws->d_samples[d] = reinterpret_cast<int *>(ws->tables + at[d][0]);
        ws->d_tap_slot[d] = reinterpret_cast<int *>(ws->tables + at[d][1]);
        ws->d_tap_weight[d] = reinterpret_cast<float *>(ws->tables + at[d][2]);
        ws->d_kernel[d] = reinterpret_cast<float *>(ws->tables + at[d][3]);
    }
    ws->conv1 = reinterpret_cast<float *>(ws->scratch + o_conv1);
    ws->conv2 = reinterpret_cast<float *>(ws->scratch + o_conv2);
    ws->be_deriv = reinterpret_cast<float *>(ws->scratch + o_be);
    ws->red = reinterpret_cast<double *>(ws->scratch + o_red);
    ws->be_partials = reinterpret_cast<double *>(ws->scratch + o_bep);
    ws->fred = reinterpret_cast<float *>(ws->scratch + o_fred);
    NRB_CUDA(cudaMemcpyAsync(ws->tables, ws->table_host.data(), t.bytes, cudaMemcpyHostToDevice, st));
    // the ring of zeros around every derivative plane
    NRB_CUDA(cudaMemsetAsync(ws->be_deriv, 0, be_bytes, st));
    if (!st) NRB_CUDA(cudaStreamSynchronize(st));  // the workspace may be used on any stream at once
    ws->bytes = bytes + t.bytes + m.bytes;
    NRB_CUDA(cudaStreamCreateWithFlags(&ws->side, cudaStreamNonBlocking));
    NRB_CUDA(cudaEventCreateWithFlags(&ws->ev_fork, cudaEventDisableTiming));
    NRB_CUDA(cudaEventCreateWithFlags(&ws->ev_join, cudaEventDisableTiming));
    return NRB_OK;
}

nrb_status fork_side(nrb_workspace *ws, cudaStream_t st) {
    NRB_CUDA(cudaEventRecord(ws->ev_fork, st));
    NRB_CUDA(cudaStreamWaitEvent(ws->side, ws->ev_fork, 0));
    return NRB_OK;
}

nrb_status join_side(nrb_workspace *ws, cudaStream_t st) {
    NRB_CUDA(cudaEventRecord(ws->ev_join, ws->side));
    NRB_CUDA(cudaStreamWaitEvent(st, ws->ev_join, 0));
    return NRB_OK;
}

void workspace_free(nrb_workspace *ws) {
    cudaStream_t st = ws->st;
    if (st) {
        dev_free(ws->tables, st);
        dev_free(ws->scratch, st);
        dev_free(ws->general_vox, st);
    } else {
        int cur = ws->device;
        cudaGetDevice(&cur);
        if (cur != ws->device) cudaSetDevice(ws->device);
        cudaDeviceSynchronize();
        auto give_back = [](void *p, size_t bytes) {
            if (p && ws_plain(bytes, nullptr)) cudaFree(p);
            else if (p) cudaFreeAsync(p, nullptr);
        };
        give_back(ws->tables, 0);  // a few entries per node and axis
        give_back(ws->scratch, ws->scratch_bytes);
        give_back(ws->general_vox, ws->vox_bytes);
        if (cur != ws->device) cudaSetDevice(cur);
    }
    // the side stream's work is ordered before st's last join; its frees above are on st
    if (ws->ev_fork) cudaEventDestroy(ws->ev_fork);
    if (ws->ev_join) cudaEventDestroy(ws->ev_join);
    if (ws->side) cudaStreamDestroy(ws->side);
}

static int be_grid(const nrb_geometry *g) {
    const long long ni = (long long)std::max(0, g->cpp_dim[0] - 2) * std::max(0, g->cpp_dim[1] - 2) *
                         std::max(0, g->cpp_dim[2] - 2);
    return (int)std::max<long long>(1, std::min<long long>((ni + NRB_RED_THREADS - 1) / NRB_RED_THREADS, NRB_RED_BLOCKS));
}

nrb_status launch_be_value(nrb_workspace *ws, const nrb_geometry *g, const float *cpp, cudaStream_t st,
                           const float *grad, const OptState *step) {
    const int grid = be_grid(g);
    KernelTimer timer(TK_BE_VALUE, 12.0 * (double)nvox(g->cpp_dim), st);
    k_be_value<<<grid, 3 * NRB_RED_THREADS, 0, st>>>(g->cpp_dim[0], g->cpp_dim[1], g->cpp_dim[2], cpp, be_basis(),
                                                  ws->be_partials, grad, step);
    NRB_LAUNCHED("k_be_value");
    return NRB_OK;
}

int be_partial_count(const nrb_geometry *g) { return be_grid(g); }

nrb_status voxel_to_node_general(const float *vox, const nrb_geometry *g, float weight, float *node,
                                 cudaStream_t st);

// The node convolution serves rows and kernels up to the extent it has always served (24 rows of
// the volume, the taps and one float per sample in 227 KB)
static nrb_status conv_supported(int nx, int R, int ns) {
    if (((size_t)24 * nx + 2 * R + 1 + ns) * 4 > 227 * 1024)
        return fail(NRB_ERR_UNSUPPORTED, "convolution: rows and kernel exceed shared memory");
    return NRB_OK;
}
// radii and taps of the axes: taps further out than a line is long meet no voxel and are left out,
// which bounds what a block stages
static void conv_kernels(const nrb_workspace *ws, const nrb_geometry *g, int R[3], const float *K[3]) {
    for (int i = 0; i < 3; ++i) {
        R[i] = std::min(ws->ax[i].radius, g->ref_dim[i] - 1);
        K[i] = ws->d_kernel[i] + (ws->ax[i].radius - R[i]);
    }
}
// opts a convolution kernel into its shared memory (CONV_SHARED_MAX)
template <typename K>
static nrb_status conv_smem(K kernel, size_t bytes) {
    if (bytes > CONV_SHARED_MAX) return fail(NRB_ERR_UNSUPPORTED, "convolution: rows and kernel exceed shared memory");
    if (bytes + CONV_STATIC_BYTES > 48 * 1024)
        NRB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CONV_SHARED_MAX));
    return NRB_OK;
}

nrb_status launch_convolve_to_nodes(nrb_workspace *ws, const nrb_geometry *g, const float *vgrad,
                                    float weight, float *node, cudaStream_t st) {
    if (ws->general) {
        // Compute::ConvolveVoxelBasedMeasureGradient (reg-lib/Compute.cpp:230-281) as written:
        // the whole gradient convolved along the image axes with the grid spacings, then every
        // node sampled through the full node -> voxel matrix
        KernelTimer timer(TK_CONV, 0.0, st);
        const long long nv = nvox(g->ref_dim);
        NRB_CUDA(cudaMemcpyAsync(ws->general_vox, vgrad, 3 * nv * sizeof(float), cudaMemcpyDeviceToDevice, st));
        for (int axis = 0; axis < 3; ++axis)
            NRB_TRY(nrb_kernel_convolution_cubic(ws->general_vox, 3, g->ref_dim, g->ref_pixdim, g->cpp_pixdim[axis],
                                                 axis, st));
        return voxel_to_node_general(ws->general_vox, g, weight, node, st);
    }
    const int nx = g->ref_dim[0], ny = g->ref_dim[1], nz = g->ref_dim[2];
    const int nsx = ws->ax[0].nsamples, nsy = ws->ax[1].nsamples, nsz = ws->ax[2].nsamples;
    // compulsory traffic of the whole voxel->node step: the voxel gradient once, the nodes once
    KernelTimer timer(TK_CONV, 12.0 * (double)nx * ny * nz + 12.0 * (double)nvox(g->cpp_dim), st);
    NRB_TRY(conv_supported(nx, ws->ax[0].radius, nsx));
    int R[3];
    const float *K[3];
    conv_kernels(ws, g, R, K);
    // x pass: [3][nz][ny][nx] -> [3][nz][ny][nsx]
    const int rows = conv_x_rows(nx, R[0], nsx);
    const size_t xsm = conv_x_bytes(rows, nx, R[0], nsx);
    auto kx = rows == 32 ? k_conv_x<32> : rows == 16 ? k_conv_x<16> : rows == 8 ? k_conv_x<8> : k_conv_x<4>;
    NRB_TRY(conv_smem(kx, xsm));
    kx<<<(unsigned)conv_x_units(rows, ny, nz), CONV_X_THREADS, xsm, st>>>(nx, ny, nz, vgrad, ws->d_samples[0], nsx,
                                                                         K[0], R[0], ws->conv1);
    NRB_LAUNCHED("k_conv_x");
    // y pass: [3][nz][ny][nsx] -> [3][nz][nsy][nsx]
    if (conv_y_tile(ny, nsx, R[1], nsy, 3LL * nz)) {
        const size_t ysm = conv_y_bytes(ny, nsx, R[1], nsy);
        NRB_TRY(conv_smem(k_conv_y, ysm));
        k_conv_y<<<3 * nz * ConvY(ny, nsx, R[1]).chunks, CONV_Y_THREADS, ysm, st>>>(ny, nsx, ws->conv1, ws->d_samples[1], nsy,
                                                                                K[1], R[1], ws->conv2);
        NRB_LAUNCHED("k_conv_y");
    } else {
        const long long ey = 3LL * nz * nsy * nsx;
        k_conv_strided<<<(unsigned)((ey + 255) / 256), 256, 0, st>>>(ey, ny, nsx, ws->conv1, ws->d_samples[1], nsy, K[1],
                                                                     R[1], ws->conv2);
        NRB_LAUNCHED("k_conv_strided(y)");
    }
    // z pass: [3][nz][nsy * nsx] -> [3][nsz][nsy * nsx] (reuses conv1)
    const long long ez = 3LL * nsz * nsy * nsx;
    k_conv_strided<<<(unsigned)((ez + 255) / 256), 256, 0, st>>>(ez, nz, nsy * nsx, ws->conv2, ws->d_samples[2], nsz, K[2],
                                                                 R[2], ws->conv1);
    NRB_LAUNCHED("k_conv_strided(z)");
    // node sampling, reorientation (floating ijk) and weighting
    float w = weight;
    for (int i = 0; i < 3; ++i) w *= g->cpp_pixdim[i] / g->ref_pixdim[i];
    const long long nc = nvox(g->cpp_dim);
    k_nodes<<<grid_for(nc, 256), 256, 0, st>>>(g->cpp_dim[0], g->cpp_dim[1], g->cpp_dim[2], nsx, nsy, nsz, ws->conv1,
                                               ws->d_tap_slot[0], ws->d_tap_weight[0], ws->d_tap_slot[1],
                                               ws->d_tap_weight[1], ws->d_tap_slot[2], ws->d_tap_weight[2],
                                               to_mat34(g->flo_ijk), w, node);
    NRB_LAUNCHED("k_nodes");
    return NRB_OK;
}

}  // namespace nrb

using namespace nrb;

// ---------------------------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------------------------
nrb_status nrb::workspace_create_on(const nrb_geometry *g, cudaStream_t st, nrb_workspace **out) {
    if (!g || !out) return fail(NRB_ERR_INVALID, "nrb_workspace_create: null pointer");
    NRB_TRY(validate_geometry(g));
    nrb_workspace *ws = new nrb_workspace();
    ws->st = st;
    nrb_status s = workspace_init(ws, g);
    if (s == NRB_OK) s = workspace_alloc(ws);
    if (s != NRB_OK) {
        workspace_free(ws);
        delete ws;
        return s;
    }
    *out = ws;
    return NRB_OK;
}

extern "C" nrb_status nrb_workspace_create(const nrb_geometry *g, nrb_workspace **out) {
    if (!g || !out) return fail(NRB_ERR_INVALID, "nrb_workspace_create: null pointer");
    NRB_TRY(validate_geometry(g));
    nrb_workspace *ws = new nrb_workspace();
    nrb_status s = workspace_init(ws, g);
    if (s == NRB_OK) s = workspace_alloc(ws);
    if (s != NRB_OK) {
        workspace_free(ws);
        delete ws;
        return s;
    }
    *out = ws;
    return NRB_OK;
}

extern "C" void nrb_workspace_destroy(nrb_workspace *ws) {
    if (!ws) return;
    workspace_free(ws);
    delete ws;
}

extern "C" nrb_status nrb_convolve_voxel_based_gradient(nrb_workspace *ws, const nrb_geometry *g,
                                                        const float *vgrad, float weight,
                                                        float *node_grad, void *stream) {
    if (!ws || !g || !vgrad || !node_grad) return fail(NRB_ERR_INVALID, "nrb_convolve_voxel_based_gradient: null pointer");
    return launch_convolve_to_nodes(ws, g, vgrad, weight, node_grad, as_stream(stream));
}

extern "C" nrb_status nrb_kernel_convolution_cubic(float *img, int nvol, const int32_t dim[3],
                                                   const float pixdim[3], float spacing_mm, int axis,
                                                   void *stream) {
    if (!img || !dim || !pixdim || nvol <= 0 || axis < 0 || axis > 2)
        return fail(NRB_ERR_INVALID, "nrb_kernel_convolution_cubic: bad argument");
    cudaStream_t st = as_stream(stream);
    double temp = 0;
    int radius = 0;
    NRB_TRY(cubic_extent("nrb_kernel_convolution_cubic", spacing_mm, pixdim[axis], temp, radius));
    if (radius <= 0 || dim[axis] <= 1) return NRB_OK;  // the reference leaves the image as is
    std::vector<float> k(2 * radius + 1);
    cubic_taps(temp, radius, k.data());
    const long long nv = (long long)dim[0] * dim[1] * dim[2];
    if (2 * radius + 1 <= NRB_STATIC_CONV_MAX_TAPS && nv > 0) {
        ConvTaps taps;
        std::copy(k.begin(), k.end(), taps.k);
        nrb_status status = NRB_OK;
        if (conv_lines(img, nvol, dim, axis, taps, radius, st, &status)) return status;
    }
    float *dk = nullptr, *tv = nullptr, *td = nullptr;
    NRB_CUDA(tmp_alloc(&dk, k.size() * 4, st));
    NRB_CUDA(tmp_alloc(&tv, nv * 4, st));
    NRB_CUDA(tmp_alloc(&td, nv * 4, st));
    NRB_CUDA(cudaMemcpyAsync(dk, k.data(), k.size() * 4, cudaMemcpyHostToDevice, st));
    for (int t = 0; t < nvol; ++t) {
        float *v = img + t * nv;
        k_conv_axis<<<grid_for(nv, 256), 256, 0, st>>>(dim[0], dim[1], dim[2], axis, v, nullptr, dk, radius, tv, td);
        NRB_LAUNCHED("k_conv_axis");
        k_conv_normalise<<<grid_for(nv, 256), 256, 0, st>>>(nv, v, tv, td, v);
        NRB_LAUNCHED("k_conv_normalise");
    }
    NRB_CUDA(cudaFreeAsync(dk, st));
    NRB_CUDA(cudaFreeAsync(tv, st));
    NRB_CUDA(cudaFreeAsync(td, st));
    return NRB_OK;
}

// ---------------------------------------------------------------------------------------------
// The same convolution with its scratch in a fixed, module-level device array.
//
// Some callers cannot allocate device memory at the moment they need this convolution: code
// that is recording a CUDA stream capture (an allocation there either fails or becomes part of
// the graph), code running under a hard per-process memory cap that is already spent, or code
// that hands out device memory from its own pool and forbids the library from touching the
// driver's allocator. For them the scratch (the kernel taps and the value/density pair of one
// volume) lives in `g_static_scratch`, which the module reserves when it is loaded.
//
// Layout: [taps: NRB_STATIC_CONV_MAX_TAPS floats, padded to 256 B][value: max voxels floats]
// [density: max voxels floats]. Nothing in it has to start at zero: every call writes the taps
// and then both temporaries of a volume in full before it reads them.
//
// There is one scratch per device and no lock: two calls whose kernels can overlap on the same
// device (different streams without ordering, or different host threads) race on it.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr size_t kStaticTapBytes = 256 * ((NRB_STATIC_CONV_MAX_TAPS * sizeof(float) + 255) / 256);
constexpr size_t kStaticScratchBytes = kStaticTapBytes + 2 * sizeof(float) * (size_t)NRB_STATIC_CONV_MAX_VOXELS;

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// the taps travel as a kernel argument, so no host-to-device copy is needed for them
__global__ void k_static_taps(const __grid_constant__ ConvTaps t, int n, float *__restrict__ dst) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = t.k[i];
}

// Address of this device's scratch. cudaGetSymbolAddress runs once per device, with that device
// current (the caller's current device); later calls read the cached pointer.
constexpr int kMaxDevices = 64;
std::mutex g_static_mutex;
unsigned char *g_static_addr[kMaxDevices] = {};

nrb_status static_scratch(unsigned char **out) {
    int dev = 0;
    NRB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(NRB_ERR_UNSUPPORTED, "static scratch: device index above 63");
    std::lock_guard<std::mutex> lock(g_static_mutex);
    if (!g_static_addr[dev]) {
        void *p = nullptr;
        NRB_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
        g_static_addr[dev] = static_cast<unsigned char *>(p);
    }
    *out = g_static_addr[dev];
    return NRB_OK;
}

}  // namespace

extern "C" nrb_status nrb_kernel_convolution_cubic_static(float *img, int nvol, const int32_t dim[3],
                                                          const float pixdim[3], float spacing_mm, int axis,
                                                          void *stream) {
    if (!img || !dim || !pixdim || nvol <= 0 || axis < 0 || axis > 2 || dim[0] <= 0 || dim[1] <= 0 || dim[2] <= 0)
        return fail(NRB_ERR_INVALID, "nrb_kernel_convolution_cubic_static: bad argument");
    const long long nv = (long long)dim[0] * dim[1] * dim[2];
    if (nv > NRB_STATIC_CONV_MAX_VOXELS)
        return fail(NRB_ERR_UNSUPPORTED, "nrb_kernel_convolution_cubic_static: volume has more voxels than the "
                                         "static scratch holds (NRB_STATIC_CONV_MAX_VOXELS = 2097152)");
    double temp = 0;
    int radius = 0;
    NRB_TRY(cubic_extent("nrb_kernel_convolution_cubic_static", spacing_mm, pixdim[axis], temp, radius));
    // the same early return as the allocating entry point, before the size limit on the taps
    if (radius <= 0 || dim[axis] <= 1) return NRB_OK;  // the reference leaves the image as is
    if (2 * radius + 1 > NRB_STATIC_CONV_MAX_TAPS)
        return fail(NRB_ERR_UNSUPPORTED, "nrb_kernel_convolution_cubic_static: kernel wider than the static "
                                         "scratch holds (NRB_STATIC_CONV_MAX_TAPS = 511 taps)");
    ConvTaps taps;
    cubic_taps(temp, radius, taps.k);
    nrb_status status = NRB_OK;
    if (conv_lines(img, nvol, dim, axis, taps, radius, as_stream(stream), &status)) return status;
    unsigned char *base = nullptr;
    NRB_TRY(static_scratch(&base));
    float *dk = reinterpret_cast<float *>(base);
    float *tv = reinterpret_cast<float *>(base + kStaticTapBytes);
    float *td = tv + NRB_STATIC_CONV_MAX_VOXELS;
    cudaStream_t st = as_stream(stream);
    k_static_taps<<<1, 256, 0, st>>>(taps, 2 * radius + 1, dk);
    NRB_LAUNCHED("k_static_taps");
    for (int t = 0; t < nvol; ++t) {
        float *v = img + t * nv;
        k_conv_axis<<<grid_for(nv, 256), 256, 0, st>>>(dim[0], dim[1], dim[2], axis, v, nullptr, dk, radius, tv, td);
        NRB_LAUNCHED("k_conv_axis");
        k_conv_normalise<<<grid_for(nv, 256), 256, 0, st>>>(nv, v, tv, td, v);
        NRB_LAUNCHED("k_conv_normalise");
    }
    return NRB_OK;
}

extern "C" nrb_status nrb_approx_bending_energy(nrb_workspace *ws, const nrb_geometry *g, const float *cpp,
                                                nrb_objective *obj, double *be_host, void *stream) {
    if (!ws || !g || !cpp) return fail(NRB_ERR_INVALID, "nrb_approx_bending_energy: null pointer");
    cudaStream_t st = as_stream(stream);
    NRB_TRY(launch_be_value(ws, g, cpp, st));
    nrb_objective *o = obj;
    nrb_objective *tmp = nullptr;
    if (!o) {
        NRB_CUDA(tmp_alloc(&tmp, sizeof(nrb_objective), st));
        o = tmp;
    }
    k_be_sum<<<1, NRB_RED_THREADS, 0, st>>>(ws->be_partials, be_grid(g), 3.0 * (double)nvox(g->cpp_dim), o);
    NRB_LAUNCHED("k_be_sum");
    if (be_host) NRB_TRY(read_back(be_host, &o->be, sizeof(double), st));
    if (tmp) NRB_CUDA(cudaFreeAsync(tmp, st));
    return NRB_OK;
}

namespace nrb {
// reg_spline_approxBendingEnergyGradient3D, first half: the 18 second-derivative values of
// every node (grid read, derivatives written)
static nrb_status be_derivatives(const nrb_geometry *g, const float *cpp, float *der, cudaStream_t st) {
    const long long nc = nvox(g->cpp_dim);
    KernelTimer timer(TK_BE_GRADIENT, (12.0 + 72.0) * (double)nc, st);
    k_be_derivatives<<<dim3(grid_for(nc, 128), 3), 128, 0, st>>>(g->cpp_dim[0], g->cpp_dim[1], g->cpp_dim[2],
                                                        to_mat34(g->cpp_xyz), cpp, be_basis(), der);
    NRB_LAUNCHED("k_be_derivatives");
    return NRB_OK;
}

// second half: the adjoint stencil, node_grad += weight / #nodes * sum (derivatives read,
// gradient read-modify-write)
static nrb_status be_accumulate(const nrb_geometry *g, const float *der, float weight, float *node_grad, cudaStream_t st) {
    const long long nc = nvox(g->cpp_dim);
    KernelTimer timer(TK_BE_GRADIENT, (72.0 + 24.0) * (double)nc, st);
    const float ratio = weight / (float)nc;
    k_be_accumulate<<<dim3(grid_for(nc, 128), 3), 128, 0, st>>>(g->cpp_dim[0], g->cpp_dim[1], g->cpp_dim[2], der, be_basis(),
                                                       ratio, node_grad);
    NRB_LAUNCHED("k_be_accumulate");
    return NRB_OK;
}

nrb_status launch_be_derivatives(nrb_workspace *ws, const nrb_geometry *g, const float *cpp, cudaStream_t st) {
    return be_derivatives(g, cpp, ws->be_deriv, st);
}
nrb_status launch_be_accumulate(nrb_workspace *ws, const nrb_geometry *g, float weight, float *node_grad,
                                cudaStream_t st) {
    return be_accumulate(g, ws->be_deriv, weight, node_grad, st);
}

// Both halves. The workspace's derivative planes fit the grid that it was made for, with zeros around
// that grid alone; the planes of any other grid are the call's own.
nrb_status be_gradient(nrb_workspace *ws, const nrb_geometry *g, const float *cpp, float weight, float *node_grad,
                       cudaStream_t st) {
    if (std::equal(g->cpp_dim, g->cpp_dim + 3, ws->g.cpp_dim)) {
        NRB_TRY(launch_be_derivatives(ws, g, cpp, st));
        return launch_be_accumulate(ws, g, weight, node_grad, st);
    }
    float *der = nullptr;
    const size_t bytes = (size_t)18 * BePad(g->cpp_dim[0], g->cpp_dim[1], g->cpp_dim[2]).size * 4;
    NRB_CUDA(tmp_alloc(&der, bytes, st));
    nrb_status s = check_cuda(cudaMemsetAsync(der, 0, bytes, st), "cudaMemsetAsync");
    if (s == NRB_OK) s = be_derivatives(g, cpp, der, st);
    if (s == NRB_OK) s = be_accumulate(g, der, weight, node_grad, st);
    cudaFreeAsync(der, st);
    return s;
}

// ---- batched levels -------------------------------------------------------------------------
// A pair's node-stage description: its workspace's convolution sampling and bending-energy
// buffers, as launch_convolve_to_nodes / launch_be_* use them for its geometry.
nrb_status batch_node_stage(const nrb_workspace *ws, const nrb_geometry *g, float sim_weight, float be_weight,
                            BatchPair& b) {
    if (ws->general) return fail(NRB_ERR_UNSUPPORTED, "batched level: the grid must be aligned with the reference");
    for (int i = 0; i < 3; ++i) {
        b.rdim[i] = g->ref_dim[i];
        b.cdim[i] = g->cpp_dim[i];
        b.ns[i] = ws->ax[i].nsamples;
        b.samples[i] = ws->d_samples[i];
        b.tap_slot[i] = ws->d_tap_slot[i];
        b.tap_weight[i] = ws->d_tap_weight[i];
    }
    NRB_TRY(conv_supported(b.rdim[0], ws->ax[0].radius, b.ns[0]));
    conv_kernels(ws, g, b.radius, b.kernel);
    b.nnode = nvox(g->cpp_dim);
    b.conv1 = ws->conv1;
    b.conv2 = ws->conv2;
    float w = sim_weight;
    for (int i = 0; i < 3; ++i) w *= g->cpp_pixdim[i] / g->ref_pixdim[i];
    b.node_weight = w;
    b.flo_ijk = to_mat34(g->flo_ijk);
    b.grid_xyz = to_mat34(g->cpp_xyz);
    b.be_partials = ws->be_partials;
    b.n_be = be_grid(g);
    b.be_norm = 3.0 * (double)b.nnode;
    b.be_der = ws->be_deriv;
    b.be_ratio = be_weight / (float)b.nnode;
    b.red = ws->red;
    return NRB_OK;
}

static int batch_grid(const std::vector<BatchPair>& pairs, long long (*units)(const BatchPair&), int threads,
                      int max_per_sm) {
    long long total = 0;
    for (const BatchPair& b : pairs) total += units(b);
    return grid_for(std::max(1LL, total), threads, max_per_sm);
}

nrb_status launch_batch_be_value(const std::vector<BatchPair>& hp, const BatchPair *d, const OptState *states,
                                 cudaStream_t st) {
    long long units = 0;
    for (const BatchPair& b : hp) units += b.n_be;
    const int grid = (int)std::max(1LL, std::min(units, 2LL * sm_count()));
    KernelTimer timer(TK_BE_VALUE, 0.0, st);
    k_b_be_value<<<grid, 3 * NRB_RED_THREADS, 0, st>>>(d, states, (int)hp.size(), be_basis());
    NRB_CUDA(cudaGetLastError());
    NRB_LAUNCHED("k_b_be_value");
    return NRB_OK;
}

static auto batch_conv_x(int rows) {
    return rows == 32 ? k_b_conv_x<32> : rows == 16 ? k_b_conv_x<16> : rows == 8 ? k_b_conv_x<8> : k_b_conv_x<4>;
}

// Rows, shared memory and grids of the convolution passes for the largest pair, opted into before a
// capture begins (a launch refused inside one would abort the level)
nrb_status batch_node_plan(const std::vector<BatchPair>& hp, BatchLaunch& L) {
    long long xb = 0, yb = 0, ye = 0, ze = 0, slices = 0;
    L.conv_rows = 32;
    L.conv_xsm = L.conv_ysm = 0;
    L.conv_ytile = true;
    for (const BatchPair& b : hp) L.conv_rows = std::min(L.conv_rows, conv_x_rows(b.rdim[0], b.radius[0], b.ns[0]));
    for (const BatchPair& b : hp) {
        L.conv_xsm = std::max(L.conv_xsm, conv_x_bytes(L.conv_rows, b.rdim[0], b.radius[0], b.ns[0]));
        L.conv_ysm = std::max(L.conv_ysm, conv_y_bytes(b.rdim[1], b.ns[0], b.radius[1], b.ns[1]));
        xb += conv_x_units(L.conv_rows, b.rdim[1], b.rdim[2]);
        yb += 3LL * b.rdim[2] * ConvY(b.rdim[1], b.ns[0], b.radius[1]).chunks;
        slices += 3LL * b.rdim[2];
        ye += 3LL * b.rdim[2] * b.ns[1] * b.ns[0];
        ze += 3LL * b.ns[2] * b.ns[1] * b.ns[0];
    }
    auto plan = [](auto kernel, long long units, int threads, size_t smem, int& grid) -> nrb_status {
        int per = 0;
        NRB_TRY(conv_smem(kernel, smem));
        NRB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem));
        if (per < 1) return fail(NRB_ERR_UNSUPPORTED, "batched level: the convolution does not fit in shared memory");
        grid = (int)std::max(1LL, std::min(units, (long long)per * sm_count()));
        return NRB_OK;
    };
    NRB_TRY(plan(batch_conv_x(L.conv_rows), xb, CONV_X_THREADS, L.conv_xsm, L.conv_xgrid));
    for (const BatchPair& b : hp)
        L.conv_ytile = L.conv_ytile && conv_y_tile(b.rdim[1], b.ns[0], b.radius[1], b.ns[1], slices);
    if (L.conv_ytile) NRB_TRY(plan(k_b_conv_y, yb, CONV_Y_THREADS, L.conv_ysm, L.conv_ygrid));
    else L.conv_ygrid = grid_for(std::max(1LL, ye), 256);
    L.conv_zgrid = grid_for(std::max(1LL, ze), 256);
    return NRB_OK;
}

nrb_status launch_batch_node_stage(const std::vector<BatchPair>& hp, const BatchLaunch& L, const BatchPair *d,
                                   const OptState *states, cudaStream_t st, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join,
                                   nrb_status (*gradient)(const BatchPair *, const OptState *, cudaStream_t, void *),
                                   void *gradient_arg) {
    const int np = (int)hp.size();
    const bool be = hp[0].be_w > 0;
    // bending-energy derivatives on the side branch, beside the voxel passes (they read best only)
    if (be) {
        NRB_CUDA(cudaEventRecord(fork, st));
        NRB_CUDA(cudaStreamWaitEvent(side, fork, 0));
        const int g = batch_grid(hp, [](const BatchPair& b) { return 3 * b.nnode; }, 128, 16);
        KernelTimer timer(TK_BE_GRADIENT, 0.0, side);
        k_b_be_derivatives<<<g, 128, 0, side>>>(d, states, np, be_basis());
        NRB_CUDA(cudaGetLastError());
        NRB_LAUNCHED("k_b_be_derivatives");
    }
    NRB_TRY(gradient(d, states, st, gradient_arg));
    {
    KernelTimer timer(TK_CONV, 0.0, st);
    batch_conv_x(L.conv_rows)<<<L.conv_xgrid, CONV_X_THREADS, L.conv_xsm, st>>>(d, states, np);
    NRB_CUDA(cudaGetLastError());
    NRB_LAUNCHED("k_b_conv_x");
    if (L.conv_ytile) k_b_conv_y<<<L.conv_ygrid, CONV_Y_THREADS, L.conv_ysm, st>>>(d, states, np);
    else k_b_conv_strided<1><<<L.conv_ygrid, 256, 0, st>>>(d, states, np);
    NRB_CUDA(cudaGetLastError());
    NRB_LAUNCHED("k_b_conv_y");
    k_b_conv_strided<2><<<L.conv_zgrid, 256, 0, st>>>(d, states, np);
    NRB_CUDA(cudaGetLastError());
    NRB_LAUNCHED("k_b_conv_strided(z)");
    const int gn = batch_grid(hp, [](const BatchPair& b) { return b.nnode; }, 256, 16);
    k_b_nodes<<<gn, 256, 0, st>>>(d, states, np);
    NRB_CUDA(cudaGetLastError());
    NRB_LAUNCHED("k_b_nodes");
    }
    if (be) {
        NRB_CUDA(cudaEventRecord(join, side));
        NRB_CUDA(cudaStreamWaitEvent(st, join, 0));
        const int g = batch_grid(hp, [](const BatchPair& b) { return 3 * b.nnode; }, 128, 16);
        KernelTimer timer2(TK_BE_GRADIENT, 0.0, st);
        k_b_be_accumulate<<<g, 128, 0, st>>>(d, states, np, be_basis());
        NRB_CUDA(cudaGetLastError());
        NRB_LAUNCHED("k_b_be_accumulate");
    }
    return NRB_OK;
}
}  // namespace nrb

extern "C" nrb_status nrb_approx_bending_energy_gradient(nrb_workspace *ws, const nrb_geometry *g,
                                                         const float *cpp, float weight, float *node_grad,
                                                         void *stream) {
    if (!ws || !g || !cpp || !node_grad) return fail(NRB_ERR_INVALID, "nrb_approx_bending_energy_gradient: null pointer");
    return be_gradient(ws, g, cpp, weight, node_grad, as_stream(stream));
}

// fred holds two partial arrays of NRB_RED_BLOCKS floats (min | max)
static nrb_status rescale_impl(float *img, int64_t n, float lo, float hi, float *fred, cudaStream_t st) {
    const int np = (int)std::max<long long>(1, std::min<long long>((n + 8 * NRB_RED_THREADS - 1) / (8 * NRB_RED_THREADS), NRB_RED_BLOCKS));
    k_minmax<<<np, 2 * NRB_RED_THREADS, 0, st>>>(n, img, fred, fred + NRB_RED_BLOCKS);
    NRB_LAUNCHED("k_minmax");
    k_rescale<<<grid_for((n + 3) / 4, 256, 8), 256, 0, st>>>(n, img, fred, fred + NRB_RED_BLOCKS, np, lo, hi);
    NRB_LAUNCHED("k_rescale");
    return NRB_OK;
}

namespace nrb {
nrb_status rescale_with(float *img, int64_t n, float lo, float hi, float *fred, cudaStream_t st) {
    return rescale_impl(img, n, lo, hi, fred, st);
}
}  // namespace nrb

extern "C" nrb_status nrb_intensity_rescale(float *img, int64_t nvox_, float new_min, float new_max, void *stream) {
    if (!img || nvox_ <= 0) return fail(NRB_ERR_INVALID, "nrb_intensity_rescale: bad argument");
    cudaStream_t st = as_stream(stream);
    float *fred = nullptr;
    NRB_CUDA(tmp_alloc(&fred, 2 * NRB_RED_BLOCKS * sizeof(float), st));
    NRB_TRY(rescale_impl(img, nvox_, new_min, new_max, fred, st));
    NRB_CUDA(cudaFreeAsync(fred, st));
    return NRB_OK;
}

extern "C" nrb_status nrb_get_maximal_length(const float *node_grad, int64_t nnode, nrb_objective *obj,
                                             double *max_host, void *stream) {
    if (!node_grad || nnode <= 0) return fail(NRB_ERR_INVALID, "nrb_get_maximal_length: bad argument");
    cudaStream_t st = as_stream(stream);
    const int np = (int)std::max<long long>(1, std::min<long long>((nnode + NRB_RED_THREADS - 1) / NRB_RED_THREADS, NRB_RED_BLOCKS));
    float *pm = nullptr;
    double *dm = nullptr;
    NRB_CUDA(tmp_alloc(&pm, np * sizeof(float), st));
    NRB_CUDA(tmp_alloc(&dm, sizeof(double), st));
    k_maxlen<<<np, NRB_RED_THREADS, 0, st>>>(nnode, node_grad, pm);
    NRB_LAUNCHED("k_maxlen");
    k_maxlen_finish<<<1, NRB_RED_BLOCKS, 0, st>>>(pm, np, obj, dm);
    NRB_LAUNCHED("k_maxlen_finish");
    if (max_host) NRB_TRY(read_back(max_host, dm, sizeof(double), st));
    NRB_CUDA(cudaFreeAsync(pm, st));
    NRB_CUDA(cudaFreeAsync(dm, st));
    return NRB_OK;
}

namespace nrb {
// max length into obj->max_grad_len then normalisation by it, scratch from the workspace
// UpdateGradientValues with the first-call branch taken on the device (flag read at run time)
nrb_status cg_update_flagged(nrb_workspace *ws, float *grad, float *g1, float *g2, int64_t n, const int *first_call,
                             cudaStream_t st) {
    const int np = (int)std::max<long long>(1, std::min<long long>((n + NRB_RED_THREADS - 1) / NRB_RED_THREADS, NRB_RED_BLOCKS));
    k_cg_dots<<<np, NRB_RED_THREADS, 0, st>>>(n, grad, g1, g2, ws->red);
    NRB_LAUNCHED("k_cg_dots");
    k_cg_update<<<grid_for(n, 256), 256, 0, st>>>(n, grad, g1, g2, ws->red, np, first_call);
    NRB_LAUNCHED("k_cg_update");
    return NRB_OK;
}

nrb_status max_and_normalise(nrb_workspace *ws, float *grad, int64_t nnode, nrb_objective *obj, cudaStream_t st) {
    const int np = (int)std::max<long long>(1, std::min<long long>((nnode + NRB_RED_THREADS - 1) / NRB_RED_THREADS, NRB_RED_BLOCKS));
    k_maxlen<<<np, NRB_RED_THREADS, 0, st>>>(nnode, grad, ws->fred);
    NRB_LAUNCHED("k_maxlen");
    k_maxlen_finish<<<1, NRB_RED_BLOCKS, 0, st>>>(ws->fred, np, obj, nullptr);
    NRB_LAUNCHED("k_maxlen_finish");
    k_normalise<<<grid_for(3 * nnode, 256), 256, 0, st>>>(3 * nnode, grad, obj, -1.0);
    NRB_LAUNCHED("k_normalise");
    return NRB_OK;
}
}  // namespace nrb

extern "C" nrb_status nrb_normalise_gradient(float *node_grad, int64_t nnode, double max_len,
                                             const nrb_objective *obj, void *stream) {
    if (!node_grad || nnode <= 0 || (max_len < 0 && !obj))
        return fail(NRB_ERR_INVALID, "nrb_normalise_gradient: bad argument");
    k_normalise<<<grid_for(3 * nnode, 256), 256, 0, as_stream(stream)>>>(3 * nnode, node_grad, obj, max_len);
    NRB_LAUNCHED("k_normalise");
    return NRB_OK;
}

extern "C" nrb_status nrb_update_control_point_position(float *cur, const float *best, const float *grad,
                                                        float scale, int64_t n, void *stream) {
    if (!cur || !best || !grad || n <= 0) return fail(NRB_ERR_INVALID, "nrb_update_control_point_position: bad argument");
    k_update<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(n, cur, best, grad, scale);
    NRB_LAUNCHED("k_update");
    return NRB_OK;
}

extern "C" nrb_status nrb_conjugate_gradient(nrb_workspace *ws, float *grad, float *g1, float *g2, int64_t n,
                                             int first_call, void *stream) {
    if (!ws || !grad || !g1 || !g2 || n <= 0) return fail(NRB_ERR_INVALID, "nrb_conjugate_gradient: bad argument");
    cudaStream_t st = as_stream(stream);
    if (first_call) {
        k_cg_init<<<grid_for(n, 256), 256, 0, st>>>(n, grad, g1, g2);
        NRB_LAUNCHED("k_cg_init");
        return NRB_OK;
    }
    const int np = (int)std::max<long long>(1, std::min<long long>((n + NRB_RED_THREADS - 1) / NRB_RED_THREADS, NRB_RED_BLOCKS));
    k_cg_dots<<<np, NRB_RED_THREADS, 0, st>>>(n, grad, g1, g2, ws->red);
    NRB_LAUNCHED("k_cg_dots");
    k_cg_update<<<grid_for(n, 256), 256, 0, st>>>(n, grad, g1, g2, ws->red, np, nullptr);
    NRB_LAUNCHED("k_cg_update");
    return NRB_OK;
}

// ---------------------------------------------------------------------------------------------
// pyramid and grid helpers used by the registration driver
// ---------------------------------------------------------------------------------------------
namespace nrb {

// Whether new_xyz followed by old_ijk, rounded (k_downsample), takes every voxel i of the new image
// to i << shift: the composed map is within 0.05 voxel of that at the corners (it is affine), and the
// float evaluation's error stays far below the rest of the rounding margin. True for every header
// the pyramid derives by halving; a degenerate matrix fails it and takes the separate passes.
static bool samples_every_other(const int32_t idim[3], const int32_t odim[3], const float new_xyz[16],
                                const float old_ijk[16], int shift[3]) {
    double mm = 0, ij = 0;
    for (int i = 0; i < 12; ++i) {
        if (!std::isfinite(new_xyz[i]) || !std::isfinite(old_ijk[i])) return false;
        mm += std::fabs((double)new_xyz[i]) * (i % 4 < 3 ? odim[i % 4] : 1);
        ij = std::max(ij, std::fabs((double)old_ijk[i]));
    }
    double off = 0;
    for (int i = 0; i < 3; ++i) off = std::max(off, std::fabs((double)old_ijk[4 * i + 3]));
    if (!(16.0 * std::ldexp(1.0, -24) * (3.0 * ij * mm + off) < 0.2)) return false;
    for (int i = 0; i < 3; ++i) {
        shift[i] = odim[i] == idim[i] ? 0 : 1;
        if (((long long)(odim[i] - 1) << shift[i]) >= idim[i]) return false;
        double t = old_ijk[4 * i + 3];
        for (int k = 0; k < 3; ++k) t += (double)old_ijk[4 * i + k] * new_xyz[4 * k + 3];
        double dev = std::fabs(t);
        for (int j = 0; j < 3; ++j) {
            double m = 0;
            for (int k = 0; k < 3; ++k) m += (double)old_ijk[4 * i + k] * new_xyz[4 * k + j];
            dev += std::fabs(m - (i == j ? 1 << shift[i] : 0)) * (odim[j] - 1);
        }
        if (!(dev < 0.05)) return false;
    }
    return true;
}

// Gaussian smoothing of reg_downsampleImage (sigma = -0.7355 voxel, all three axes in one
// reg_tools_kernelConvolution call, density normalised once at the end), then nearest-neighbour
// downsampling.
nrb_status smooth_and_downsample(const float *in, const int32_t idim[3], float *out, const int32_t odim[3],
                                 const float new_xyz[16], const float old_ijk[16], cudaStream_t st) {
    const double temp = 0.7355;  // |sigma|, voxel units
    const int radius = (int)(temp * 3.0f);
    static_assert((int)(0.7355 * 3.0f) == SMOOTH_R, "the fused smoothing is written for this radius");
    std::vector<float> k(2 * radius + 1);
    for (int i = -radius; i <= radius; ++i)
        k[radius + i] = (float)(std::exp(-(double)(i * i) / (2.0 * temp * temp)) / (temp * 2.506628274631));
    SmoothParams P;
    // slices are addressed with 32-bit offsets in the fused pass
    if ((long long)idim[0] * idim[1] < (1LL << 31) && samples_every_other(idim, odim, new_xyz, old_ijk, P.s)) {
        for (int i = 0; i < 3; ++i) {
            P.n[i] = idim[i];
            P.o[i] = odim[i];
        }
        for (int i = 0; i < SMOOTH_TAPS; ++i) P.k[i] = k[i];
        const dim3 cols((odim[0] + SMOOTH_X - 1) / SMOOTH_X, (odim[1] + SMOOTH_Y - 1) / SMOOTH_Y);
        // runs of output slices: two rounds of resident blocks when the volume has that many, no
        // run shorter than 4 slices (the 2 * SMOOTH_R slices a run re-reads)
        const long long want = std::max<long long>(1, 2LL * 4 * sm_count() / ((long long)cols.x * cols.y));
        P.zrun = std::max(4, (int)((odim[2] + want - 1) / want));
        const unsigned runs = (unsigned)((odim[2] + P.zrun - 1) / P.zrun);
        if (cols.y <= 65535 && runs <= 65535) {
            auto kernel = P.s[0] && P.s[1] && P.s[2] ? k_smooth_downsample<true> : k_smooth_downsample<false>;
            kernel<<<dim3(cols.x, cols.y, runs), SMOOTH_THREADS, 0, st>>>(P, in, out);
            NRB_LAUNCHED("k_smooth_downsample");
            return NRB_OK;
        }
    }
    float *dk = nullptr, *tmp = nullptr;
    const long long nv = nvox(idim);
    NRB_CUDA(tmp_alloc(&dk, k.size() * 4, st));
    NRB_CUDA(tmp_alloc(&tmp, 4 * nv * sizeof(float), st));
    NRB_CUDA(cudaMemcpyAsync(dk, k.data(), k.size() * 4, cudaMemcpyHostToDevice, st));
    float *v0 = tmp, *d0 = tmp + nv, *v1 = tmp + 2 * nv, *d1 = tmp + 3 * nv;
    const int g = grid_for(nv, 256);
    k_conv_axis<<<g, 256, 0, st>>>(idim[0], idim[1], idim[2], 0, in, nullptr, dk, radius, v0, d0);
    NRB_LAUNCHED("k_conv_axis");
    k_conv_axis<<<g, 256, 0, st>>>(idim[0], idim[1], idim[2], 1, v0, d0, dk, radius, v1, d1);
    NRB_LAUNCHED("k_conv_axis");
    k_conv_axis<<<g, 256, 0, st>>>(idim[0], idim[1], idim[2], 2, v1, d1, dk, radius, v0, d0);
    NRB_LAUNCHED("k_conv_axis");
    k_conv_normalise<<<g, 256, 0, st>>>(nv, in, v0, d0, v1);
    NRB_LAUNCHED("k_conv_normalise");
    const long long no = nvox(odim);
    k_downsample<<<grid_for(no, 256), 256, 0, st>>>(odim[0], odim[1], odim[2], idim[0], idim[1], idim[2],
                                                    to_mat34(new_xyz), to_mat34(old_ijk), v1, out);
    NRB_LAUNCHED("k_downsample");
    NRB_CUDA(cudaFreeAsync(dk, st));
    NRB_CUDA(cudaFreeAsync(tmp, st));
    return NRB_OK;
}

nrb_status grid_identity(const int32_t cdim[3], const float cxyz[16], float *cpp, cudaStream_t st) {
    const long long nc = nvox(cdim);
    k_grid_identity<<<grid_for(nc, 256), 256, 0, st>>>(cdim[0], cdim[1], cdim[2], to_mat34(cxyz), cpp);
    NRB_LAUNCHED("k_grid_identity");
    return NRB_OK;
}

nrb_status grid_refine(const int32_t odim[3], const float *old, const int32_t ndim[3], float *out, cudaStream_t st) {
    const long long nc = nvox(ndim);
    k_grid_refine<<<grid_for(nc, 256), 256, 0, st>>>(odim[0], odim[1], odim[2], ndim[0], ndim[1], ndim[2], old, out);
    NRB_LAUNCHED("k_grid_refine");
    return NRB_OK;
}

}  // namespace nrb
