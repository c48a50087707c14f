// anl_common.cuh -- shared definitions of the anneal_gb300 CUDA library (sm_103a).
//
// Grid conventions follow the anneal voxel grid (fem.py:87-127): element
// e = i + nx*(j + ny*k), node n = i + (nx+1)*(j + (ny+1)*k), DOF = 3*n + c. Nodal vectors
// are stored interleaved (the three components of a node are adjacent), element fields
// are stored on the full grid with zeros on inactive elements.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <cstdio>
#include <algorithm>
#include <mutex>

#include "../../include/anneal_gb300.h"

namespace anl {

// ------------------------------------------------------------------ errors

#define ANL_CUDA(call)                                                                     \
    do {                                                                                   \
        cudaError_t _e = (call);                                                           \
        if (_e != cudaSuccess) {                                                           \
            anl::set_error("%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(_e)); \
            return ANL_ERR_CUDA;                                                           \
        }                                                                                  \
    } while (0)

// Every kernel launch of the library is followed by exactly one ANL_LAUNCH_CHECK, which
// also counts it (anl_launch_count).
#define ANL_LAUNCH_CHECK()                                                                 \
    do {                                                                                   \
        anl::count_launch();                                                               \
        cudaError_t _e = cudaGetLastError();                                               \
        if (_e != cudaSuccess) {                                                           \
            anl::set_error("%s:%d launch: %s", __FILE__, __LINE__, cudaGetErrorString(_e)); \
            return ANL_ERR_CUDA;                                                           \
        }                                                                                  \
    } while (0)

#define ANL_TRY(expr)                 \
    do {                              \
        int _s = (expr);              \
        if (_s != ANL_OK) return _s;  \
    } while (0)

void set_error(const char* fmt, ...);

// ------------------------------------------------------------------ debug bounds checks
//
// ANL_IN_RANGE(i, n) is `true` in the normal build. In the debug build (-DANL_DEBUG=1,
// `python -m anneal_gb300.build --debug`, loaded with ANL_DEBUG_LIB=1) it tests 0 <= i < n for
// a global-memory index before the access; a miss is counted in this translation unit's
// device record (the first miss keeps its index, extent and source line) and the caller skips
// the access, so a bad index is reported instead of touching memory out of range.
// anl_debug_oob collects the records of every unit. Without relocatable device code each
// unit has its own record: ANL_DEBUG_UNIT(name) defines the unit's reader.
#if ANL_DEBUG
struct OobRecord {
    unsigned long long count;
    long long index, extent, line;
};
static __device__ OobRecord g_oob;
__device__ __forceinline__ bool debug_in_range(long long i, long long n, int line) {
    if (i >= 0 && i < n) return true;
    if (atomicAdd(&g_oob.count, 1ull) == 0ull) {
        g_oob.index = i;
        g_oob.extent = n;
        g_oob.line = line;
    }
    return false;
}
#define ANL_IN_RANGE(i, n) ::anl::debug_in_range((long long)(i), (long long)(n), __LINE__)
// reads and clears this unit's record (host)
#define ANL_DEBUG_UNIT(name)                                                        \
    int debug_take_##name(unsigned long long* count, long long* first) {          \
        OobRecord r{}, z{};                                                          \
        ANL_CUDA(cudaMemcpyFromSymbol(&r, g_oob, sizeof(r)));                       \
        ANL_CUDA(cudaMemcpyToSymbol(g_oob, &z, sizeof(z)));                         \
        *count += r.count;                                                           \
        if (r.count && first[2] == 0) {                                              \
            first[0] = r.index;                                                      \
            first[1] = r.extent;                                                     \
            first[2] = r.line;                                                       \
        }                                                                            \
        return ANL_OK;                                                               \
    }
#else
#define ANL_IN_RANGE(i, n) true
#define ANL_DEBUG_UNIT(name)
#endif

// Held while a stream is captured into a CUDA graph and around every call that synchronises
// the whole device (cudaFree, cudaFreeHost, context set-up): such a call from another host
// thread would invalidate an ongoing capture, and several contexts may run in parallel
// threads (one per load case or per part).
std::recursive_mutex& device_sync_mutex();
void count_launch();
void count_launches(long long n);  // kernels replayed by a CUDA graph

// Grows a device buffer to at least `need` elements of `elem` bytes (contents are not kept).
template <class P>
inline int grow(P*& p, size_t& cap, size_t need, size_t elem) {
    if (need <= cap) return ANL_OK;
    std::lock_guard<std::recursive_mutex> lock(device_sync_mutex());
    cudaFree(p);
    p = nullptr;
    cap = 0;
    const size_t n = std::max<size_t>(need, 1);
    if (cudaMalloc((void**)&p, n * elem) != cudaSuccess) {
        cudaGetLastError();
        set_error("cudaMalloc of %zu bytes failed", n * elem);
        return ANL_ERR_NOMEM;
    }
    cap = n;
    return ANL_OK;
}

// ------------------------------------------------------------------ grid

struct Dims {
    int nx, ny, nz;  // elements
    __host__ __device__ int64_t ne() const { return (int64_t)nx * ny * nz; }
    __host__ __device__ int64_t nn() const { return (int64_t)(nx + 1) * (ny + 1) * (nz + 1); }
    __host__ __device__ int64_t node(int i, int j, int k) const {
        return (int64_t)i + (int64_t)(nx + 1) * ((int64_t)j + (int64_t)(ny + 1) * k);
    }
    __host__ __device__ int64_t elem(int i, int j, int k) const {
        return (int64_t)i + (int64_t)nx * ((int64_t)j + (int64_t)ny * k);
    }
};

// Node mask bits: bit c (c = 0,1,2) set when DOF c of the node is free; bit 3 set when the
// node is touched by an active element (fem.py:145-150).
enum : uint8_t { NODE_FREE_X = 1, NODE_FREE_Y = 2, NODE_FREE_Z = 4, NODE_USED = 8 };

// ------------------------------------------------------------------ element matrix

// The 24x24 hex8 stiffness of a unit cube (E = 1) has the reflection structure
//   Ke[a][b] (3x3 block) = S_a * B0(|p_b - p_a|) * S_a,   S_a = diag(1 - 2 p_a),
// with p_a the local position of node a in {0,1}^3, and every block row sums to zero
// (rigid translations store no energy). So 8 blocks B0(delta), delta in {0,1}^3, carry
// the whole matrix. blk[d] is B0(delta) with d = dx + 2 dy + 4 dz, row-major 3x3.
template <class T>
struct KeBlocks {
    T blk[8][9];
};

// Host: fills ke[576] (row-major) for a cube of side h (fem.py:71-84).
void hex8_ke(double nu, double h, double* ke);
// Host: extracts the 8 base blocks from ke and checks the reflection structure; returns
// the largest deviation found.
double ke_blocks(const double* ke, KeBlocks<double>* out);

// The same Ke in the basis of the 8 trilinear modes of a brick. A displacement component
// on the 8 corners p in {0,1}^3 is a combination of 1, sx, sy, sz, sx sy, sy sz, sz sx,
// sx sy sz (s = 2p - 1); its mode amplitudes beta_m = sum_p s_m(p) u_p are a Walsh-Hadamard
// transform. Ke u = T (KA / 64) T^T u with KA = T^T Ke T, and for an isotropic material KA
// is sparse: 45 non-zeros in 24 x 24, set by 8 numbers (the rigid translations, mode 1, carry
// none). So one element costs about 200 flops instead of the 1152 of the dense 24 x 24
// product, and the transform can be taken from edge differences u(p + e_d) - u(p), which
// keeps FP32 products proportional to the local strain, not to |u|.
// Constants (of KA / 64; modes x y z xy yz zx xyz = 1..7, components x y z):
//   g1x = A b1x + B (b2y + b3z)   and cyclic      -> ab = A - B, b = B (trace form)
//   g1y = g2x = C (b1y + b2x)     and cyclic      -> c
//   g4x = D b4x + F b5z, g5z = F b4x + D b5z, ... -> d, f
//   g4z = G b4z + H (b5x + b6y)   and cyclic      -> gh = G - H, h = H
//   g7c = J b7c                                   -> j
template <class T>
struct KeModal {
    T ab, b, c, d, f, gh, h, j;
};

// Host: the modal constants of ke (unit E); returns the largest deviation between ke and
// the matrix that modal_element applies, relative to max |ke| (a full 24 x 24 check).
double ke_modal(const double* ke, KeModal<double>* out);

// A nodal 3-vector: x and y as a pair, z alone. In FP32 the pair is a float2 driven by the
// packed f32x2 instructions of sm_100+ (one instruction for both lanes), which takes a third
// of the instructions out of the element transforms; in FP64 it is two doubles.
struct dpair {
    double x, y;
};
template <class T>
struct PairOf;
template <>
struct PairOf<float> {
    using type = float2;
};
template <>
struct PairOf<double> {
    using type = dpair;
};
template <class T>
struct V3 {
    typename PairOf<T>::type xy;
    T z;
};

__host__ __device__ __forceinline__ dpair padd(dpair a, dpair b) { return {a.x + b.x, a.y + b.y}; }
__host__ __device__ __forceinline__ dpair psub(dpair a, dpair b) { return {a.x - b.x, a.y - b.y}; }
__host__ __device__ __forceinline__ dpair pscale(double s, dpair a) { return {s * a.x, s * a.y}; }
#ifdef __CUDACC__
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) {  // a - b, one rounding
    return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
__device__ __forceinline__ float2 pscale(float s, float2 a) { return __fmul2_rn(make_float2(s, s), a); }
__device__ __forceinline__ float2 ptwice_plus(float2 a, float2 b) { return __ffma2_rn(a, make_float2(2.f, 2.f), b); }
#endif
__host__ __device__ __forceinline__ dpair ptwice_plus(dpair a, dpair b) { return {2.0 * a.x + b.x, 2.0 * a.y + b.y}; }

#pragma nv_exec_check_disable
template <class T>
__host__ __device__ __forceinline__ V3<T> operator+(const V3<T>& a, const V3<T>& b) {
    return V3<T>{padd(a.xy, b.xy), a.z + b.z};
}
#pragma nv_exec_check_disable
template <class T>
__host__ __device__ __forceinline__ V3<T> operator-(const V3<T>& a, const V3<T>& b) {
    return V3<T>{psub(a.xy, b.xy), a.z - b.z};
}
#pragma nv_exec_check_disable
template <class T>
__host__ __device__ __forceinline__ V3<T> operator*(T s, const V3<T>& a) {
    return V3<T>{pscale(s, a.xy), s * a.z};
}
__host__ __device__ __forceinline__ float twice_plus(float a, float b) { return 2.f * a + b; }
__host__ __device__ __forceinline__ double twice_plus(double a, double b) { return 2.0 * a + b; }
// 2 a + b
#pragma nv_exec_check_disable
template <class T>
__host__ __device__ __forceinline__ V3<T> twice_plus(const V3<T>& a, const V3<T>& b) {
    return V3<T>{ptwice_plus(a.xy, b.xy), twice_plus(a.z, b.z)};
}
template <class T>
__host__ __device__ __forceinline__ V3<T> v3zero() {
    V3<T> v;
    v.xy.x = T(0);
    v.xy.y = T(0);
    v.z = T(0);
    return v;
}

// E Ke u_e of one brick from its edge differences (p = corner in {0,1}^3):
//   dxb[py] = u(1,py,0) - u(0,py,0),  dxt[py] = u(1,py,1) - u(0,py,1)
//   dyb[px] = u(px,1,0) - u(px,0,0),  dyt[px] = u(px,1,1) - u(px,0,1)
//   dz[px][py] = u(px,py,1) - u(px,py,0)
// and writes the corner forces f[px][py][pz].
// Mode amplitudes b1..b7 (x y z xy yz zx xyz) of a brick from its edge differences: the
// Walsh-Hadamard transform of the corner values, taken through the edges.
#pragma nv_exec_check_disable
template <class T>
__host__ __device__ __forceinline__ void modal_amplitudes(const V3<T> (&dxb)[2], const V3<T> (&dxt)[2],
                                                          const V3<T> (&dyb)[2], const V3<T> (&dyt)[2],
                                                          const V3<T> (&dz)[2][2], V3<T> (&b)[8]) {
    const V3<T> s0 = dxb[0] + dxb[1], s1 = dxt[0] + dxt[1];
    b[1] = s0 + s1;
    b[6] = s1 - s0;
    const V3<T> p0 = dxb[1] - dxb[0], p1 = dxt[1] - dxt[0];
    b[4] = p0 + p1;
    b[7] = p1 - p0;
    const V3<T> t0 = dyb[0] + dyb[1], t1 = dyt[0] + dyt[1];
    b[2] = t0 + t1;
    b[5] = t1 - t0;
    b[3] = (dz[0][0] + dz[1][0]) + (dz[0][1] + dz[1][1]);
}

// u_e^T Ke u_e (unit E) from the mode amplitudes: beta^T (KA / 64) beta written as sums of
// squares in which every rigid rotation cancels inside a square (b1y + b2x for a rotation
// about z, ...), so FP32 keeps the energy of an element that turns a lot but strains little.
#pragma nv_exec_check_disable
template <class T>
__host__ __device__ __forceinline__ T modal_energy(const KeModal<T>& k, const V3<T> (&b)[8]) {
    const T b1x = b[1].xy.x, b1y = b[1].xy.y, b1z = b[1].z, b2x = b[2].xy.x, b2y = b[2].xy.y, b2z = b[2].z;
    const T b3x = b[3].xy.x, b3y = b[3].xy.y, b3z = b[3].z, b4x = b[4].xy.x, b4y = b[4].xy.y, b4z = b[4].z;
    const T b5x = b[5].xy.x, b5y = b[5].xy.y, b5z = b[5].z, b6x = b[6].xy.x, b6y = b[6].xy.y, b6z = b[6].z;
    const T tr = b1x + b2y + b3z, s3 = b4z + b5x + b6y;
    const T q1 = b1y + b2x, q2 = b1z + b3x, q3 = b2z + b3y;
    T e = k.ab * (b1x * b1x + b2y * b2y + b3z * b3z) + k.b * tr * tr + k.c * (q1 * q1 + q2 * q2 + q3 * q3);
    e += k.d * (b4x * b4x + b5z * b5z + b4y * b4y + b6z * b6z + b5y * b5y + b6x * b6x);
    e += T(2) * k.f * (b4x * b5z + b4y * b6z + b5y * b6x);
    e += k.gh * (b4z * b4z + b5x * b5x + b6y * b6y) + k.h * s3 * s3;
    e += k.j * (b[7].xy.x * b[7].xy.x + b[7].xy.y * b[7].xy.y + b[7].z * b[7].z);
    return e;
}

// The modal forces g1..g7 of the amplitudes b1..b7: the sparse modal stiffness, scaled by E (g0 is
// zero: the rigid translations carry no force).
#pragma nv_exec_check_disable
template <class T>
__host__ __device__ __forceinline__ void modal_forces(const KeModal<T>& k, T E, const V3<T> (&b)[8], V3<T> (&g)[8]) {
    const T ab = E * k.ab, bb = E * k.b, cc = E * k.c, dd = E * k.d, ff = E * k.f, gh = E * k.gh, hh = E * k.h,
            jj = E * k.j;
    const T tr = bb * (b[1].xy.x + b[2].xy.y + b[3].z);
    g[1].xy.x = ab * b[1].xy.x + tr;
    g[2].xy.y = ab * b[2].xy.y + tr;
    g[3].z = ab * b[3].z + tr;
    g[1].xy.y = g[2].xy.x = cc * (b[1].xy.y + b[2].xy.x);
    g[1].z = g[3].xy.x = cc * (b[1].z + b[3].xy.x);
    g[2].z = g[3].xy.y = cc * (b[2].z + b[3].xy.y);
    g[4].xy.x = dd * b[4].xy.x + ff * b[5].z;
    g[5].z = ff * b[4].xy.x + dd * b[5].z;
    g[4].xy.y = dd * b[4].xy.y + ff * b[6].z;
    g[6].z = ff * b[4].xy.y + dd * b[6].z;
    g[5].xy.y = dd * b[5].xy.y + ff * b[6].xy.x;
    g[6].xy.x = ff * b[5].xy.y + dd * b[6].xy.x;
    const T s3 = hh * (b[4].z + b[5].xy.x + b[6].xy.y);
    g[4].z = gh * b[4].z + s3;
    g[5].xy.x = gh * b[5].xy.x + s3;
    g[6].xy.y = gh * b[6].xy.y + s3;
    g[7] = jj * b[7];
}

#pragma nv_exec_check_disable
template <class T>
__host__ __device__ __forceinline__ void modal_element(const KeModal<T>& k, T E, const V3<T> (&dxb)[2],
                                                       const V3<T> (&dxt)[2], const V3<T> (&dyb)[2],
                                                       const V3<T> (&dyt)[2], const V3<T> (&dz)[2][2],
                                                       V3<T> (&f)[2][2][2]) {
    // as modal_amplitudes with the y and z edges of the side px = 0 alone: the edges of the other
    // side differ from them by differences of x edges, dy(1) - dy(0) = dx(py = 1) - dx(py = 0)
    V3<T> b[8], g[8];
    const V3<T> s0 = dxb[0] + dxb[1], s1 = dxt[0] + dxt[1];
    b[1] = s0 + s1;
    b[6] = s1 - s0;
    const V3<T> p0 = dxb[1] - dxb[0], p1 = dxt[1] - dxt[0];
    b[4] = p0 + p1;
    b[7] = p1 - p0;
    b[2] = twice_plus(dyb[0] + dyt[0], b[4]);
    b[5] = twice_plus(dyt[0] - dyb[0], b[7]);
    b[3] = twice_plus(dz[0][0] + dz[0][1], b[6]);
    modal_forces<T>(k, E, b, g);
    // back to the corners: f(p) = sum_m s_m(p) g_m = A(py,pz) + sx B(py,pz)
    const V3<T> am = g[2] - g[5], ap = g[2] + g[5];
    const V3<T> n00 = am + g[3], a10 = am - g[3], a01 = g[3] - ap, a11 = ap + g[3];  // A(0,0) = -n00
    const V3<T> cm = g[1] - g[6], cp = g[1] + g[6], dm = g[4] - g[7], dp = g[4] + g[7];
    const V3<T> q00 = cm - dm, q10 = cm + dm, q01 = cp - dp, q11 = cp + dp;
    f[0][0][0] = v3zero<T>() - (n00 + q00);
    f[1][0][0] = q00 - n00;
    f[0][1][0] = a10 - q10;
    f[1][1][0] = a10 + q10;
    f[0][0][1] = a01 - q01;
    f[1][0][1] = a01 + q01;
    f[0][1][1] = a11 - q11;
    f[1][1][1] = a11 + q11;
}

// ------------------------------------------------------------------ reductions

// Deterministic two-stage reductions: every block writes its partial sums to a scratch
// array; the last block to finish (ticket counter) adds the partials in block order and
// writes the result. Nothing depends on atomic ordering, so reruns are bit-identical.
struct RedScratch {
    double* partials;    // capacity_blocks * max_vals
    unsigned* counter;   // one ticket counter per concurrent reduction slot
    int capacity_blocks;
    int max_vals;
};

constexpr int kMaxRedVals = 16;
constexpr int kRedBlocks = 1216;  // 152 SMs x 8: grid of the grid-stride vector kernels

// Sum of `val` over the block, for NV values; result valid in the thread with flat index 0.
// `tid` is the flat thread index (threadIdx.x for 1D blocks).
template <int NV, int NT>
__device__ __forceinline__ void block_sum(double (&val)[NV], double* smem /* NV*NT/32 */, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        double s = val[v];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) smem[v * (NT / 32) + warp] = s;
    }
    __syncthreads();
    if (tid == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            double s = 0;
            for (int w = 0; w < NT / 32; ++w) s += smem[v * (NT / 32) + w];
            val[v] = s;
        }
    }
}

// s + e = a + b exactly (TwoSum)
__device__ __forceinline__ void two_sum_f(float a, float b, float& s, float& e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}
// Block sum of NV float pairs (hi + lo per thread), entirely on the FP32 pipes: the warp tree
// adds pairs with TwoSum, then thread 0 adds the warps' pairs in order. FP64 arithmetic on this
// part runs at a small fraction of the FP32 rate: even a few FP64 instructions per warp, in every
// block of a 1,216-block reduction, cost several microseconds. About 48 significant bits; deterministic.
// Result in thread 0 (in place).
template <int NV, int NT>
__device__ __forceinline__ void block_pair_sum(float (&hi)[NV], float (&lo)[NV], float2* smem /* NV*NT/32 */,
                                               int tid) {
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        float h = hi[v], l = lo[v];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float h2 = __shfl_down_sync(0xffffffffu, h, o), l2 = __shfl_down_sync(0xffffffffu, l, o);
            float t, e;
            two_sum_f(h, h2, t, e);
            h = t;
            l += l2 + e;
        }
        if (lane == 0) smem[v * (NT / 32) + warp] = make_float2(h, l);
    }
    __syncthreads();
    if (tid == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            float2 a = smem[v * (NT / 32)];
            for (int w = 1; w < NT / 32; ++w) {
                const float2 b = smem[v * (NT / 32) + w];
                float t, e;
                two_sum_f(a.x, b.x, t, e);
                a = make_float2(t, a.y + b.y + e);
            }
            hi[v] = a.x;
            lo[v] = a.y;
        }
    }
}

// finish_reduction for float pairs (after block_pair_sum, the pairs valid in thread 0): each
// block stores its pairs in the 8-byte partial slots, the last block adds them in the fixed
// order of finish_reduction with TwoSum and block_pair_sum, and thread 0 writes
// out[v] = hi + lo as a double. Returns true in the block that wrote the result.
template <int NV, int NT>
__device__ __forceinline__ bool finish_pair_reduction(const float (&hi)[NV], const float (&lo)[NV], int bid,
                                                      int nblocks, double* partials, unsigned* counter, double* out,
                                                      int tid, float2* smem /* NV*NT/32 */) {
    __shared__ bool last;
    float2* p = reinterpret_cast<float2*>(partials);
    __syncthreads();  // smem of block_pair_sum is reused below
    if (tid == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) p[(int64_t)bid * NV + v] = make_float2(hi[v], lo[v]);
        __threadfence();
        const unsigned t = atomicAdd(counter, 1u);
        last = (t == (unsigned)nblocks - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    float h[NV], l[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        h[v] = 0.f;
        l[v] = 0.f;
        for (int b = tid; b < nblocks; b += NT) {
            const float2 q = __ldcg(p + (int64_t)b * NV + v);
            float t, e;
            two_sum_f(h[v], q.x, t, e);
            h[v] = t;
            l[v] += q.y + e;
        }
    }
    block_pair_sum<NV, NT>(h, l, smem, tid);
    if (tid == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) out[v] = (double)h[v] + (double)l[v];
        *counter = 0u;
    }
    return true;
}

// block_pair_sum and finish_pair_reduction for many values (NV at most the block's warps): one warp
// per value adds the warps' pairs, and in the last block the blocks' pairs, where the versions above
// add them value by value in one thread (15 values of 512 threads and 152 blocks: 12 us of a pass).
// smem: NV*NT/32 pairs of shared memory. True in the block that wrote the result.
__device__ __forceinline__ float2 warp_pair_sum(float2 a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float h2 = __shfl_down_sync(0xffffffffu, a.x, o), l2 = __shfl_down_sync(0xffffffffu, a.y, o);
        float t, e;
        two_sum_f(a.x, h2, t, e);
        a = make_float2(t, a.y + (l2 + e));
    }
    return a;
}
template <int NV, int NT>
__device__ __forceinline__ bool reduce_pairs_wide(const float (&hi)[NV], const float (&lo)[NV], int bid, int nblocks,
                                                  double* partials, unsigned* counter, double* out, int tid,
                                                  float2* smem) {
    static_assert(NV <= NT / 32 && NT <= 1024, "a warp per value");
    __shared__ bool last;
    const int lane = tid & 31, warp = tid >> 5;
    float2* p = reinterpret_cast<float2*>(partials);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const float2 a = warp_pair_sum(make_float2(hi[v], lo[v]));
        if (lane == 0) smem[v * (NT / 32) + warp] = a;
    }
    __syncthreads();
    if (warp < NV) {
        const float2 a = warp_pair_sum(lane < NT / 32 ? smem[warp * (NT / 32) + lane] : make_float2(0.f, 0.f));
        if (lane == 0) {
            p[(int64_t)bid * NV + warp] = a;
            __threadfence();
        }
    }
    __syncthreads();
    if (tid == 0) last = atomicAdd(counter, 1u) == (unsigned)nblocks - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    if (warp < NV) {
        float2 a = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int b = lane; b < nblocks; b += 32) {
            const float2 q = __ldcg(p + (int64_t)b * NV + warp);
            float t, e;
            two_sum_f(a.x, q.x, t, e);
            a = make_float2(t, a.y + (q.y + e));
        }
        a = warp_pair_sum(a);
        if (lane == 0) out[warp] = (double)a.x + (double)a.y;
    }
    __syncthreads();
    if (tid == 0) *counter = 0u;
    return true;
}

// The same for FP64 values: the threads' values meet in shared memory, where a warp per value adds them
// (39 FP64 instructions for 3 values of 256 threads, 120 by a tree in every warp), in trees: with serial
// chains an OC update at 160x80x80, 7 passes of 500 blocks, takes 474 us instead of 469.
// smem: NV*NT doubles, which the block may have used until here.
__device__ __forceinline__ double warp_sum(double a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    return a;
}
template <int NV, int NT>
__device__ __forceinline__ bool reduce_doubles_wide(const double (&val)[NV], int bid, int nblocks, double* partials,
                                                    unsigned* counter, double* out, int tid, double* smem) {
    static_assert(NV <= NT / 32, "a warp per value");
    __shared__ bool last;
    const int lane = tid & 31, warp = tid >> 5;
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; ++v) smem[v * NT + tid] = val[v];
    __syncthreads();
    if (warp < NV) {
        double t[NT / 32];
#pragma unroll
        for (int q = 0; q < NT / 32; ++q) t[q] = smem[warp * NT + 32 * q + lane];
#pragma unroll
        for (int w = NT / 64; w > 0; w >>= 1)
#pragma unroll
            for (int q = 0; q < w; ++q) t[q] += t[q + w];
        const double a = warp_sum(t[0]);
        if (lane == 0) {
            partials[(int64_t)bid * NV + warp] = a;
            __threadfence();
        }
    }
    __syncthreads();
    if (tid == 0) last = atomicAdd(counter, 1u) == (unsigned)nblocks - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    if (warp < NV) {
        double t[4] = {0.0, 0.0, 0.0, 0.0};
        for (int b = lane; b < nblocks; b += 128)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (b + 32 * q < nblocks) t[q] += __ldcg(partials + (int64_t)(b + 32 * q) * NV + warp);
        const double a = warp_sum((t[0] + t[1]) + (t[2] + t[3]));
        if (lane == 0) out[warp] = a;
    }
    __syncthreads();
    if (tid == 0) *counter = 0u;
    return true;
}

// Finishes a reduction: block `bid` of `nblocks` stores its NV partials; the last block to
// arrive adds them and writes out[0..NV) (from thread 0). The last block sums in parallel:
// thread t adds partials t, t+NT, t+2NT, ... in order, then a fixed tree combines the
// threads, so the result depends only on the partials, never on which block came last.
// Call with every thread of the block after block_sum (val valid in thread 0); `smem` holds
// NV*NT/32 doubles. Returns true in the block that wrote the result.
template <int NV, int NT>
__device__ __forceinline__ bool finish_reduction(const double (&val)[NV], int bid, int nblocks, double* partials,
                                                 unsigned* counter, double* out, int tid, double* smem) {
    __shared__ bool last;
    __syncthreads();  // smem of block_sum is reused below
    if (tid == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) partials[(int64_t)bid * NV + v] = val[v];
        __threadfence();
        unsigned t = atomicAdd(counter, 1u);
        last = (t == (unsigned)nblocks - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        double s = 0.0;
        for (int b = tid; b < nblocks; b += NT) s += __ldcg(partials + (int64_t)b * NV + v);
        acc[v] = s;
    }
    block_sum<NV, NT>(acc, smem, tid);
    if (tid == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) out[v] = acc[v];
        *counter = 0u;
    }
    return true;
}

// Error-free product and sum (Dekker/Knuth): exact s + e == a*b, a+b in FP32. Used for
// dot products whose per-thread partials must carry ~FP48 accuracy before they are
// promoted to FP64 (FP64 arithmetic on this part runs at a small fraction of FP32).
__device__ __forceinline__ void two_prod(float a, float b, float& p, float& e) {
    p = a * b;
    e = fmaf(a, b, -p);
}
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// A double-float: the unevaluated sum hi + lo of two floats, about 48 significant bits.
// Sums and products cost a few FP32 instructions (TwoSum, FMA-based TwoProd), far less than
// FP64 arithmetic on this part. Used for the accurate residual of the FP64 operator.
struct alignas(8) DF {
    float hi, lo;
    DF() = default;
    __host__ __device__ constexpr DF(float h, float l) : hi(h), lo(l) {}
    __host__ __device__ constexpr DF(float v) : hi(v), lo(0.f) {}
    __host__ __device__ explicit constexpr DF(int v) : hi((float)v), lo(0.f) {}
    __host__ __device__ explicit DF(double v) : hi((float)v), lo((float)(v - (double)(float)v)) {}
    __host__ __device__ explicit operator float() const { return hi + lo; }
    __host__ __device__ double value() const { return (double)hi + (double)lo; }
};
#ifdef __CUDACC__
__device__ __forceinline__ DF df_norm(float s, float e) {  // |s| >= |e|
    const float h = s + e;
    return DF(h, e - (h - s));
}
__device__ __forceinline__ DF operator+(DF a, DF b) {
    float s, e;
    two_sum(a.hi, b.hi, s, e);
    e += a.lo + b.lo;
    return df_norm(s, e);
}
__device__ __forceinline__ DF operator-(DF a, DF b) { return a + DF(-b.hi, -b.lo); }
__device__ __forceinline__ DF operator*(DF a, DF b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, e);
    e = fmaf(a.lo, b.hi, e);
    return df_norm(p, e);
}
__device__ __forceinline__ DF operator/(DF a, DF b) { return DF(a.value() / b.value()); }  // not on a hot path
// 1 / a to about 48 bits: the FP32 reciprocal refined by one Newton step in pair arithmetic
// (r + r (1 - a r) doubles the number of correct bits)
__device__ __forceinline__ DF df_recip(DF a) {
    const float r0 = 1.f / a.hi;
    const DF e = DF(1.f) - a * DF(r0);
    return DF(r0) + DF(r0) * e;
}
__device__ __forceinline__ DF& operator+=(DF& a, DF b) { return a = a + b; }
__device__ __forceinline__ bool operator>(DF a, DF b) { return a.value() > b.value(); }
#endif
#ifdef __CUDACC__
// A double as an unevaluated float pair hi + lo, by integer and FP32 operations only (FP64
// arithmetic on this part runs at a small fraction of the FP32 rate, and a conversion per
// value is FP64 work): hi keeps the leading 24 significant bits (truncated), lo the next 29
// rounded to 24, so hi + lo is within 2^-48 of d. |d| below 2^-120 becomes (signed) zero and
// |d| beyond the float range takes the FP64 path; neither occurs in the fields split here.
__device__ __forceinline__ void split_double(double d, float& hi, float& lo) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
    const int e = (int)((b >> 52) & 0x7FF);
    if (e < 1023 - 120) {
        hi = __uint_as_float(sign);
        lo = 0.f;
        return;
    }
    if (e > 1023 + 127) {
        hi = (float)d;
        lo = 0.f;
        return;
    }
    const unsigned long long m = b & 0xFFFFFFFFFFFFFull;
    hi = __uint_as_float(sign | ((unsigned)(e - 896) << 23) | (unsigned)(m >> 29));
    const unsigned r = (unsigned)(m & 0x1FFFFFFFull);  // the 29 bits below hi, weight 2^(e - 1075)
    const float scale = e > 948 ? __uint_as_float((unsigned)(e - 948) << 23) : 0.f;
    const float l = __uint2float_rn(r) * scale;
    lo = sign ? -l : l;
}
// (a_hi + a_lo) - (b_hi + b_lo) rounded to FP32
__device__ __forceinline__ float df_diff(float ah, float al, float bh, float bl) {
    float s, e;
    two_sum(ah, -bh, s, e);
    return s + (e + (al - bl));
}
#endif
struct dfpair {
    DF x, y;
};
template <>
struct PairOf<DF> {
    using type = dfpair;
};
#ifdef __CUDACC__
__device__ __forceinline__ dfpair padd(dfpair a, dfpair b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ dfpair psub(dfpair a, dfpair b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ dfpair pscale(DF s, dfpair a) { return {s * a.x, s * a.y}; }
__device__ __forceinline__ DF twice_plus(DF a, DF b) { return DF(2.f * a.hi, 2.f * a.lo) + b; }
__device__ __forceinline__ dfpair ptwice_plus(dfpair a, dfpair b) { return {twice_plus(a.x, b.x), twice_plus(a.y, b.y)}; }
#endif

// Compensated accumulator: adds a*b exactly up to FP32 rounding of the error terms.
struct Acc2 {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add_prod(float a, float b) {
        float p, e, t, f;
        two_prod(a, b, p, e);
        two_sum(s, p, t, f);
        s = t;
        c += f + e;
    }
    __device__ __forceinline__ void add_prod(double a, double b) {  // FP64 inputs
        add_d(a * b);
    }
    __device__ __forceinline__ void add_d(double v) {
        float hi = (float)v;
        float lo = (float)(v - (double)hi);
        float t, f;
        two_sum(s, hi, t, f);
        s = t;
        c += f + lo;
    }
    __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

// ------------------------------------------------------------------ PCG device scalars

struct PcgScalars {
    double rz[2];   // r.z of the current / next iteration (ping-pong on iteration parity)
    double pq;      // p.K p
    double zq;      // z_new.q (flexible beta)
    double rr;      // ||r||^2
    double bb;      // ||b||^2
    double alpha;
    // the next step's alpha and beta in both precisions, formed by the reductions' last thread (a
    // division in every thread of a full grid is 6 us of FP64 on this part)
    double step, beta;
    float step_f, beta_f;
    int step_bad;   // p.K p is not positive, or alpha no number
    double tol2;    // (rtol ||b||)^2
    double rr_true; // ||b - K x||^2 from the last residual replacement
    int done;       // 0 running, 1 converged, 2 maxiter, 3 non-finite, 4 breakdown; every
                    // kernel of the CG loop returns early while it is non-zero
    int iters;      // iterations performed
    int nonfinite;  // a non-finite scalar was seen
    int maxiter;
};

#ifdef __CUDACC__
// after pq: alpha = r.z / p.K p (one thread)
__device__ __forceinline__ void pcg_set_step(PcgScalars* sc) {
    const double pq = sc->pq, v = sc->rz[sc->iters & 1] / pq;
    sc->step = v;
    sc->step_f = (float)v;
    sc->step_bad = !(pq > 0.0) || !isfinite(v);
}
__device__ __forceinline__ float pcg_step(const PcgScalars* sc, float) { return sc->step_f; }
__device__ __forceinline__ double pcg_step(const PcgScalars* sc, double) { return sc->step; }
__device__ __forceinline__ float pcg_beta(const PcgScalars* sc, float) { return sc->beta_f; }
__device__ __forceinline__ double pcg_beta(const PcgScalars* sc, double) { return sc->beta; }
#endif

inline int ceil_div(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

}  // namespace anl
