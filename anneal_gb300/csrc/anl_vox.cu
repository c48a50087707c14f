// anl_vox.cu -- the voxeliser: the fill fraction of every grid element inside a closed
// triangle mesh.
//
// Replaces geometry.voxel_fill (geometry.py:89-149). The method is the reference's: s x s x s
// sample points per element, a ray along +z through every (x, y) sample column, a sample is
// inside when an odd number of the column's triangle crossings lie below it, and the fill
// fraction is the inside share of the element's samples. The reference gathers every
// crossing as a key (column index + normalised height), sorts all keys and counts the keys
// below each sample by binary search. Here nothing is sorted:
//  1. k_vox_zrange: the lowest and highest vertex z (they normalise the crossing heights);
//  2. k_vox_axes: the sample coordinates along x and y and the normalised sample heights;
//  3. k_vox_count: per triangle, the sample columns inside its xy bounding box (binary
//     search on the sample axes) and the triangle's part of the test; an exclusive scan gives
//     every (triangle, column) pair a slot;
//  4. k_vox_hits: the barycentric test of every pair. A crossing flips the bit of the lowest
//     sample above it in the column's bit row (atomicXor), so that
//  5. k_vox_parity: a prefix XOR along each column turns the flips into inside bits, and
//  6. k_vox_fill: the popcount of an element's s^3 sample bits, divided by s^3.
// Every number that decides a crossing or a comparison is the reference's FP64 expression,
// evaluated one rounded operation at a time (__dmul_rn, __dadd_rn, __dsub_rn: nothing is
// contracted into an FMA; every quotient is the correctly rounded one). A crossing is counted below
// a sample exactly when the reference's sorted search counts it, so the inside bits and the
// fill fractions are the reference's, bit for bit.
#include <new>

#include "anl_common.cuh"
#include "anl_scan.cuh"

namespace anl {

constexpr int VOX_T = 256;
constexpr int VOX_MAX_S = 16;
constexpr int VOX_HT = 128;              // k_vox_hits: threads of a block, and blocks
constexpr int VOX_HIT_BLOCKS = 152 * 6;

struct VoxGrid {
    int nx, ny, nz, s;
    int nxs, nys, nzs;  // sample counts per axis (n * s)
    int64_t ncol;       // nxs * nys
    int W;              // 32-bit words per column bit row
    double h, ox, oy, oz;
    double up;          // samples per unit of height
};

// doubles ordered as unsigned integers (atomicMin/atomicMax on finite values)
__device__ __forceinline__ unsigned long long dkey(double d) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double dunkey(unsigned long long k) {
    const unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)b);
}

// Correctly rounded a / b from r = 1 / b (correctly rounded): Markstein's correction (IBM J. Res.
// Dev. 34, 1990). a r is within two ulps of the quotient; the first step brings it within one, and
// from there the second gives the rounded quotient, as the remainder a - q b of a q that close is
// exact. That needs every step far from overflow and underflow: other operands are divided. Five
// operations on the FP64 pipe, which takes one warp instruction in 19 cycles per SM.
__device__ __forceinline__ bool div_safe(double v) {  // 2^-400 <= |v| < 2^401
    return ((((unsigned)__double2hiint(v) >> 20) & 0x7ffu) - 623u) <= 800u;
}
__device__ __forceinline__ double div_by(double a, double b, double r) {
    if (!(div_safe(a) && div_safe(b))) return a / b;
    double q = __dmul_rn(a, r);
    q = __fma_rn(__fma_rn(-q, b, a), r, q);
    return __fma_rn(__fma_rn(-q, b, a), r, q);
}
// False only if the rounded a / b is negative or no number, from the signs and exponents alone (no
// FP64 instruction); b's high word, kVoxNone where no quotient by b is a number or b is zero. Signs
// that differ give a negative quotient unless it underflows to -0 (which counts as inside): the
// exponents rule that out.
constexpr int kVoxNone = 0x7fffffff;
__device__ __forceinline__ bool may_be_inside(double a, int bhi) {
    const int ahi = __double2hiint(a);
    const int ea = (ahi >> 20) & 0x7ff, eb = (bhi >> 20) & 0x7ff;
    const bool zero = ((ahi & 0x7fffffff) | __double2loint(a)) == 0;
    return !((ahi ^ bhi) < 0 && !zero && eb < 0x7ff && ea - eb > -1000);
}

// True only if the sum of two numerators of the determinant's sign is more than 1 + 2^-21 times the
// determinant, or no number (high words that differ by more than one unit of 2^-20): 1 - l0 - l1 is
// negative then, whatever the roundings.
__device__ __forceinline__ bool past(double sum, int bhi) {
    return (__double2hiint(sum) & 0x7fffffff) - (bhi & 0x7fffffff) > 1;
}

// zmm[0] = key of min z, zmm[1] = key of max z (initialised to ~0 and 0)
__global__ void __launch_bounds__(VOX_T) k_vox_zrange(const double* __restrict__ tri, int64_t ntri,
                                                      unsigned long long* zmm) {
    unsigned long long lo = ~0ull, hi = 0ull;
    for (int64_t v = blockIdx.x * (int64_t)VOX_T + threadIdx.x; v < 3 * ntri; v += (int64_t)gridDim.x * VOX_T) {
        const unsigned long long k = dkey(tri[3 * v + 2]);
        lo = min(lo, k);
        hi = max(hi, k);
    }
    __shared__ unsigned long long sm[2][VOX_T / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        sm[0][threadIdx.x >> 5] = lo;
        sm[1][threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // one atomic pair per block: they queue at one address
        for (int w = 1; w < VOX_T / 32; ++w) {
            lo = min(lo, sm[0][w]);
            hi = max(hi, sm[1][w]);
        }
        atomicMin(zmm, lo);
        atomicMax(zmm + 1, hi);
    }
}

// xs, ys: sample coordinates (geometry.py:91-94); zq: normalised, clipped sample heights
// (geometry.py:144); zs_out[0..2] = zlo, zr, 1 / zr
__global__ void __launch_bounds__(VOX_T) k_vox_axes(VoxGrid G, const unsigned long long* zmm, double* xs,
                                                    double* ys, double* zq, double* frac, double* zs_out) {
    const double zlo = dunkey(zmm[0]), zhi = dunkey(zmm[1]);
    const double zr = __dadd_rn(__dmul_rn(__dsub_rn(zhi, zlo), 1.001), 1e-9);
    const int n = G.nxs + G.nys + G.nzs;
    for (int t = blockIdx.x * VOX_T + threadIdx.x; t < n; t += gridDim.x * VOX_T) {
        int axis, m = t;
        if (m < G.nxs) {
            axis = 0;
        } else if ((m -= G.nxs) < G.nys) {
            axis = 1;
        } else {
            m -= G.nys;
            axis = 2;
        }
        const int i = m / G.s, a = m - i * G.s;
        const double sub = ((double)a + 0.5) / (double)G.s;
        const double o = axis == 0 ? G.ox : axis == 1 ? G.oy : G.oz;
        const double c = __dadd_rn(o, __dmul_rn(G.h, __dadd_rn((double)i, sub)));
        if (axis == 0) {
            xs[m] = __dadd_rn(c, __dmul_rn(G.h, 6.18e-6));
        } else if (axis == 1) {
            ys[m] = __dadd_rn(c, __dmul_rn(G.h, 4.14e-6));
        } else {
            const double q = __dsub_rn(c, zlo) / zr;
            zq[m] = fmin(fmax(q, 0.0), 0.999999);
        }
    }
    // the fill fractions of 0..s^3 samples: k_vox_fill's divisions, once
    const int n3 = G.s * G.s * G.s;
    for (int c = blockIdx.x * VOX_T + threadIdx.x; c <= n3; c += gridDim.x * VOX_T) frac[c] = (double)c / (double)n3;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        zs_out[0] = zlo;
        zs_out[1] = zr;
        zs_out[2] = 1.0 / zr;
    }
}

// first index with a[i] >= v (right = false) or a[i] > v (right = true): numpy searchsorted
__device__ __forceinline__ int vox_search(const double* __restrict__ a, int n, double v, bool right) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const double x = a[mid];
        if (right ? (x <= v) : (x < v))
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// the same, first trying the place where even spacing from a[0] puts v: two comparisons instead of a
// chain of nine dependent loads and FP64 comparisons on an axis of 384
__device__ __forceinline__ int vox_locate(const double* __restrict__ a, int n, double v, bool right, double o, double up) {
    const int at = min(max((int)ceil((v - o) * up), 0), n);
    auto before = [&](int i) { return right ? (a[i] <= v) : (a[i] < v); };
    if ((at == 0 || before(at - 1)) && (at == n || !before(at))) return at;
    return vox_search(a, n, v, right);
}

// What the barycentric test takes from the triangle alone: vertex 2, the edges and the determinant
struct alignas(16) VoxTri {
    double x2, y2, y12, x21, y20, x02, d, r;  // r = 1 / d
};

// per triangle: the first sample column along x and y inside its bounding box, the box width and the
// determinant's high word; cnt = the number of columns in the box (geometry.py:99-105)
__global__ void __launch_bounds__(VOX_T) k_vox_count(const double* __restrict__ tri, int64_t ntri, VoxGrid G,
                                                     const double* __restrict__ xs, const double* __restrict__ ys,
                                                     int4* __restrict__ box, long long* __restrict__ cnt,
                                                     VoxTri* __restrict__ rec) {
    const double x0 = xs[0], y0 = ys[0];
    for (int64_t t = blockIdx.x * (int64_t)VOX_T + threadIdx.x; t < ntri; t += (int64_t)gridDim.x * VOX_T) {
        const double* v = tri + 9 * t;
        const double xmin = fmin(fmin(v[0], v[3]), v[6]), xmax = fmax(fmax(v[0], v[3]), v[6]);
        const double ymin = fmin(fmin(v[1], v[4]), v[7]), ymax = fmax(fmax(v[1], v[4]), v[7]);
        const int ix0 = vox_locate(xs, G.nxs, xmin, false, x0, G.up), ix1 = vox_locate(xs, G.nxs, xmax, true, x0, G.up);
        const int iy0 = vox_locate(ys, G.nys, ymin, false, y0, G.up), iy1 = vox_locate(ys, G.nys, ymax, true, y0, G.up);
        const int nxr = max(ix1 - ix0, 0), nyr = max(iy1 - iy0, 0);
        VoxTri q;
        q.x2 = v[6], q.y2 = v[7];
        q.y12 = __dsub_rn(v[4], q.y2), q.x21 = __dsub_rn(q.x2, v[3]);
        q.y20 = __dsub_rn(q.y2, v[1]), q.x02 = __dsub_rn(v[0], q.x2);
        q.d = __dadd_rn(__dmul_rn(q.y12, q.x02), __dmul_rn(q.x21, __dsub_rn(v[1], q.y2)));
        q.r = 1.0 / q.d;
        rec[t] = q;
        const bool none = q.d == 0.0 || q.d != q.d;
        box[t] = make_int4(ix0, iy0, nxr, none ? kVoxNone : __double2hiint(q.d));
        cnt[t] = (long long)nxr * nyr;
    }
}

// A pair whose barycentric numerators have the determinant's sign
struct alignas(16) VoxPair {
    double n0, n1;
    long long t, c;  // triangle, column
};
constexpr int VOX_PAIRS = 2 * VOX_HT;      // pairs a block takes at a time
constexpr int VOX_CAP = 2 * VOX_PAIRS;    // of its list
constexpr int VOX_RANGE = 2 * VOX_PAIRS;  // of its triangles' staged offsets

// The triangle of pair p: the last t with off[t] <= p (triangles without columns have no slot). A warp
// probes 32 places at a time.
__device__ __forceinline__ int64_t vox_find_warp(const long long* __restrict__ off, int64_t ntri, long long p, int lane) {
    int64_t lo = 0, hi = ntri;
    while (lo < hi) {
        const int64_t step = (hi - lo + 31) / 32, at = lo + lane * step + step - 1;
        const int below = __popc(__ballot_sync(0xffffffffu, at < hi && off[at] <= p));
        lo += below * step;
        hi = min(hi, lo + step - 1);
    }
    return lo - 1;
}

// The barycentric test of geometry.py:124-131 and the flip of the lowest sample the crossing lies
// below (geometry.py:139-146), bound by the FP64 pipe (one warp instruction in 19 cycles per SM).
// More than half of the pairs of a bounding box miss the triangle, and a warp that tests 32 of them
// pays for the divisions and the heights if one hits. So a block first takes the numerators and their
// signs of its pairs (9 FP64 instructions each), lists those that can hit in shared memory, and runs
// the rest on full warps of them, with the quotients from reciprocals (div_by) and the sample from the
// height instead of a search over the samples. The 0.2 million pairs of 20,480 triangles over 384x192
// columns: 19 us from cold caches (10 of them FP64 issue, the rest the chain of loads to a block's
// triangles), 40 us with the whole test and both searches in one thread per pair.
__global__ void __launch_bounds__(VOX_HT) k_vox_hits(const double* __restrict__ tri, int64_t ntri, VoxGrid G,
                                                    const double* __restrict__ xs, const double* __restrict__ ys,
                                                    const double* __restrict__ zq, const double* __restrict__ zs,
                                                    const int4* __restrict__ box, const VoxTri* __restrict__ rec,
                                                    const long long* __restrict__ off,
                                                    const long long* __restrict__ total, unsigned* __restrict__ bits,
                                                    unsigned long long* __restrict__ nhits) {
    __shared__ VoxPair list[VOX_CAP];
    __shared__ int first[VOX_RANGE];
    __shared__ int64_t ends[2];
    __shared__ int listed;
    __shared__ unsigned long long hits;
    const long long np = *total;
    const double zlo = zs[0], zr = zs[1], rzr = zs[2];
    const int lane = threadIdx.x & 31;
    unsigned mine = 0;
    int n = 0;  // pairs in the list
    if (threadIdx.x == 0) {
        listed = 0;
        hits = 0;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    const long long stride = (long long)gridDim.x * VOX_PAIRS;
    for (long long p0 = blockIdx.x * (long long)VOX_PAIRS; p0 < np; p0 += stride) {
        // the pairs' triangles t0..t1 and their offsets in shared memory: a search of all offsets by
        // every thread is 15 dependent loads
        const int here = (int)min((long long)VOX_PAIRS, np - p0);
        if (warp < 2) {
            const int64_t t = vox_find_warp(off, ntri, warp == 0 ? p0 : p0 + here - 1, lane);
            if (lane == 0) ends[warp] = t;
        }
        __syncthreads();
        const int64_t t0 = ends[0], t1 = ends[1];
        const bool staged = t1 - t0 < VOX_RANGE;
        if (staged) {
            for (int k = threadIdx.x; k <= (int)(t1 - t0); k += VOX_HT) first[k] = (int)max(off[t0 + k] - p0, -1ll);
            __syncthreads();
        }
        int found = 0;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int k = half * VOX_HT + threadIdx.x;
            bool in = false;
            VoxPair e;
            if (k < here) {
                if (staged) {
                    int lo = 1, hi = (int)(t1 - t0) + 1;  // the first triangle starts at or before k
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (first[mid] <= k)
                            lo = mid + 1;
                        else
                            hi = mid;
                    }
                    e.t = t0 + lo - 1;
                } else {
                    int64_t lo = t0 + 1, hi = t1 + 1;
                    while (lo < hi) {
                        const int64_t mid = (lo + hi) >> 1;
                        if (off[mid] <= p0 + k)
                            lo = mid + 1;
                        else
                            hi = mid;
                    }
                    e.t = lo - 1;
                }
                const int4 b = box[e.t];
                const long long local = p0 + k - off[e.t];
                int lx, ly;
                if (local <= 0x7fffffff) {
                    ly = (int)((unsigned)local / (unsigned)b.z);
                    lx = (int)local - ly * b.z;
                } else {
                    lx = (int)(local % b.z);
                    ly = (int)(local / b.z);
                }
                const int cx = b.x + lx, cy = b.y + ly;
                e.c = cx + (long long)G.nxs * cy;
                if (b.w != kVoxNone) {
                    const VoxTri& q = rec[e.t];
                    const double pxd = __dsub_rn(xs[cx], q.x2), pyd = __dsub_rn(ys[cy], q.y2);
                    e.n0 = __dadd_rn(__dmul_rn(q.y12, pxd), __dmul_rn(q.x21, pyd));
                    e.n1 = __dadd_rn(__dmul_rn(q.y20, pxd), __dmul_rn(q.x02, pyd));
                    in = may_be_inside(e.n0, b.w) && may_be_inside(e.n1, b.w) &&
                         !past(__dadd_rn(e.n0, e.n1), b.w);
                }
            }
            found += in;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (m) {
                int at = 0;
                if (lane == 0) at = atomicAdd(&listed, __popc(m));
                at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
                if (in) list[at] = e;
            }
        }
        // (a sum over the block: `listed` already counts the next round in a faster warp)
        n += __syncthreads_count(found > 0) + __syncthreads_count(found > 1);
        if (n > VOX_CAP - VOX_PAIRS || p0 + stride >= np) {  // no room for another round, or the last one
            for (int k = threadIdx.x; k < n; k += VOX_HT) {
                const VoxPair& w = list[k];
                const VoxTri& q = rec[w.t];
                const double l0 = div_by(w.n0, q.d, q.r), l1 = div_by(w.n1, q.d, q.r);
                const double l2 = __dsub_rn(__dsub_rn(1.0, l0), l1);
                if (!(l0 >= 0.0 && l1 >= 0.0 && l2 >= 0.0)) continue;
                const double* v = tri + 9 * w.t;
                const double z = __dadd_rn(__dadd_rn(__dmul_rn(l0, v[2]), __dmul_rn(l1, v[5])), __dmul_rn(l2, v[8]));
                const double zn = div_by(__dsub_rn(z, zlo), zr, rzr);
                // The reference sorts keys col + zn and counts, for sample m of column c, the keys in
                // [c, c + zq[m]) (both ends rounded to FP64 like the keys). A key that rounds below its
                // own column is therefore counted nowhere, and one that reaches the next column's
                // range belongs to that column.
                long long c = w.c;
                double cd = G.ncol <= 0x7fffffff ? (double)(int)c : (double)c;
                const double key = __dadd_rn(cd, zn);
                if (key < cd) continue;
                const double next = __dadd_rn(cd, 1.0);  // exact: columns are below 2^40
                if (key >= next) {
                    if (++c >= G.ncol) continue;
                    cd = next;
                }
                ++mine;
                // the lowest sample with c + zq[sample] > key: the one above the height, if the two
                // comparisons that make it the lowest agree
                auto above = [&](int i) { return __dadd_rn(cd, zq[i]) > key; };
                int at = min(max((int)ceil((z - G.oz) * G.up - 0.5), 0), G.nzs);
                if (!((at == G.nzs || above(at)) && (at == 0 || !above(at - 1)))) {
                    int lo = 0, hi = G.nzs;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (above(mid))
                            hi = mid;
                        else
                            lo = mid + 1;
                    }
                    at = lo;
                }
                if (at < G.nzs) atomicXor(bits + (int64_t)(at >> 5) * G.ncol + c, 1u << (at & 31));
            }
            __syncthreads();
            if (threadIdx.x == 0) listed = 0;
            n = 0;
            __syncthreads();
        }
    }
    // one atomic per block: they queue at one address
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0 && mine) atomicAdd(&hits, (unsigned long long)mine);
    __syncthreads();
    if (threadIdx.x == 0 && hits) atomicAdd(nhits, hits);
}

// bit rows of flips -> inside bits (prefix XOR along z); rows are word-major: bits[w*ncol + c]. A
// column's words are loaded eight at a time before the first is stored (3.8 us for 384x192 columns of
// six words, 5.8 one after the other).
__global__ void __launch_bounds__(VOX_T) k_vox_parity(VoxGrid G, unsigned* __restrict__ bits) {
    for (int64_t c = blockIdx.x * (int64_t)VOX_T + threadIdx.x; c < G.ncol; c += (int64_t)gridDim.x * VOX_T) {
        unsigned carry = 0;
        for (int w0 = 0; w0 < G.W; w0 += 8) {
            unsigned q[8];
#pragma unroll
            for (int w = 0; w < 8; ++w) q[w] = w0 + w < G.W ? bits[(int64_t)(w0 + w) * G.ncol + c] : 0u;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                unsigned x = q[w];
                x ^= x << 1;
                x ^= x << 2;
                x ^= x << 4;
                x ^= x << 8;
                x ^= x << 16;
                x ^= carry;
                carry = (x >> 31) ? ~0u : 0u;
                if (w0 + w < G.W) bits[(int64_t)(w0 + w) * G.ncol + c] = x;
            }
        }
    }
}

// fill fraction per element (x fastest): inside samples / s^3 (geometry.py:147-149), the quotient
// from a table: an FP64 division per element took 18 of 26 us at 128x64x64. A thread takes up to
// four elements of a column whose samples one 32-bit window holds (one or two words per sample
// column for the four of them), I: unsigned where the threads fit 32 bits (a 64-bit division by a
// variable is a hundred instructions): 5.9 us at 128x64x64, 10.6 with a thread per element.
constexpr int VOX_STACK = 4;
__host__ __device__ constexpr int vox_stack(int s) { return 32 / s < VOX_STACK ? 32 / s : VOX_STACK; }
template <class I>
__global__ void __launch_bounds__(VOX_T) k_vox_fill(VoxGrid G, const unsigned* __restrict__ bits,
                                                    const double* __restrict__ frac, double* __restrict__ fill) {
    const int stack = vox_stack(G.s);
    const int64_t plane = (int64_t)G.nx * G.ny;
    const int64_t n = plane * ((G.nz + stack - 1) / stack);
    const unsigned mask = (1u << G.s) - 1u;
    for (int64_t e = blockIdx.x * (int64_t)VOX_T + threadIdx.x; e < n; e += (int64_t)gridDim.x * VOX_T) {
        const I r = (I)e / (I)G.nx;
        const int i = (int)((I)e - r * (I)G.nx);
        const int j = (int)(r % (I)G.ny), k = (int)(r / (I)G.ny) * stack;
        const int m = k * G.s, w = m >> 5, sh = m & 31;
        const bool two = sh + stack * G.s > 32 && w + 1 < G.W;
        int count[VOX_STACK] = {};
        const unsigned* p = bits + (int64_t)w * G.ncol + (int64_t)i * G.s + (int64_t)G.nxs * ((int64_t)j * G.s);
        for (int b = 0; b < G.s; ++b, p += G.nxs)
            for (int a = 0; a < G.s; ++a) {
                const unsigned x = __funnelshift_r(p[a], two ? p[G.ncol + a] : 0u, sh);
#pragma unroll
                for (int q = 0; q < VOX_STACK; ++q)
                    if (q < stack) count[q] += __popc((x >> (q * G.s)) & mask);
            }
        double* out = fill + (int64_t)k * plane + (int64_t)j * G.nx + i;
#pragma unroll
        for (int q = 0; q < VOX_STACK; ++q)
            if (q < stack && k + q < G.nz) out[q * plane] = frac[count[q]];
    }
}

inline int vox_blocks(int64_t n) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + VOX_T - 1) / VOX_T, 152 * 16));
}

}  // namespace anl

using namespace anl;

struct anl_vox {
    int4* box = nullptr;
    size_t box_cap = 0;
    long long* cnt = nullptr;
    size_t cnt_cap = 0;
    long long* off = nullptr;
    size_t off_cap = 0;
    VoxTri* rec = nullptr;
    size_t rec_cap = 0;
    double* axes = nullptr;  // xs | ys | zq | fill fractions
    size_t axes_cap = 0;
    unsigned* bits = nullptr;
    size_t bits_cap = 0;
    long long* part = nullptr;  // SCAN_BLOCKS
    // scalars: [0..1] z range keys, [2] pair total, [3] hits, then zlo, zr, 1 / zr as doubles
    unsigned long long* sc = nullptr;
    unsigned long long* host = nullptr;
};

namespace {

void vox_free(anl_vox* v) {
    std::lock_guard<std::recursive_mutex> lock(device_sync_mutex());
    cudaFree(v->box);
    cudaFree(v->cnt);
    cudaFree(v->off);
    cudaFree(v->rec);
    cudaFree(v->axes);
    cudaFree(v->bits);
    cudaFree(v->part);
    cudaFree(v->sc);
    if (v->host) cudaFreeHost(v->host);
    delete v;
}

}  // namespace

extern "C" {

int anl_vox_create(anl_vox** out) {
    if (!out) {
        set_error("anl_vox_create: null argument");
        return ANL_ERR_BADARG;
    }
    *out = nullptr;
    anl_vox* v = new (std::nothrow) anl_vox();
    if (!v) return ANL_ERR_NOMEM;
    std::lock_guard<std::recursive_mutex> lock(device_sync_mutex());
    if (cudaMalloc((void**)&v->part, SCAN_BLOCKS * sizeof(long long)) != cudaSuccess ||
        cudaMalloc((void**)&v->sc, 8 * sizeof(unsigned long long)) != cudaSuccess ||
        cudaMallocHost((void**)&v->host, 8 * sizeof(unsigned long long)) != cudaSuccess) {
        cudaGetLastError();
        set_error("anl_vox_create: allocation failed");
        vox_free(v);
        return ANL_ERR_NOMEM;
    }
    *out = v;
    return ANL_OK;
}

void anl_vox_destroy(anl_vox* v) {
    if (v) vox_free(v);
}

int anl_voxel_fill(anl_vox* v, const double* tri, int64_t ntri, int nx, int ny, int nz, double h,
                   const double* origin_h, int s, double* fill, int64_t* stats_h, anl_stream_t stream) {
    if (!v || !tri || !origin_h || !fill || ntri < 1 || nx < 1 || ny < 1 || nz < 1 || s < 1 || s > VOX_MAX_S ||
        !(h > 0) || !std::isfinite(h)) {
        set_error("anl_voxel_fill: bad argument%s", ntri < 1 ? " (the mesh has no triangles)" : "");
        return ANL_ERR_BADARG;
    }
    const int64_t nxs = (int64_t)nx * s, nys = (int64_t)ny * s, nzs = (int64_t)nz * s;
    if (nxs > (1 << 28) || nys > (1 << 28) || nzs > (1 << 28) || nxs * nys > ((int64_t)1 << 40) ||
        ntri > ((int64_t)1 << 40)) {
        set_error("anl_voxel_fill: grid or mesh too large");
        return ANL_ERR_BADARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    VoxGrid G;
    G.nx = nx, G.ny = ny, G.nz = nz, G.s = s;
    G.nxs = (int)nxs, G.nys = (int)nys, G.nzs = (int)nzs;
    G.ncol = nxs * nys;
    G.W = (int)((nzs + 31) / 32);
    G.up = s / h;
    G.h = h, G.ox = origin_h[0], G.oy = origin_h[1], G.oz = origin_h[2];
    const size_t nbits = (size_t)G.W * (size_t)G.ncol;
    ANL_TRY(grow(v->box, v->box_cap, (size_t)ntri, sizeof(int4)));
    ANL_TRY(grow(v->cnt, v->cnt_cap, (size_t)ntri, sizeof(long long)));
    ANL_TRY(grow(v->off, v->off_cap, (size_t)ntri, sizeof(long long)));
    ANL_TRY(grow(v->rec, v->rec_cap, (size_t)ntri, sizeof(VoxTri)));
    ANL_TRY(grow(v->axes, v->axes_cap, (size_t)(nxs + nys + nzs + s * s * s + 1), sizeof(double)));
    ANL_TRY(grow(v->bits, v->bits_cap, nbits, sizeof(unsigned)));
    double* xs = v->axes;
    double* ys = xs + nxs;
    double* zq = ys + nys;
    double* frac = zq + nzs;
    double* zs = (double*)(v->sc + 4);
    ANL_CUDA(cudaMemsetAsync(v->sc, 0xff, sizeof(unsigned long long), st));
    ANL_CUDA(cudaMemsetAsync(v->sc + 1, 0, 3 * sizeof(unsigned long long), st));
    ANL_CUDA(cudaMemsetAsync(v->bits, 0, nbits * sizeof(unsigned), st));
    k_vox_zrange<<<vox_blocks(3 * ntri), VOX_T, 0, st>>>(tri, ntri, v->sc);
    ANL_LAUNCH_CHECK();
    k_vox_axes<<<vox_blocks(nxs + nys + nzs), VOX_T, 0, st>>>(G, v->sc, xs, ys, zq, frac, zs);
    ANL_LAUNCH_CHECK();
    k_vox_count<<<vox_blocks(ntri), VOX_T, 0, st>>>(tri, ntri, G, xs, ys, v->box, v->cnt, v->rec);
    ANL_LAUNCH_CHECK();
    ANL_TRY(scan_exclusive<long long>(v->cnt, ntri, v->off, v->part, (long long*)(v->sc + 2), st));
    k_vox_hits<<<VOX_HIT_BLOCKS, VOX_HT, 0, st>>>(tri, ntri, G, xs, ys, zq, zs, v->box, v->rec, v->off,
                                                 (const long long*)(v->sc + 2), v->bits, v->sc + 3);
    ANL_LAUNCH_CHECK();
    k_vox_parity<<<vox_blocks(G.ncol), VOX_T, 0, st>>>(G, v->bits);
    ANL_LAUNCH_CHECK();
    const int64_t stacks = (int64_t)nx * ny * ((nz + vox_stack(s) - 1) / vox_stack(s));
    if (stacks <= 0xffffffffll) k_vox_fill<unsigned><<<vox_blocks(stacks), VOX_T, 0, st>>>(G, v->bits, frac, fill);
    else k_vox_fill<int64_t><<<vox_blocks(stacks), VOX_T, 0, st>>>(G, v->bits, frac, fill);
    ANL_LAUNCH_CHECK();
    if (stats_h) {
        ANL_CUDA(cudaMemcpyAsync(v->host, v->sc + 2, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
        ANL_CUDA(cudaStreamSynchronize(st));
        stats_h[0] = (int64_t)v->host[0];
        stats_h[1] = (int64_t)v->host[1];
    }
    return ANL_OK;
}

}  // extern "C"
