// anl_design.cu -- design-variable kernels of one SIMP iteration: density filter,
// projection, stiffness scale, sensitivity, OC bisection and the history statistics.
//
// Element fields are FP32 on the full grid (x fastest, zero on inactive elements). Sums are float
// pairs (about 48 bits) across threads, where k_oc_vol_bank adds a thread's own share in FP32; the OC
// update's projected volumes are FP64 sums.
#include <algorithm>
#include <climits>
#include <cstddef>
#include <cmath>
#include <cstring>

#include "anl_ctx.cuh"

namespace anl {

constexpr int DT = 256;
static inline int dgrid(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>(kRedBlocks, (n + DT - 1) / DT)); }

// ------------------------------------------------------------------ density filter

// Filter (optimize.py:24-47). One CTA of 32x8 threads owns a 32x8 column of elements and marches
// up z, one staged plane (with an R-element halo in x and y) per layer, double-buffered with one
// barrier. The cone's weight depends on (|dx|, |dy|, |dz|) alone and not on the order of |dx| and
// |dy|, so a thread sums its plane's (2R+1)^2 values once by class (|dx|, |dy|), weighs the class
// sums for each |dz| and adds these R + 1 partial results to the 2R + 1 output layers they belong
// to, kept in registers. Against a ring of 2R + 2 planes re-read for every layer this takes a
// (2R+1)-th of the shared-memory loads and, at R = 2, 42 instead of 125 multiply-adds: the kernel
// was bound by them at R >= 2 and by its latency chain at R = 1. Forward with projection and
// backward at 128x64x64, r = 2.6: 166 -> 23 us together (memory floor 2 us).
enum { F_HS = 0, F_FWD = 1, F_BWD = 2, F_PHYS = 3 };

constexpr int FT_X = 32, FT_Y = 8, FT_ZC = 16, FT_N = FT_X * FT_Y;
// Layers per CTA. A chunk stages 2R layers more than it writes, and a layer is a chain of memory
// latencies, so a grid of few columns is cut into shorter chunks until it has about three CTAs
// per SM (4 layers at least; with 16 at 128x64x64 a third of the SMs had one CTA and the others
// none).
static inline int filter_chunk(const Dims& d) {
    const int columns = ceil_div(d.nx, FT_X) * ceil_div(d.ny, FT_Y);
    return std::max(4, std::min(FT_ZC, ceil_div(d.nz, ceil_div(3 * 152, columns))));
}
static inline dim3 filter_grid(const Dims& d) {
    return dim3(ceil_div(d.nx, FT_X), ceil_div(d.ny, FT_Y), ceil_div(d.nz, filter_chunk(d)));
}
int filter_blocks(const Dims& d) {
    const dim3 g = filter_grid(d);
    return (int)(g.x * g.y * g.z);
}

struct FilterArgs {
    Dims d;
    int zc;                // layers per CTA
    float wc[kMaxFilterR + 1][kFilterClasses];  // cone weights by |dz| and class (|dx|, |dy|)
    const uint8_t* active;
    const float* Hs;
    const float* in;       // FWD/BWD/PHYS input field
    float* out;
    // PHYS
    const uint8_t* frozen;
    float* dxp;
    float beta, eta, t0, t1;
};

// optimize.py:150-152: ratio = sqrt(max(-dcx,0) / max(dvx*lam, 1e-300)),
// xn = clip(x*ratio, max(0, x-mv), min(1, x+mv)). Split into the part of an element that does
// not depend on lambda (x sqrt(max(-dcx,0)/dvx)) and one multiply by 1/sqrt(lambda), so a bank
// of lambdas costs a multiply and a clamp each.
struct OcElem {
    float s;       // x sqrt(max(-dcx, 0) / dvx)
    float dvx;
    float lo, hi;  // the move limits
    bool grows;    // max(-dcx, 0) > 0 and x > 0: the ratio is huge where dvx lambda underflows
};
__device__ __forceinline__ OcElem oc_elem(float x, float dcx, float dvx, float move) {
    OcElem o;
    const float num = fmaxf(-dcx, 0.f);
    o.s = dvx > 0.f ? x * sqrtf(num / dvx) : 0.f;
    o.dvx = dvx;
    o.lo = fmaxf(0.f, x - move);
    o.hi = fminf(1.f, x + move);
    o.grows = num > 0.f && x > 0.f;
    return o;
}
__device__ __forceinline__ float oc_rl(float lam) { return 1.f / sqrtf(lam); }
__device__ __forceinline__ float oc_xn(const OcElem& o, float lam, float rl) {
    const float v = o.dvx * lam > 1e-30f ? o.s * rl : (o.grows ? INFINITY : 0.f);
    return fminf(fmaxf(v, o.lo), o.hi);
}
__device__ __forceinline__ float oc_xn(float x, float dcx, float dvx, float lam, float move) {
    return oc_xn(oc_elem(x, dcx, dvx, move), lam, oc_rl(lam));
}

// the filter's input value of element e (zero on inactive elements): the active flag and the
// field are loaded independently of each other
template <int MODE>
__device__ __forceinline__ float filter_input(const FilterArgs& a, int64_t e) {
    if (!ANL_IN_RANGE(e, a.d.ne())) return 0.f;
    const bool act = a.active[e] != 0;
    float v = 1.f;
    if (MODE == F_FWD || MODE == F_PHYS) v = a.in[e];
    else if (MODE == F_BWD) v = a.in[e] / a.Hs[e];
    return act ? v : 0.f;
}

// The staged plane of a halo-R tile: which elements this thread stages.
template <int R>
struct FilterTile {
    static constexpr int TX = FT_X + 2 * R, PL = TX * (FT_Y + 2 * R), PF = (PL + FT_N - 1) / FT_N;
    int64_t exy[PF];  // index within an element plane, -1 outside the grid or the tile
    __device__ FilterTile(const Dims& d, int i0, int j0, int tid) {
#pragma unroll
        for (int q = 0; q < PF; ++q) {
            const int t = tid + q * FT_N, y = t / TX, x = t - y * TX, gi = i0 - R + x, gj = j0 - R + y;
            exy[q] = t < PL && gi >= 0 && gj >= 0 && gi < d.nx && gj < d.ny ? gi + (int64_t)d.nx * gj : -1;
        }
    }
};

// Adds the plane's contribution around (tx, ty) to the 2R + 1 layers of acc: acc[R] is the
// plane's own layer.
template <int R>
__device__ __forceinline__ void filter_plane(const float (&wc)[kMaxFilterR + 1][kFilterClasses], const float* pl,
                                             int tx, int ty, float (&acc)[2 * R + 1]) {
    constexpr int NC = (R + 1) * (R + 2) / 2;
    float cs[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) cs[c] = 0.f;
#pragma unroll
    for (int dy = -R; dy <= R; ++dy)
#pragma unroll
        for (int dx = -R; dx <= R; ++dx) {
            const int ax = dx < 0 ? -dx : dx, ay = dy < 0 ? -dy : dy;
            cs[filter_class(ax, ay)] += pl[(ty + R + dy) * FilterTile<R>::TX + tx + R + dx];
        }
#pragma unroll
    for (int q = 0; q <= R; ++q) {
        float s = wc[q][0] * cs[0];
#pragma unroll
        for (int c = 1; c < NC; ++c) s = fmaf(wc[q][c], cs[c], s);
        acc[R - q] += s;
        if (q > 0) acc[R + q] += s;
    }
}

template <int MODE, int R>
__global__ void __launch_bounds__(FT_N) k_filter(FilterArgs a) {
    using Tile = FilterTile<R>;
    __shared__ float pl[2][Tile::PL];
    const Dims d = a.d;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + FT_X * ty;
    const int i0 = blockIdx.x * FT_X, j0 = blockIdx.y * FT_Y, kb = blockIdx.z * a.zc;
    const int kend = min(kb + a.zc, d.nz);
    const int64_t eplane = (int64_t)d.nx * d.ny;
    const Tile tile(d, i0, j0, tid);
    float pf[Tile::PF];  // the next plane's values of this thread, loaded a layer ahead
    auto prefetch = [&](int gk) {
#pragma unroll
        for (int q = 0; q < Tile::PF; ++q)
            pf[q] = tile.exy[q] >= 0 && gk >= 0 && gk < d.nz ? filter_input<MODE>(a, tile.exy[q] + gk * eplane) : 0.f;
    };
    prefetch(kb - R);
    const int i = i0 + tx, j = j0 + ty;
    const bool in_xy = i < d.nx && j < d.ny;
    float acc[2 * R + 1];
#pragma unroll
    for (int q = 0; q < 2 * R + 1; ++q) acc[q] = 0.f;
    for (int gk = kb - R; gk < kend + R; ++gk) {
        float* buf = pl[gk & 1];
#pragma unroll
        for (int q = 0; q < Tile::PF; ++q)
            if (tid + q * FT_N < Tile::PL) buf[tid + q * FT_N] = pf[q];
        if (gk + 1 < kend + R) prefetch(gk + 1);
        // the epilogue inputs of the layer that this plane completes
        const int k = gk - R;
        const int64_t e = in_xy && k >= kb ? d.elem(i, j, k) : 0;
        const bool in_e = in_xy && k >= kb && ANL_IN_RANGE(e, d.ne());
        bool act = false, fzn = false;
        float hs = 1.f;
        if (in_e) {
            act = a.active[e] != 0;
            if (MODE == F_FWD || MODE == F_PHYS) hs = a.Hs[e];
            if (MODE == F_PHYS) fzn = a.frozen[e] != 0;
        }
        __syncthreads();
        filter_plane<R>(a.wc, buf, tx, ty, acc);
        const float s = acc[0];
#pragma unroll
        for (int q = 0; q < 2 * R; ++q) acc[q] = acc[q + 1];
        acc[2 * R] = 0.f;
        if (in_e) {
            if (MODE == F_HS) {
                a.out[e] = s == 0.f ? 1.f : s;
            } else if (MODE == F_FWD) {
                a.out[e] = act ? s / hs : 0.f;
            } else if (MODE == F_BWD) {
                a.out[e] = act ? s : 0.f;
            } else {
                // physical(): projection (optimize.py:81-87), frozen -> 1 (optimize.py:92)
                float xp = act ? s / hs : 0.f, g = 1.f;
                if (a.beta > 0.f) {
                    const float th = tanhf(a.beta * (xp - a.eta));
                    xp = (a.t0 + th) / (a.t0 + a.t1);
                    g = a.beta * (1.f - th * th) / (a.t0 + a.t1);
                }
                a.out[e] = act ? (fzn ? 1.f : xp) : 0.f;
                if (a.dxp) a.dxp[e] = act ? g : 0.f;
            }
        }
    }
}

static FilterArgs filter_args(const anl_ctx* c) {
    FilterArgs a{};
    a.d = c->d;
    a.active = c->active;
    a.Hs = c->filt.Hs;
    std::memcpy(a.wc, c->filt.wc, sizeof(a.wc));
    a.zc = filter_chunk(a.d);
    return a;
}

template <int MODE>
static int launch_filter(anl_ctx* c, const FilterArgs& a, cudaStream_t s) {
    const dim3 grid = filter_grid(a.d), block(FT_X, FT_Y);
    switch (c->filt.R) {
        case 1: k_filter<MODE, 1><<<grid, block, 0, s>>>(a); break;
        case 2: k_filter<MODE, 2><<<grid, block, 0, s>>>(a); break;
        case 3: k_filter<MODE, 3><<<grid, block, 0, s>>>(a); break;
        case 4: k_filter<MODE, 4><<<grid, block, 0, s>>>(a); break;
        default: k_filter<MODE, 5><<<grid, block, 0, s>>>(a); break;
    }
    ANL_LAUNCH_CHECK();
    return ANL_OK;
}

int filter_init(anl_ctx* c, double r, cudaStream_t s) {
    int R = (int)std::ceil(r) - 1;
    if (R < 1) R = 1;
    if (R > kMaxFilterR || !(r > 0)) {
        set_error("filter radius %.3f voxels needs a %d-element halo; at most %d is supported", r, R, kMaxFilterR);
        return ANL_ERR_BADARG;
    }
    for (int q = 0; q <= kMaxFilterR; ++q)
        for (int ax = 0; ax <= kMaxFilterR; ++ax)
            for (int ay = 0; ay <= ax; ++ay) {
                const double v = r - std::sqrt((double)(ax * ax + ay * ay + q * q));
                c->filt.wc[q][filter_class(ax, ay)] = v > 0 ? (float)v : 0.f;
            }
    c->filt.R = R;
    c->filt.r = r;
    FilterArgs a = filter_args(c);
    a.out = c->filt.Hs;
    ANL_TRY(launch_filter<F_HS>(c, a, s));
    ANL_CUDA(cudaStreamSynchronize(s));  // Hs is read by calls on any stream from here on
    c->filt.ready = true;
    return ANL_OK;
}

int filter_apply(anl_ctx* c, bool forward, const float* in, float* out, cudaStream_t s) {
    FilterArgs a = filter_args(c);
    a.in = in;
    a.out = out;
    return forward ? launch_filter<F_FWD>(c, a, s) : launch_filter<F_BWD>(c, a, s);
}

int physical(anl_ctx* c, const float* x, const uint8_t* frozen, double beta, double eta, float* xphys, float* dxp,
             cudaStream_t s) {
    FilterArgs a = filter_args(c);
    a.in = x;
    a.out = xphys;
    a.frozen = frozen;
    a.dxp = dxp;
    a.beta = (float)beta;
    a.eta = (float)eta;
    if (beta > 0) {
        a.t0 = (float)std::tanh(beta * eta);
        a.t1 = (float)std::tanh(beta * (1 - eta));
    }
    return launch_filter<F_PHYS>(c, a, s);
}

// ------------------------------------------------------------------ stiffness scale

__global__ void k_escale(int64_t ne, const uint8_t* active, const float* xphys, const float* phi, float E0, float emin,
                         float p, float* escale) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
        float v = 0.f;
        if (active[e]) {
            const float xp = xphys[e];
            const float xpp = p == 1.f ? xp : (p == 3.f ? xp * xp * xp : powf(xp, p));
            v = E0 * phi[e] * (emin + xpp * (1.f - emin));
        }
        escale[e] = v;
    }
}

int stiffness_scale(anl_ctx* c, const float* xphys, const float* phi, double E0, double emin, double p, float* escale,
                    cudaStream_t s) {
    const int64_t ne = c->d.ne();
    k_escale<<<dgrid(ne), DT, 0, s>>>(ne, c->active, xphys, phi, (float)E0, (float)emin, (float)p, escale);
    ANL_LAUNCH_CHECK();
    return ANL_OK;
}

// ------------------------------------------------------------------ sensitivity

constexpr int kMaxCases = 16;
struct SensArgs {
    Dims d;
    const uint8_t* active;
    const DF* u;      // nrhs nodal vectors as float pairs (k_split_pairs)
    int nrhs;
    int64_t stride;   // 3 * nn
    float coef[kMaxCases];
    const float* xphys;
    const float* dxp;
    const float* phi;
    float p, emin, E0, h;
    float* out;       // dc (combined, clipped, times dxp) or ce (energy only)
    float* dv;        // phi * dxp (optional)
    int energy_only;
};

// The FP64 displacements as float pairs, once per node (split_double: no FP64 arithmetic);
// the element kernel then reads each corner as one 8-byte pair instead of splitting it again
// for each of its up to 8 elements.
__global__ void k_split_pairs(int64_t n, const double* x, DF* xdf) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float h, l;
        split_double(x[i], h, l);
        xdf[i] = DF(h, l);
    }
}

// u_e^T Ke u_e from the modal energy form (modal_energy): edge differences are formed in
// double-float arithmetic from the FP64 displacements and rounded once to FP32, and rigid
// rotations cancel inside squares, so the result keeps its accuracy relative to the element's
// own strain energy.
__device__ __forceinline__ float element_energy(const KeModal<float>& K, const DF* u, const Dims& d, int i, int j,
                                                int k) {
    const int64_t sx = 1, sy = d.nx + 1, sz = (int64_t)(d.nx + 1) * (d.ny + 1);
    const int64_t n0 = d.node(i, j, k);
    if (!ANL_IN_RANGE(n0, d.nn()) || !ANL_IN_RANGE(n0 + sx + sy + sz, d.nn())) return 0.f;
    float ch[2][2][2][3], cl[2][2][2][3];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int px = q & 1, py = (q >> 1) & 1, pz = (q >> 2) & 1;
        const int64_t n = n0 + px * sx + py * sy + pz * sz;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 t = __ldg(reinterpret_cast<const float2*>(u + 3 * n + c));
            ch[px][py][pz][c] = t.x;
            cl[px][py][pz][c] = t.y;
        }
    }
    auto diff = [&](int ax, int bx, int ay, int by, int az, int bz) {
        V3<float> v;
        v.xy.x = df_diff(ch[ax][ay][az][0], cl[ax][ay][az][0], ch[bx][by][bz][0], cl[bx][by][bz][0]);
        v.xy.y = df_diff(ch[ax][ay][az][1], cl[ax][ay][az][1], ch[bx][by][bz][1], cl[bx][by][bz][1]);
        v.z = df_diff(ch[ax][ay][az][2], cl[ax][ay][az][2], ch[bx][by][bz][2], cl[bx][by][bz][2]);
        return v;
    };
    V3<float> dxb[2], dxt[2], dyb[2], dyt[2], dz[2][2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        dxb[q] = diff(1, 0, q, q, 0, 0);
        dxt[q] = diff(1, 0, q, q, 1, 1);
        dyb[q] = diff(q, q, 1, 0, 0, 0);
        dyt[q] = diff(q, q, 1, 0, 1, 1);
#pragma unroll
        for (int r = 0; r < 2; ++r) dz[q][r] = diff(q, q, r, r, 1, 0);
    }
    V3<float> bm[8];
    modal_amplitudes<float>(dxb, dxt, dyb, dyt, dz, bm);
    return modal_energy<float>(K, bm);
}

__global__ void k_sens(SensArgs a, KeModal<float> K) {
    const Dims d = a.d;
    const int64_t ne = d.ne();
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
        float v = 0.f;
        if (a.active[e]) {
            const int i = (int)(e % d.nx), j = (int)((e / d.nx) % d.ny), k = (int)(e / ((int64_t)d.nx * d.ny));
            if (a.energy_only) {
                v = a.h * element_energy(K, a.u, d, i, j, k);
            } else {
                const float xp = a.xphys[e];
                const float dpow = a.p == 1.f ? 1.f : (a.p == 3.f ? xp * xp : powf(xp, a.p - 1.f));
                const float pre = -a.p * dpow * (1.f - a.emin) * a.E0 * a.phi[e] * a.h;
                float dc = 0.f;
                for (int c = 0; c < a.nrhs; ++c) dc += a.coef[c] * pre * element_energy(K, a.u + c * a.stride, d, i, j, k);
                dc = fminf(dc, 0.f);
                v = a.dxp ? dc * a.dxp[e] : dc;
            }
        }
        a.out[e] = v;
        if (a.dv) a.dv[e] = a.active[e] ? (a.dxp ? a.phi[e] * a.dxp[e] : a.phi[e]) : 0.f;
    }
}

// Element-centre stress (fem.py:244-263): at the centre only the linear modes have slopes,
// du_c/dx_d = b_dc / (4 h) with b_dc = sum of the 4 edge differences of component c along d,
// so the strain is eps = (b1x, b2y, b3z, b2x + b1y, b3y + b2z, b1z + b3x) / (4 h) (Voigt,
// engineering shear) and sigma = E D eps with the isotropic D of unit modulus. FP64.
__global__ void k_stress(Dims d, const uint8_t* active, const double* u, const double* Emat, double Escalar, double h,
                         double lam, double mu, double* sig, double* vm) {
    const int64_t ne = d.ne();
    const int64_t sx = 1, sy = d.nx + 1, sz = (int64_t)(d.nx + 1) * (d.ny + 1);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
        if (!active[e]) {
            if (sig)
                for (int q = 0; q < 6; ++q) sig[6 * e + q] = 0.0;
            if (vm) vm[e] = 0.0;
            continue;
        }
        const int i = (int)(e % d.nx), j = (int)((e / d.nx) % d.ny), k = (int)(e / ((int64_t)d.nx * d.ny));
        const int64_t n0 = d.node(i, j, k);
        double g[3][3] = {};  // g[c][dir]: sum of edge differences of component c along dir
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int a = q & 1, b = q >> 1;
            const int64_t ex = n0 + a * sy + b * sz, ey = n0 + a * sx + b * sz, ez = n0 + a * sx + b * sy;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                g[c][0] += u[3 * (ex + sx) + c] - u[3 * ex + c];
                g[c][1] += u[3 * (ey + sy) + c] - u[3 * ey + c];
                g[c][2] += u[3 * (ez + sz) + c] - u[3 * ez + c];
            }
        }
        const double s = 1.0 / (4.0 * h);
        const double exx = g[0][0] * s, eyy = g[1][1] * s, ezz = g[2][2] * s;
        const double gxy = (g[0][1] + g[1][0]) * s, gyz = (g[1][2] + g[2][1]) * s, gzx = (g[2][0] + g[0][2]) * s;
        const double E = Emat ? Emat[e] : Escalar;
        const double tr = exx + eyy + ezz;
        const double S[6] = {E * (lam * tr + 2 * mu * exx), E * (lam * tr + 2 * mu * eyy), E * (lam * tr + 2 * mu * ezz),
                             E * mu * gxy, E * mu * gyz, E * mu * gzx};
        if (sig)
            for (int q = 0; q < 6; ++q) sig[6 * e + q] = S[q];
        if (vm)
            vm[e] = sqrt(0.5 * ((S[0] - S[1]) * (S[0] - S[1]) + (S[1] - S[2]) * (S[1] - S[2]) + (S[2] - S[0]) * (S[2] - S[0])) +
                         3.0 * (S[3] * S[3] + S[4] * S[4] + S[5] * S[5]));
    }
}

int element_stress(anl_ctx* c, const double* u, const double* Emat, double Escalar, double* sig, double* vm,
                   cudaStream_t s) {
    const double nu = c->nu;
    const double lam = nu / ((1 + nu) * (1 - 2 * nu)), mu = 1.0 / (2 * (1 + nu));
    k_stress<<<dgrid(c->d.ne()), DT, 0, s>>>(c->d, c->active, u, Emat, Escalar, c->h, lam, mu, sig, vm);
    ANL_LAUNCH_CHECK();
    return ANL_OK;
}

int sensitivity(anl_ctx* c, const double* u, int nrhs, const double* coef, const float* xphys, const float* dxp,
                const float* phi, double p, double emin, double E0, float* out, float* dv, bool energy_only,
                cudaStream_t s) {
    if (nrhs < 1 || nrhs > kMaxCases) {
        set_error("sensitivity supports 1..%d load cases, got %d", kMaxCases, nrhs);
        return ANL_ERR_BADARG;
    }
    const int64_t ndof = 3 * c->d.nn();
    ANL_TRY(grow(c->sens_df, c->sens_df_cap, (size_t)nrhs * ndof, sizeof(DF)));
    k_split_pairs<<<dgrid(nrhs * ndof), DT, 0, s>>>(nrhs * ndof, u, c->sens_df);
    ANL_LAUNCH_CHECK();
    SensArgs a{};
    a.d = c->d;
    a.active = c->active;
    a.u = c->sens_df;
    a.nrhs = nrhs;
    a.stride = ndof;
    for (int k = 0; k < nrhs; ++k) a.coef[k] = coef ? (float)coef[k] : 1.f;
    a.xphys = xphys;
    a.dxp = dxp;
    a.phi = phi;
    a.p = (float)p;
    a.emin = (float)emin;
    a.E0 = (float)E0;
    a.h = (float)c->h;
    a.out = out;
    a.dv = energy_only ? nullptr : dv;
    a.energy_only = energy_only ? 1 : 0;
    const int64_t ne = c->d.ne();
    k_sens<<<dgrid(ne), DT, 0, s>>>(a, c->kmf);
    ANL_LAUNCH_CHECK();
    return ANL_OK;
}

// ------------------------------------------------------------------ OC update

// sums over design (active, non-frozen) elements: -dcx, dvx, count
// a float-pair running sum (TwoSum per term): FP32 instructions only
struct PairSum {
    float h = 0.f, l = 0.f;
    __device__ __forceinline__ void add(float x) {
        float t, e;
        two_sum_f(h, x, t, e);
        h = t;
        l += e;
    }
};
template <int NV>
__device__ __forceinline__ bool finish_pair_sums(const PairSum (&v)[NV], double* partials, unsigned* counter,
                                                 double* out, float2* smem) {
    float h[NV], l[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        h[q] = v[q].h;
        l[q] = v[q].l;
    }
    block_pair_sum<NV, DT>(h, l, smem, threadIdx.x);
    return finish_pair_reduction<NV, DT>(h, l, blockIdx.x, gridDim.x, partials, counter, out, threadIdx.x, smem);
}

__global__ void k_oc_scale(int64_t ne, const uint8_t* active, const uint8_t* frozen, const float* dcx, const float* dvx,
                           double* partials, unsigned* counter, double* out) {
    __shared__ float2 sm[3 * DT / 32];
    PairSum v[3];
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x)
        if (active[e] && !frozen[e]) {
            v[0].add(-dcx[e]);
            v[1].add(dvx[e]);
            v[2].add(1.f);
        }
    finish_pair_sums<3>(v, partials, counter, out, sm);
}

// The bisection (optimize.py:147-160) on the device. Its answer is the last midpoint lambda, the
// updates use lambda in FP32, and the volume falls with lambda, so the bisection is decided once
// two neighbouring floats are known with the volume above the target at the lower one and not
// above it at the upper one: its midpoints then fall on either side without another volume.
// Each pass evaluates the volume at a bank of lambdas inside the bracket known so far and its last
// block narrows the bracket and picks the next bank (oc_advance): 4 passes of 15 or 5-7 passes of 3
// lambdas instead of one volume for each of the 36 steps.
//  * No projection: the volume is linear in xn, vol = sum_j wv_j xn_j + sum_frozen phi, with
//    wv = Filter.backward(phi on non-frozen elements): k_oc_vol_bank, a stream over the elements,
//    issue-bound at 15 lambdas (about 8 instructions per lambda and element).
//  * Projection: xn is filtered and projected for each lambda: k_oc_vol_proj, the filter's march
//    with 3 lambdas side by side (their staged planes share the loads; more lambdas cost more
//    than the passes they save).
// The part of each element's update that does not depend on lambda is formed once per OC update
// (k_oc_prep): (s, dvx, lo, hi) and (g, w), with g the value where dvx lambda underflows (hi if
// the element grows, else lo) and w the weight of the volume, frozen elements as lo = hi = 1 and
// inactive ones with w = 0. A lambda then costs a multiply, a compare and a clamp per element.
constexpr int OC_BANK = 15, OC_PROJ = 3;
static_assert(OC_BANK <= kMaxRedVals, "one partial per lambda and block");
static_assert(OC_BANK <= 16, "the bank's volumes fit red_out");
struct OcBank {
    float lam[OC_BANK];
    int n;
};

__global__ void k_oc_prep(int64_t ne, const uint8_t* __restrict__ active, const uint8_t* __restrict__ frozen,
                          const float* __restrict__ x, const float* __restrict__ dcx, const float* __restrict__ dvx,
                          const float* __restrict__ wv, float move, float4* __restrict__ el, float2* __restrict__ gw) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
        if (!active[e]) {
            el[e] = make_float4(0.f, 1.f, 0.f, 0.f);
            gw[e] = make_float2(0.f, 0.f);
        } else if (frozen[e]) {
            el[e] = make_float4(0.f, 1.f, 1.f, 1.f);
            gw[e] = make_float2(1.f, wv[e]);
        } else {
            const OcElem o = oc_elem(x[e], dcx[e], dvx[e], move);
            el[e] = make_float4(o.s, o.dvx, o.lo, o.hi);
            gw[e] = make_float2(o.grows ? o.hi : o.lo, wv[e]);
        }
    }
}

// The search's state in device memory: the passes and the final update run back to back on the
// stream with no host round trip. Positive floats order like their bits, so the bracket is kept
// in bits: an interval of them is a range of lambda on a nearly logarithmic scale.
struct OcState {
    double lo, hi, lam;  // the bisection's first bracket; its last midpoint
    double vfrozen, vtarget;
    int steps, stop;
    int tlo, thi;        // bits of the largest lambda known above the target volume and of the smallest
                         // one not above it; next to the bisection's bracket while not known
    int width;           // the interval before the last pass (0: a side was not known)
    int known;           // bit 0: tlo is such a lambda, bit 1: thi is
    double flo, fhi;     // their volumes
    OcBank bank;         // the lambdas of the next pass
};

// one warp: after a pass, narrow the bracket; then either replay the bisection or choose the next
// bank of at most nmax lambdas
__device__ void oc_advance(OcState* st, const double* vols, int nmax, int lane) {
    int tlo = st->tlo, thi = st->thi;
    const int n = st->bank.n, width = st->width;
    int known = st->known;
    double flo = st->flo, fhi = st->fhi;
    const double target = st->vtarget;
    // a lane per lambda: the largest above the target, then the smallest not above it beyond that
    const int pj = lane < n ? __float_as_int(st->bank.lam[lane]) : -1;
    const double vj = lane < n ? vols[lane] + st->vfrozen : 0.0;
    const bool above = vj > target;
    const int up = __reduce_max_sync(0xffffffffu, lane < n && above ? pj : -1);
    if (up > tlo) {
        tlo = up;
        known |= 1;
        flo = __shfl_sync(0xffffffffu, vj, __ffs(__ballot_sync(0xffffffffu, lane < n && above && pj == up)) - 1);
    }
    const bool low = lane < n && !above && pj > tlo;
    const int dn = __reduce_min_sync(0xffffffffu, low ? pj : INT_MAX);
    if (dn < thi) {
        thi = dn;
        known |= 2;
        fhi = __shfl_sync(0xffffffffu, vj, __ffs(__ballot_sync(0xffffffffu, low && pj == dn)) - 1);
    }
    const int gap = thi - tlo - 1;
    if (gap <= 0) {
        if (lane == 0) {  // the bisection's own steps, each decided by the bracket
            double lo = st->lo, hi = st->hi, lam = st->lam;
            int steps = 0;
            while (steps < 100) {
                lam = sqrt(lo * hi);
                (__float_as_int((float)lam) <= tlo ? lo : hi) = lam;
                ++steps;
                if (hi < lo * (1 + 1e-9)) break;
            }
            st->lam = lam;
            st->steps = steps;
            st->stop = 1;
        }
        return;
    }
    // Next: from a known side towards the other end in octaves 2, 8, 32, ...; every float while they
    // fit the bank; around the zero of the line through the two ends (its error shrinks with the
    // square of the interval) at doubling distances; or, where that did not halve the interval or a
    // volume is not finite, at even distances
    const int m = min(nmax, gap), h = (m - 1) / 2;
    const bool both = known == 3, line = isfinite(flo) && isfinite(fhi);
    int p;
    if (gap <= nmax) {
        p = tlo + 1 + lane;
    } else if (!both) {
        const long long d = 2ll << (23 + 2 * min(lane, 8));
        p = known == 1 ? (int)min(tlo + d, (long long)thi - 1) : (int)max(thi - d, (long long)tlo + 1);
    } else if (!line || (width > 0 && thi - tlo > width / 2)) {
        p = tlo + (int)((int64_t)(thi - tlo) * (lane + 1) / (m + 1));
    } else {
        const double d = thi - tlo;
        const int r = max(tlo + 1, min(thi - 1, tlo + (int)(d * ((flo - target) / (flo - fhi)))));
        const double near = fmax(1.0, fmin(d * d * (1.0 / 8388608.0 / 16.0), d / (double)(1 << h)));
        const int t = lane - h;
        const double off = t == 0 ? 0.0 : near * (double)(1 << (min(abs(t), 16) - 1));
        p = t < 0 ? r - (int)off : r + (int)off;
        p = max(tlo + 1, min(thi - 1, p));
    }
    if (lane < m) st->bank.lam[lane] = __int_as_float(p);
    if (lane == 0) {
        st->bank.n = m;
        st->tlo = tlo;
        st->thi = thi;
        st->known = known;
        st->width = both ? thi - tlo : 0;
        st->flo = flo;
        st->fhi = fhi;
    }
}

// one warp: the bisection's bracket and the first bank, two octaves around the mean ratio
__global__ void k_oc_begin(OcState* st, const double* sums, const double* vfrozen, double vtarget, int n) {
    const int lane = threadIdx.x;
    // optimize.py:145: the bracket from the mean sensitivities of the design elements
    double scale = 1.0;
    const double nd = sums[2];
    if (nd > 0) {
        const double mdc = sums[0] / nd, mdv = sums[1] / nd;
        scale = fmax(mdc / fmax(mdv, 1e-30), 1e-300);
    }
    const double lo = scale * 1e-8, hi = scale * 1e8;
    const int a = __float_as_int((float)lo), b = __float_as_int((float)hi), c = __float_as_int((float)scale);
    if (lane < n) {
        const int h = (n - 1) / 2;
        const long long p = c + (2ll << 23) * (lane - h) / h;
        st->bank.lam[lane] = __int_as_float((int)max((long long)a, min((long long)b, p)));
    }
    if (lane == 0) {
        st->lo = lo;
        st->hi = hi;
        st->lam = sqrt(lo * hi);
        st->vfrozen = vfrozen ? *vfrozen : 0.0;
        st->vtarget = vtarget;
        st->steps = 0;
        st->stop = 0;
        st->tlo = a - 1;
        st->thi = b + 1;
        st->width = 0;
        st->known = 0;
        st->flo = st->fhi = NAN;
        st->bank.n = n;
    }
}

constexpr int OCB_T = 512;  // threads of a bank pass: one CTA per SM, each thread ~54 elements at 12.8M DOF
__global__ void __launch_bounds__(OCB_T, 1) k_oc_vol_bank(int64_t ne, const float4* __restrict__ el,
                                                    const float2* __restrict__ gw, OcState* st,
                                                    double* partials, unsigned* counter, double* out) {
    if (st->stop) return;  // the same for every block
    const OcBank bank = st->bank;
    __shared__ float2 sm[OC_BANK * OCB_T / 32];
    float acc[OC_BANK], rl[OC_BANK];
#pragma unroll
    for (int j = 0; j < OC_BANK; ++j) {
        acc[j] = 0.f;
        rl[j] = oc_rl(bank.lam[j]);
    }
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    constexpr int U = 4;  // elements per trip, their loads issued before any is used
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += U * stride) {
        float4 q[U];
        float2 t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = e + u * stride < ne;
            q[u] = in ? el[e + u * stride] : make_float4(0.f, 1.f, 0.f, 0.f);
            t[u] = in ? gw[e + u * stride] : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < OC_BANK; ++j) {
            if (j < bank.n) {  // oc_xn with the elements' lambda-free parts
                float a = acc[j];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float v = q[u].y * bank.lam[j] > 1e-30f ? fminf(fmaxf(q[u].x * rl[j], q[u].z), q[u].w)
                                                                   : t[u].x;
                    a = fmaf(t[u].y, v, a);
                }
                acc[j] = a;
            }
        }
    }
    float lo[OC_BANK];
#pragma unroll
    for (int j = 0; j < OC_BANK; ++j) lo[j] = 0.f;
    if (reduce_pairs_wide<OC_BANK, OCB_T>(acc, lo, blockIdx.x, gridDim.x, partials, counter, out, threadIdx.x, sm) &&
        threadIdx.x < 32)
        oc_advance(st, out, OC_BANK, threadIdx.x);
}

// The double of a float without the FP64 pipe, which converts a warp in some 19 cycles per SM. In
// k_oc_vol_proj it pays where the filter's registers leave few warps to hide that: an update takes 760
// instead of 805 us at 192x90x90, R = 3, 251 either way at 97x50x41, R = 2, but 479 instead of 472 at
// 160x80x80, R = 1 (before reduce_doubles_wide added in trees).
__device__ __forceinline__ double widen(float v) {
    const unsigned b = __float_as_uint(v), e = (b >> 23) & 0xffu;
    if (e - 1u >= 254u) return (double)v;  // zero, denormal, infinite, no number
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// One pass with projection: the volume sum phi physical(xn(lambda)) of each lambda of the bank,
// xn filtered as in k_filter; phi xp is formed (exactly) and summed in FP64.
struct OcProjArgs {
    FilterArgs f;
    const float4* el;
    const float2* gw;
    OcState* st;
    double* partials;
    unsigned* counter;
    double* out;
};
template <int R>
__global__ void __launch_bounds__(FT_N) k_oc_vol_proj(OcProjArgs a) {
    if (a.st->stop) return;  // the same for every block
    using Tile = FilterTile<R>;
    __shared__ __align__(8) float pl[2][OC_PROJ][Tile::PL];
    const Dims d = a.f.d;
    const int n = a.st->bank.n;
    float lam[OC_PROJ], rl[OC_PROJ];
#pragma unroll
    for (int m = 0; m < OC_PROJ; ++m) {
        lam[m] = a.st->bank.lam[min(m, n - 1)];
        rl[m] = oc_rl(lam[m]);
    }
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + FT_X * ty;
    const int i0 = blockIdx.x * FT_X, j0 = blockIdx.y * FT_Y, kb = blockIdx.z * a.f.zc;
    const int kend = min(kb + a.f.zc, d.nz);
    const int64_t eplane = (int64_t)d.nx * d.ny;
    const Tile tile(d, i0, j0, tid);
    float4 pe[Tile::PF];  // the next plane's elements of this thread, loaded a layer ahead
    float pg[Tile::PF];
    auto prefetch = [&](int gk) {
#pragma unroll
        for (int q = 0; q < Tile::PF; ++q) {
            const int64_t e = tile.exy[q] + gk * eplane;
            const bool in = tile.exy[q] >= 0 && gk >= 0 && gk < d.nz && ANL_IN_RANGE(e, d.ne());
            pe[q] = in ? a.el[e] : make_float4(0.f, 1.f, 0.f, 0.f);
            pg[q] = in ? a.gw[e].x : 0.f;
        }
    };
    prefetch(kb - R);
    const int i = i0 + tx, j = j0 + ty;
    const bool in_xy = i < d.nx && j < d.ny;
    float acc[OC_PROJ][2 * R + 1];
    double vol[OC_PROJ];
#pragma unroll
    for (int m = 0; m < OC_PROJ; ++m) {
        vol[m] = 0.0;
#pragma unroll
        for (int q = 0; q < 2 * R + 1; ++q) acc[m][q] = 0.f;
    }
    for (int gk = kb - R; gk < kend + R; ++gk) {
        float(&buf)[OC_PROJ][Tile::PL] = pl[gk & 1];
#pragma unroll
        for (int q = 0; q < Tile::PF; ++q)
            if (tid + q * FT_N < Tile::PL) {
#pragma unroll
                for (int m = 0; m < OC_PROJ; ++m)  // oc_xn with the element's lambda-free parts
                    buf[m][tid + q * FT_N] = pe[q].y * lam[m] > 1e-30f
                                                 ? fminf(fmaxf(pe[q].x * rl[m], pe[q].z), pe[q].w) : pg[q];
            }
        if (gk + 1 < kend + R) prefetch(gk + 1);
        const int k = gk - R;
        const int64_t e = in_xy && k >= kb ? d.elem(i, j, k) : 0;
        const bool in_e = in_xy && k >= kb && ANL_IN_RANGE(e, d.ne());
        bool fzn = false;
        float hs = 1.f, ph = 0.f;
        if (in_e) {
            ph = a.gw[e].y;  // zero on inactive elements
            hs = a.f.Hs[e];
            fzn = a.f.frozen[e] != 0;
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < OC_PROJ; ++m) {
            filter_plane<R>(a.f.wc, buf[m], tx, ty, acc[m]);
            if (in_e) {
                const float th = tanhf(a.f.beta * (acc[m][0] / hs - a.f.eta));
                const float xp = fzn ? 1.f : (a.f.t0 + th) / (a.f.t0 + a.f.t1);
                vol[m] = R > 2 ? fma(widen(ph), widen(xp), vol[m]) : fma((double)ph, (double)xp, vol[m]);
            }
#pragma unroll
            for (int q = 0; q < 2 * R; ++q) acc[m][q] = acc[m][q + 1];
            acc[m][2 * R] = 0.f;
        }
    }
    static_assert(sizeof(pl) >= OC_PROJ * FT_N * sizeof(double), "the threads' sums in place of the planes");
    const int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    if (reduce_doubles_wide<OC_PROJ, FT_N>(vol, bid, gridDim.x * gridDim.y * gridDim.z, a.partials, a.counter, a.out, tid,
                                           reinterpret_cast<double*>(&pl[0][0][0])) && tid < 32)
        oc_advance(a.st, a.out, OC_PROJ, tid);
}

__global__ void k_oc_weights(int64_t ne, const uint8_t* active, const uint8_t* frozen, const float* phi, float* v,
                             double* partials, unsigned* counter, double* out) {
    __shared__ float2 sm[DT / 32];
    PairSum f[1];
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
        const bool a = active[e] != 0, fz = frozen[e] != 0;
        v[e] = a && !fz ? phi[e] : 0.f;
        if (a && fz) f[0].add(phi[e]);
    }
    finish_pair_sums<1>(f, partials, counter, out, sm);
}

__global__ void k_oc_final(int64_t ne, const uint8_t* active, const uint8_t* frozen, const float* x, const float* dcx,
                           const float* dvx, const OcState* st, float move, float* xnew) {
    const float lam = (float)st->lam;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x)
        xnew[e] = active[e] ? (frozen[e] ? 1.f : oc_xn(x[e], dcx[e], dvx[e], lam, move)) : 0.f;
}

static int read_red(anl_ctx* c, int nv, cudaStream_t s) {
    ANL_CUDA(cudaMemcpyAsync(c->red_h, c->red_out, nv * sizeof(double), cudaMemcpyDeviceToHost, s));
    ANL_CUDA(cudaStreamSynchronize(s));
    return ANL_OK;
}

int oc_update(anl_ctx* c, const float* x, const float* dcx, const float* dvx, const float* phi, const uint8_t* frozen,
              double move, double beta, double eta, double vtarget, float* xnew, int* steps_out, double* lam_out,
              cudaStream_t s) {
    const int64_t ne = c->d.ne();
    ANL_TRY(grow(c->oc_state, c->oc_state_cap, 1, sizeof(OcState)));
    OcState* st = reinterpret_cast<OcState*>(c->oc_state);
    k_oc_scale<<<dgrid(ne), DT, 0, s>>>(ne, c->active, frozen, dcx, dvx, c->partials, c->counter, c->red_out);
    ANL_LAUNCH_CHECK();
    const double mv = beta <= 1 ? move : move / 2;  // optimize.py:151
    ANL_TRY(grow(c->oc_el, c->oc_el_cap, (size_t)ne, sizeof(float4)));
    ANL_TRY(grow(c->oc_gw, c->oc_gw_cap, (size_t)ne, sizeof(float2)));
    const bool linear = !(beta > 0);
    const float* weight = phi;
    if (linear) {  // frozen volume and filtered weights: the volume is linear in xn
        k_oc_weights<<<dgrid(ne), DT, 0, s>>>(ne, c->active, frozen, phi, c->ftmp2, c->partials, c->counter,
                                              c->red_out + 8);
        ANL_LAUNCH_CHECK();
        weight = c->ftmp;
    }
    k_oc_begin<<<1, 32, 0, s>>>(st, c->red_out, linear ? c->red_out + 8 : nullptr, vtarget, linear ? OC_BANK : OC_PROJ);
    ANL_LAUNCH_CHECK();
    if (linear) ANL_TRY(filter_apply(c, false, c->ftmp2, c->ftmp, s));
    k_oc_prep<<<dgrid(ne), DT, 0, s>>>(ne, c->active, frozen, x, dcx, dvx, weight, (float)mv, c->oc_el, c->oc_gw);
    ANL_LAUNCH_CHECK();
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    const int bank_blocks = (int)std::max<int64_t>(1, std::min<int64_t>(sms, (ne + OCB_T - 1) / OCB_T));
    OcProjArgs pa{};
    dim3 pgrid, pblock(FT_X, FT_Y);
    if (!linear) {
        pa.f = filter_args(c);
        pa.f.frozen = frozen;
        pa.f.beta = (float)beta;
        pa.f.eta = (float)eta;
        pa.f.t0 = (float)std::tanh(beta * eta);
        pa.f.t1 = (float)std::tanh(beta * (1 - eta));
        pa.el = c->oc_el;
        pa.gw = c->oc_gw;
        pa.st = st;
        pa.partials = c->partials;
        pa.counter = c->counter;
        pa.out = c->red_out;
        pgrid = filter_grid(pa.f.d);
        if ((int64_t)pgrid.x * pgrid.y * pgrid.z > c->part_cap) {
            set_error("filter reduction needs %d blocks, scratch holds %d", pgrid.x * pgrid.y * pgrid.z, c->part_cap);
            return ANL_ERR_BADARG;
        }
    }
    // the usual number of passes at once (a pass after the last decision returns at once), then
    // two more at a time: every pass or the one after it narrows the bracket at least to half
    int passes = linear ? 4 : 6;
    for (int done = 0; done < 80; done += passes, passes = 2) {
        for (int q = 0; q < passes; ++q) {
            if (linear) {
                k_oc_vol_bank<<<bank_blocks, OCB_T, 0, s>>>(ne, c->oc_el, c->oc_gw, st, c->partials, c->counter,
                                                            c->red_out);
            } else {
                switch (c->filt.R) {
                    case 1: k_oc_vol_proj<1><<<pgrid, pblock, 0, s>>>(pa); break;
                    case 2: k_oc_vol_proj<2><<<pgrid, pblock, 0, s>>>(pa); break;
                    case 3: k_oc_vol_proj<3><<<pgrid, pblock, 0, s>>>(pa); break;
                    case 4: k_oc_vol_proj<4><<<pgrid, pblock, 0, s>>>(pa); break;
                    default: k_oc_vol_proj<5><<<pgrid, pblock, 0, s>>>(pa); break;
                }
            }
            ANL_LAUNCH_CHECK();
        }
        ANL_CUDA(cudaMemcpyAsync(c->red_h, st, offsetof(OcState, tlo), cudaMemcpyDeviceToHost, s));
        ANL_CUDA(cudaStreamSynchronize(s));
        if (reinterpret_cast<const OcState*>(c->red_h)->stop) break;
    }
    if (!reinterpret_cast<const OcState*>(c->red_h)->stop) {
        set_error("OC update: the multiplier's bracket did not close");
        return ANL_ERR_STATE;
    }
    k_oc_final<<<dgrid(ne), DT, 0, s>>>(ne, c->active, frozen, x, dcx, dvx, st, (float)mv, xnew);
    ANL_LAUNCH_CHECK();
    const OcState& r = *reinterpret_cast<const OcState*>(c->red_h);
    if (steps_out) *steps_out = r.steps;
    if (lam_out) *lam_out = r.lam;
    return ANL_OK;
}

// ------------------------------------------------------------------ history statistics

__global__ void k_stats(int64_t ne, const uint8_t* active, const uint8_t* frozen, const float* xold, const float* xnew,
                        const float* xphys, const float* phi, double* partials, unsigned* counter, double* out) {
    // grey count, design count, volume as float-pair sums; the largest change as a fifth
    // partial (a maximum is exact in any order), carried as the pair (max, 0)
    __shared__ float2 sm[4 * DT / 32];
    __shared__ float smax[DT / 32];
    __shared__ bool last;
    PairSum v[3];
    float mx = 0.f;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
        if (!active[e]) continue;
        const float xp = xphys[e];
        float pv, pe;
        two_prod(phi[e], xp, pv, pe);  // the exact product as a pair
        v[2].add(pv);
        v[2].add(pe);
        if (!frozen[e]) {
            mx = fmaxf(mx, fabsf(xnew[e] - xold[e]));
            if (xp > 0.1f && xp < 0.9f) v[0].add(1.f);
            v[1].add(1.f);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    if (lane == 0) smax[warp] = mx;
    float h[3], l[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        h[q] = v[q].h;
        l[q] = v[q].l;
    }
    block_pair_sum<3, DT>(h, l, sm, threadIdx.x);  // its barrier also publishes smax
    float2* p = reinterpret_cast<float2*>(partials);
    if (threadIdx.x == 0) {
        float m = 0.f;
        for (int w = 0; w < DT / 32; ++w) m = fmaxf(m, smax[w]);
        for (int q = 0; q < 3; ++q) p[(int64_t)blockIdx.x * 4 + q] = make_float2(h[q], l[q]);
        p[(int64_t)blockIdx.x * 4 + 3] = make_float2(m, 0.f);
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    float m = 0.f;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        h[q] = 0.f;
        l[q] = 0.f;
    }
    for (unsigned b = threadIdx.x; b < gridDim.x; b += DT) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float2 x = __ldcg(p + (int64_t)b * 4 + q);
            float t, e;
            two_sum_f(h[q], x.x, t, e);
            h[q] = t;
            l[q] += x.y + e;
        }
        m = fmaxf(m, __ldcg(p + (int64_t)b * 4 + 3).x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    __syncthreads();
    if (lane == 0) smax[warp] = m;
    block_pair_sum<3, DT>(h, l, sm, threadIdx.x);
    if (threadIdx.x == 0) {
        float mm = 0.f;
        for (int w = 0; w < DT / 32; ++w) mm = fmaxf(mm, smax[w]);
        double r[3];
        for (int q = 0; q < 3; ++q) r[q] = (double)h[q] + (double)l[q];
        // change, grey fraction of the design elements, volume, design element count
        out[0] = mm;
        out[1] = r[1] > 0 ? r[0] / r[1] : 0.0;
        out[2] = r[2];
        out[3] = r[1];
        *counter = 0u;
    }
}

int design_stats(anl_ctx* c, const float* xold, const float* xnew, const float* xphys, const float* phi,
                 const uint8_t* frozen, double* out, cudaStream_t s) {
    const int64_t ne = c->d.ne();
    k_stats<<<dgrid(ne), DT, 0, s>>>(ne, c->active, frozen, xold, xnew, xphys, phi, c->partials, c->counter, c->red_out);
    ANL_LAUNCH_CHECK();
    ANL_TRY(read_red(c, 4, s));
    for (int q = 0; q < 4; ++q) out[q] = c->red_h[q];
    return ANL_OK;
}

ANL_DEBUG_UNIT(design)

}  // namespace anl
