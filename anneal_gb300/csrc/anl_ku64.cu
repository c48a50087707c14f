// anl_ku64.cu -- the FP64 K u passes of small and middle levels in two kernels.
//
// FP64 arithmetic on this part issues one warp instruction per SM in 16 cycles (19 measured), so an FP64 pass
// costs its instructions on the busiest SM and next to nothing else. The z-marching kernel
// (anl_ku.cu) shares the work in whole CTA layers: 8 warps of about 150 FP64 instructions, 10 us,
// for every layer of its longest z-segment, the halo rows and the layer below included. On a
// 64x32x32 grid that is 50 us where the elements alone take 21 us on 152 SMs, and on the levels
// below 20-30 us where they take 2. Here the first kernel gives every element to one thread, without
// halos, and writes its 8 corner forces; the second sums them at every node in a fixed order and
// applies the pass's epilogue. The forces (192 bytes per element) stay in L2 at these sizes; above
// about 128x64x64 the march is the faster one again (its halo shrinks, the forces go to HBM).
#include "anl_common.cuh"
#include "anl_kernels.cuh"

namespace anl {

namespace {

// F[(3 q + c) ne + e]: the force of element e on its corner q = px + 2 py + 4 pz
__global__ void __launch_bounds__(128) k_ku64_elements(Dims d, const float* __restrict__ E, const double* __restrict__ u,
                                                       KeModal<double> km, double* __restrict__ F, const int* done) {
    if (done != nullptr && *done) return;
    const int ne = (int)d.ne(), e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const int i = e % d.nx, j = e / d.nx % d.ny, k = e / (d.nx * d.ny);
    const int64_t n0 = d.node(i, j, k), sy = d.nx + 1, sz = sy * (d.ny + 1);
    const double Ee = E[e];
    V3<double> f[2][2][2];
    V3<double> v[2][2][2];  // loaded whatever the scale: one latency for both
    if (!ANL_IN_RANGE(n0 + 1 + sy + sz, d.nn())) return;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const double* p = u + 3 * (n0 + (q & 1) + ((q >> 1) & 1) * sy + (q >> 2) * sz);
        v[q & 1][(q >> 1) & 1][q >> 2] = V3<double>{{p[0], p[1]}, p[2]};
    }
    if (Ee != 0.0) {
        V3<double> dxb[2], dxt[2], dyb[2], dyt[2], dz[2][2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            dxb[q] = v[1][q][0] - v[0][q][0];
            dxt[q] = v[1][q][1] - v[0][q][1];
            dyb[q] = v[q][1][0] - v[q][0][0];
            dyt[q] = v[q][1][1] - v[q][0][1];
#pragma unroll
            for (int r = 0; r < 2; ++r) dz[q][r] = v[q][r][1] - v[q][r][0];
        }
        modal_element<double>(km, Ee, dxb, dxt, dyb, dyt, dz, f);
    } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) (&f[0][0][0])[q] = v3zero<double>();
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const V3<double>& c = f[q & 1][(q >> 1) & 1][q >> 2];
        double* o = F + (int64_t)(3 * q) * ne + e;
        o[0] = c.xy.x;
        o[ne] = c.xy.y;
        o[2 * (int64_t)ne] = c.z;
    }
}

constexpr int NT64 = 128;

template <int MODE>
__global__ void __launch_bounds__(NT64) k_ku64_nodes(KuArgs<double> a, const double* __restrict__ F) {
    __shared__ double sred[NT64 / 32];
    if (a.done != nullptr && *a.done) return;
    const Dims d = a.d;
    const int ne = (int)d.ne(), nn = (int)d.nn(), n = blockIdx.x * NT64 + threadIdx.x;
    double dot = 0.0;
    if (n < nn) {
        const int NX = d.nx + 1, NY = d.ny + 1;
        const int i = n % NX, j = n / NX % NY, k = n / (NX * NY);
        const uint8_t nm = a.nmask[n];
        // no load waits for a test: corners outside the grid are read at an element inside. (Not all 24
        // values are in flight at once: the kernel has 32 registers, so they come in groups.)
        double f[8][3];
        bool in[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int ie = i - (q & 1), je = j - ((q >> 1) & 1), ke = k - (q >> 2);
            in[q] = ie >= 0 && je >= 0 && ke >= 0 && ie < d.nx && je < d.ny && ke < d.nz;
            const double* p = F + (int64_t)(3 * q) * ne + (in[q] ? ie + d.nx * (je + d.ny * ke) : 0);
#pragma unroll
            for (int c = 0; c < 3; ++c) f[q][c] = p[(int64_t)c * ne];
        }
        double y[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (in[q])
#pragma unroll
                for (int c = 0; c < 3; ++c) y[c] += f[q][c];
        const int64_t n3 = 3 * (int64_t)n;
        const double inv = MODE == KU_CHEB ? (double)a.diag[n] : 0.0;
        const double c1 = MODE == KU_CHEB && !a.c1_zero ? a.cheb[0] : 0.0, c2 = MODE == KU_CHEB ? a.cheb[1] : 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const bool on = (nm >> c) & 1;
            if (MODE == KU_APPLY || MODE == KU_APPLY_DOT) {
                const double v = on ? y[c] : 0.0;
                a.y[n3 + c] = v;
                if (MODE == KU_APPLY_DOT) dot = fma(a.u[n3 + c], v, dot);
            } else if (MODE == KU_RESID) {
                a.y[n3 + c] = on ? a.b[n3 + c] - y[c] : 0.0;
            } else {
                double dn = 0.0, xn = 0.0;
                if (on) {
                    dn = c2 * (a.b[n3 + c] - y[c]) * inv;
                    if (!a.c1_zero) dn += c1 * a.dv[n3 + c];
                    xn = a.u[n3 + c] + dn;
                }
                if (a.dv_keep) a.dv[n3 + c] = dn;
                a.xout[n3 + c] = xn;
            }
        }
    }
    if (MODE == KU_APPLY_DOT) {
        double v[1] = {dot};
        block_sum<1, NT64>(v, sred, threadIdx.x);
        if (finish_reduction<1, NT64>(v, blockIdx.x, gridDim.x, a.partials, a.counter, a.red_out, threadIdx.x, sred) &&
            threadIdx.x == 0 && a.sc != nullptr)
            pcg_set_step(a.sc);
    }
}

}  // namespace

// Whether a level's FP64 passes take the two kernels: the FP64 instructions of the busiest SM
// (counted at the nominal 16 cycles; with the 19 measured the choice differs for 0.2 % of grids of 4 to
// 256 elements a side), march against elements and nodes, and 8,000 cycles for the second launch.
// One pass, two kernels against the march: 64x32x32 34.9 against 60.2 us, 128x64x64 216 against 252;
// at 256x128x128 the forces alone would be 800 MB and the march takes 1.6 ms.
bool ku64_split(const Dims& d, int sms, int march_ox, int march_oy, int march_warps) {
    if (d.ne() > (1 << 20)) return false;  // 200 MB of forces
    const int64_t planes = (int64_t)ceil_div(d.nx + 1, march_ox) * ceil_div(d.ny + 1, march_oy) * (d.nz + 1);
    const int64_t march = ((planes + sms - 1) / sms + 1) * march_warps * 150;
    const int64_t split = ceil_div(ceil_div(d.ne(), 32), sms) * (int64_t)190 + ceil_div(ceil_div(d.nn(), 32), sms) * (int64_t)35;
    return 16 * split + 8000 < 16 * march;
}

// KU_APPLY, KU_APPLY_DOT, KU_RESID and KU_CHEB; dv is interleaved here (dv[3 n + c])
int launch_ku64(int mode, const KuArgs<double>& a, const KeModal<double>& km, double* F, cudaStream_t s) {
    const int ne = (int)a.d.ne();
    // one warp to a block while that spreads the warps over more SMs
    const int bt = ne <= 32 * 152 * 4 ? 32 : 128, blocks = ceil_div(a.d.nn(), NT64);
    if (mode == KU_APPLY_DOT && blocks > a.partial_capacity) {
        set_error("K u dot: %d blocks exceed the reduction scratch (%d)", blocks, a.partial_capacity);
        return ANL_ERR_BADARG;
    }
    k_ku64_elements<<<ceil_div(ne, bt), bt, 0, s>>>(a.d, a.E, a.u, km, F, a.done);
    ANL_LAUNCH_CHECK();
    switch (mode) {
        case KU_APPLY: k_ku64_nodes<KU_APPLY><<<blocks, NT64, 0, s>>>(a, F); break;
        case KU_APPLY_DOT: k_ku64_nodes<KU_APPLY_DOT><<<blocks, NT64, 0, s>>>(a, F); break;
        case KU_RESID: k_ku64_nodes<KU_RESID><<<blocks, NT64, 0, s>>>(a, F); break;
        case KU_CHEB: k_ku64_nodes<KU_CHEB><<<blocks, NT64, 0, s>>>(a, F); break;
        default: return ANL_ERR_BADARG;
    }
    ANL_LAUNCH_CHECK();
    return ANL_OK;
}

ANL_DEBUG_UNIT(ku64)

}  // namespace anl
