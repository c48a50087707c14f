// anl_ctx.cuh -- the solver context behind the opaque anl_ctx handle.
#pragma once

#include <vector>

#include "anl_common.cuh"
#include "anl_kernels.cuh"

namespace anl {

// One level of the voxel hierarchy. Level 0 is the user's grid; level l+1 halves every
// element dimension (rounded up). Vectors are in the context's precision T.
struct Level {
    Dims d{};
    float* E = nullptr;       // element scale (times h at level 0; children sum / 4 below)
    uint8_t* eact = nullptr;  // element is (or covers) an active element
    uint8_t* nmask = nullptr; // node mask bits
    float* diag = nullptr;    // inverse diagonal of K per node (the same for its 3 DOFs; 0 if unused)
    void* x = nullptr;        // V-cycle iterate (level 0: z = M r)
    void* xt = nullptr;       // Chebyshev double buffer
    void* b = nullptr;        // right-hand side (level 0: the CG residual r)
    void* r = nullptr;        // residual scratch
    void* dv = nullptr;       // Chebyshev direction
    double lmax = 0.0;        // upper end of the smoothed spectrum of D^-1 K (diagnostics)
    // x, xt, b, r and dv hold one vector per right-hand-side slot, vs values apart (3 nn
    // rounded up to 64 values, so every slot starts on a 256-byte boundary)
    int64_t vs = 0;
    bool split = false;       // FP64 contexts: the level's K u passes are anl_ku64.cu's
};

constexpr int kMaxFilterR = 5;
// the taps of a filter layer by (|dx|, |dy|) in either order
constexpr int kFilterClasses = (kMaxFilterR + 1) * (kMaxFilterR + 2) / 2;
__host__ __device__ constexpr int filter_class(int a, int b) {
    return a >= b ? a * (a + 1) / 2 + b : b * (b + 1) / 2 + a;
}

struct FilterState {
    bool ready = false;
    int R = 0;
    double r = 0.0;
    float wc[kMaxFilterR + 1][kFilterClasses];  // cone weights by |dz| and class
    float* Hs = nullptr;                        // conv(active), zeros replaced by 1
};

constexpr int kChebMax = 32;
constexpr int kChebStride = 1 + 2 * kChebMax;

}  // namespace anl

struct anl_ctx {
    anl::Dims d{};
    double h = 1.0, nu = 0.3;
    int flags = 0;
    bool fp64 = false;
    size_t tsize = 4;  // bytes per vector entry

    double ke[576];                 // Ke(1) row-major (host)
    double* ke_d = nullptr;         // Ke(1) on the device (coarse assembly)
    anl::KeBlocks<double> kbd{};  // the reflection structure of Ke (checked at creation)
    anl::KeModal<double> kmd{};
    anl::KeModal<float> kmf{};
    anl::KeModal<anl::DF> kmdf{};  // kmd as double-floats (the accurate residual)
    double kdiag = 0.0;
    // lambda_max(Ke) / Ke_00 >= lambda_max(D^-1 K) for every field of element scales (the
    // element-by-element bound: x.Kx = sum_e E_e x_e.Ke x_e <= bound sum_e E_e Ke_00 |x_e|^2)
    double lmax_bound = 0.0;

    bool domain_set = false;
    int64_t nfree = 0;
    uint8_t* active = nullptr;      // level-0 active flags (ne)
    std::vector<anl::Level> lev;
#ifndef ANL_MG_DEGREE
#define ANL_MG_DEGREE 2  // Chebyshev steps per pre- and post-smoothing
#endif
    int mg_degree = ANL_MG_DEGREE;
    // Levels 2 and below: their launches cost about the same whatever their size (launch and
    // pipeline-fill latency), so more and deeper smoothing there is nearly free and saves CG
    // iterations. Measured on the 256x128x128 L-bracket (interval low ends fine / coarse,
    // coarse degree: CG iterations per solve, SIMP iterations/s):
    //   0.05 / 0.05, 2: 48.3, 21.4     0.05 / 0.05, 6: 32.6, 25.3    0.03 / 0.01, 6: 28.8, 28.2
    //   0.03 / 0.002, 6: 27.7, 29.2    0.03 / 0.002, 8: 24.1, 30.4   0.03 / 0.0005, 8: 24.5, 30.0
    // FP64 contexts take 5 steps from 0.006: there a step on these levels costs 3-10 us of FP64 issue
    // (an as-built solve at 64x32x32, low end and degree: ms, CG iterations)
    //   0.002, 8: 56.4, 96   0.004, 6: 50.7, 97   0.006, 5: 47.0, 96   0.01, 4: 45.9, 101   0.03, 3: 47.0, 112
    // and at 96x48x48
    //   0.002, 8: 94.3, 90   0.004, 6: 85.0, 88   0.006, 5: 81.3, 88   0.01, 4: 83.0, 94    0.03, 3: 89.5, 107
#ifndef ANL_MG_DEGREE_COARSE
#define ANL_MG_DEGREE_COARSE 8
#endif
#ifndef ANL_MG_DEGREE_COARSE64
#define ANL_MG_DEGREE_COARSE64 5
#endif
    int mg_degree_coarse = ANL_MG_DEGREE_COARSE;
    int degree(size_t l) const { return l >= 2 ? mg_degree_coarse : mg_degree; }
    // the finest level's K u passes on the tensor cores (anl_kutc.cu; FP32 contexts)
    bool use_tc = false;
    // first level of the V-cycle tail (anl_vtail.cu), -1 for none, and the CTAs of
    // its cluster
    int tail_from = -1, tail_ctas = 0;
    int tail_lose_from = 1 << 30;  // TailArgs::lose_from (ANL_TAIL_LOSE_FROM)
    // right-hand-side slots (ANL_FLAG_RHS): the solve's per-vector state (the hierarchy's
    // vectors, p, q, the FP64 solution and right-hand side, its float-pair split, the PCG
    // scalars, the restart flags, the reduction scratch) exists once per slot; a batched solve
    // advances rb slots in lockstep, every kernel of its CG chunk taking its slot from the grid
    int rmax = 1;
    int rb = 1;                   // slots of the chunk being enqueued (1 outside a batched solve)
    int slot = 0;                 // the slot the single-vector code paths work on
    std::vector<int> last_status; // each right-hand side's status in the last anl_solve
    int cg_rb = 0;                // slots of the captured CG chunk
    int64_t part_stride = 0;      // doubles of reduction scratch per slot
    int* restart_d = nullptr;     // per-slot restart flags (p = z on the next direction update)
    // slot 0 of the per-slot arrays (the single-vector code paths point at one slot at a time)
    void* b0_base = nullptr;
    double* xbuf_base = nullptr;
    double* bbuf_base = nullptr;
    void* bdf_base = nullptr;
    anl::PcgScalars* sc_base = nullptr;
    anl::DF* sens_df = nullptr;  // the sensitivity's displacements as float pairs (grows)
    size_t sens_df_cap = 0;
    float4* oc_el = nullptr;     // the OC update's lambda-free element data (grows)
    size_t oc_el_cap = 0;
    float2* oc_gw = nullptr;
    size_t oc_gw_cap = 0;
    double* oc_state = nullptr;  // the OC bisection's device state (OcState, anl_design.cu)
    size_t oc_state_cap = 0;
    float* ainv_hi = nullptr;  // the coarsest dense inverse as float pairs (the tail's coarse solve)
    float* ainv_lo = nullptr;
#ifndef ANL_CHEB_LO
#define ANL_CHEB_LO 0.1
#endif
#ifndef ANL_CHEB_LO_COARSE
#define ANL_CHEB_LO_COARSE 0.002
#endif
#ifndef ANL_CHEB_LO_COARSE64
#define ANL_CHEB_LO_COARSE64 0.006
#endif
    // Lower ends of the smoothed intervals, as fractions of their upper end (levels 0-1, 2+). With
    // two steps 0.1 damps what the next level cannot represent and leaves the rest to it; CG
    // iterations per solve with 0.03, 0.1, 0.15, 0.2: developed designs at 256x128x128 46.3, 39.0,
    // 39.7, 48.0, at 97x53x34 23.7, 22.3, 23.0, 24.0; SIMP runs from a uniform design at 256x128x128
    // 27.0, 26.3, 27.1, 27.9, at 113x41x57 20.2, 19.6, 19.7, 20.2.
    double cheb_lo = ANL_CHEB_LO, cheb_lo_coarse = ANL_CHEB_LO_COARSE;
    // per level: {lambda_max bound, then (c1, c2) for up to kChebMax steps}, read by the
    // smoothing kernels from device memory
    double* cheb_d = nullptr;

    // coarsest level: dense inverse or a Chebyshev fallback when too large
    int nc = 0;
    bool dense_coarse = false;
    bool coarse_ready = false;
    double* A = nullptr;     // nc x nc, scratch of the inversion
    double* Ainv = nullptr;  // nc x nc inverse
    double* coarse_dmax = nullptr;  // largest diagonal entry of the coarsest matrix

    // CG vectors (precision T) and FP64 solution / right-hand side
    void* p = nullptr;
    void* q = nullptr;
    void* xhi = nullptr;
    void* xlo = nullptr;
    void* xdf = nullptr;  // FP32 mode: x as (hi, lo) float pairs for the accurate residual
    void* bdf = nullptr;  // FP32 mode: the right-hand side as (hi, lo) float pairs
    void* y1 = nullptr;
    void* y2 = nullptr;
    void* tmp = nullptr;
    double* f64 = nullptr;  // FP64 mode: the element forces of the split levels
    double* xbuf = nullptr;
    double* bbuf = nullptr;

    anl::PcgScalars* sc = nullptr;    // device
    anl::PcgScalars* sc_h = nullptr;  // pinned host mirror

    // reduction scratch
    double* partials = nullptr;
    unsigned* counter = nullptr;
    double* red_out = nullptr;  // small device result area
    double* red_h = nullptr;    // pinned host mirror
    int part_cap = 0;

    // the CG iteration chunk as a CUDA graph, captured on an internal stream and replayed on
    // the caller's stream; invalidated whenever the hierarchy's smoother spectra change
    cudaStream_t cap_stream = nullptr;
    cudaGraphExec_t cg_exec = nullptr;
    bool cg_valid = false;
    int cg_nodes = 0;
    bool use_graph = true;

    anl::FilterState filt;
    float* ftmp = nullptr;   // element-field scratch (ne)
    float* ftmp2 = nullptr;  // element-field scratch (ne)
};
