// anl_vtail.cu -- the small levels of the V-cycle in one thread-block cluster, in shared memory.
//
// On a level of at most a few thousand elements a smoothing step is pure latency: as a launch of
// its own it costs 6-7 us whatever it moves, and there are some 17 of them per level and V-cycle.
// Here one cluster (16 CTAs, 8 where the part cannot place 16) takes the right-hand side of the
// first level that fits it and returns its V-cycle correction: it smooths, restricts, solves the
// coarsest grid with the dense inverse (kept as float pairs), prolongs and smooths back up. The
// arithmetic is that of the per-level kernels: the modal element product (modal_element),
// Chebyshev on D^-1 K with the level's coefficients, trilinear transfers, masks on fixed DOFs.
//
// A level is cut into slabs of element layers along AXIS, the first level's longest side. A CTA
// owns its layers' lower node planes (the last CTA also the top plane) and computes its own
// element layers and the one below, so a step needs its neighbours' boundary planes of the
// iterate and nothing else:
//   1. every element writes its 8 corner forces to shared memory;
//   2. __syncthreads; every owned node sums the forces that meet there in a fixed order, applies
//      its Chebyshev update and writes its new value to its own copy of the iterate and, from a
//      boundary plane, to the neighbour's halo plane: st.async into distributed shared memory,
//      counted by the neighbour's mbarrier;
//   3. the CTA waits for its own two halo planes only (FP32: only the elements at them do, the
//      others are computed meanwhile). The iterate is double-buffered and there is
//      a barrier per direction and buffer: a neighbour can be one step ahead, never two, since it
//      needs this CTA's plane of every step. (A cluster barrier a step costs 0.9 us: its release
//      drains the remote stores first.)
// A node stays with its thread for a whole sweep: its right-hand side, direction, inverse
// diagonal and mask stay in registers. A level's forces have a zero row and column between their
// rows, so a node sums 8 corners without a test; they lie 25 words apart (an odd stride, so
// neither phase has bank conflicts). The transfers between levels, whose slabs do not match, go
// through the levels' vectors in global memory, every load of a node in flight at once.
//
// What bounds it: the chain of one step (about 48 shared-memory accesses and 250 instructions per
// element, then 24 and 80 per node, the halo's flight, two block barriers). The tail's own vectors
// between levels are in slab-major order, so a warp's loads of them coalesce whatever the axis.
#include "anl_common.cuh"
#include "anl_kernels.cuh"

namespace anl {

namespace {

// TT: threads of a CTA, NPT: owned nodes of a thread. Levels of at most ALONE elements stay in one
// CTA; levels with more than MOST elements in a CTA are left to launches of their own.
template <class T>
struct TailCfg;
template <>
struct TailCfg<float> {
    // one CTA's step takes 0.9 us at 128 elements, shorter than a shared one, whose halo flight
    // alone takes 0.7 us; at 432 it is not (2 us)
    static constexpr int TT = 512, NPT = 2, ALONE = 256, MOST = 1 << 30;
    // EARLY: only the elements that need a halo plane wait for it, the others work meanwhile (per CG
    // iteration 96x48x48 185.2 -> 181.8 us, 256x128x128 850.9 -> 841.0; in FP64, where a CTA has one
    // layer of its own and so no such element, the test costs 1 %)
    static constexpr bool EARLY = true;
};
template <>
struct TailCfg<double> {
    // A warp of elements holds the FP64 pipe for 1.6 us (176 instructions, 19 cycles each), so one
    // CTA takes no more than one warp of them, and above five warps in each of 16 CTAs the 152 SMs
    // of a launch are faster again.
    static constexpr int TT = 256, NPT = 2, ALONE = 32, MOST = 160;
    static constexpr bool EARLY = false;
};
constexpr int FW = 25;          // words between two elements' forces (24 and one of padding)
constexpr int kWaitTries = 1 << 20;  // bound of a halo wait
constexpr int kTailMaxDegree = 16;  // Chebyshev steps per sweep there is room for

// A level's slabs: A x B elements per layer, L layers along the tail's axis, `per` layers to a CTA.
TailGeo slab_geo(int axis, const Dims& d, int ctas, int alone) {
    const int n[3] = {d.nx, d.ny, d.nz};
    const int ax = axis == 0 ? 1 : 0, bx = axis == 2 ? 1 : 2;
    const int nstr[3] = {1, d.nx + 1, (d.nx + 1) * (d.ny + 1)}, estr[3] = {1, d.nx, d.nx * d.ny};
    TailGeo g;
    g.A = n[ax];
    g.B = n[bx];
    g.L = n[axis];
    g.ns = nstr[axis], g.na = nstr[ax], g.nb = nstr[bx];
    g.es = estr[axis], g.ea = estr[ax], g.eb = estr[bx];
    const int use = d.ne() <= alone ? 1 : ctas;
    g.per = (g.L + use - 1) / use;
    g.active = (g.L + g.per - 1) / g.per;
    g.PA = g.A + 1;
    g.planeN = g.PA * (g.B + 1);
    // the slab-major node order of the tail's own vectors: index = s planeN + b PA + a
    g.p[axis] = g.planeN;
    g.p[ax] = 1;
    g.p[bx] = g.PA;
    return g;
}
// sizes that hold for every CTA
int max_nodes(const TailGeo& g) { return (g.per + 1) * g.planeN; }
int max_elems(const TailGeo& g) { return (g.per + (g.active > 1 ? 1 : 0)) * g.A * g.B; }
int max_padded(const TailGeo& g) { return (g.per + 2) * g.planeN + g.A + 2; }

// shared-memory carve-up in values of the context's precision: the iterate twice (own planes and two halo planes), the coarsest
// right-hand side, then per level the forces and the elements' (scale, packed indices) pairs
template <class T>
TailLayout tail_layout(const TailLevel<T>* lev, int nlev) {
    TailLayout t{};
    for (int l = 0; l < nlev - 1; ++l) t.xlen = std::max(t.xlen, 3 * (max_nodes(lev[l].g) + 2 * lev[l].g.planeN));
    t.xlen = (t.xlen + 3) / 4 * 4;
    int o = 2 * t.xlen;
    for (int l = 0; l < nlev - 1; ++l) {
        t.e[l] = o;
        o += ((int)(sizeof(float2) / sizeof(T)) * max_elems(lev[l].g) + 3) / 4 * 4;
        t.f[l] = o;
        t.flen[l] = (FW * max_padded(lev[l].g) + 3) / 4 * 4;
        o += t.flen[l];
    }
    t.c = o;
    t.words = o + 3 * (int)lev[nlev - 1].d.nn();
    return t;
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// one value to another CTA of the cluster, counted on that CTA's barrier
__device__ __forceinline__ void st_async(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
                 "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// false once the wait has run out
__device__ __forceinline__ bool bar_wait(uint32_t bar, unsigned parity) {
    for (int q = 0; q < kWaitTries; ++q) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

// components c0 .. c0 + NC - 1 of (R r)(I, J, K): trilinear weights 1, 1/2, 1/4, 1/8 of the fine
// residual r (slab-major, strides p); nodes outside the grid are read at its edge with weight 0, so
// no load depends on a test and a plane's loads are in flight together
template <int NC, class T>
__device__ __forceinline__ void restrict_at(const TailLevel<T>& f, const T* r, int I, int J, int K, int c0, T (&acc)[NC]) {
    const Dims& d = f.d;
    const int px = 3 * f.g.p[0], py = 3 * f.g.p[1], pz = 3 * f.g.p[2];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = T(0);
#pragma unroll 1
    for (int dk = -1; dk <= 1; ++dk) {
        const int k = 2 * K + dk;
        const T* p = r + pz * min(max(k, 0), d.nz) + c0;
        const T wk = k < 0 || k > d.nz ? T(0) : dk ? T(0.5) : T(1);
        T v[9][NC];
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const int i = min(max(2 * I + q % 3 - 1, 0), d.nx), j = min(max(2 * J + q / 3 - 1, 0), d.ny);
#pragma unroll
            for (int c = 0; c < NC; ++c) v[q][c] = p[px * i + py * j + c];
        }
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const int di = q % 3 - 1, dj = q / 3 - 1, i = 2 * I + di, j = 2 * J + dj;
            const bool in = i >= 0 && j >= 0 && i <= d.nx && j <= d.ny;
            const T w = in ? (di ? T(0.5) : T(1)) * (dj ? T(0.5) : T(1)) * wk : T(0);
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[c] = fma(w, v[q][c], acc[c]);
        }
    }
}

// (P xc)(i, j, k): the mean of the coarse nodes the fine node lies between (the unused ones of the
// 8 are read at the node itself); xc has node strides p
template <class T>
__device__ __forceinline__ void prolong_at(const int (&p)[3], const T* xc, int i, int j, int k, T (&acc)[3]) {
    const int di = i & 1, dj = j & 1, dk = k & 1;
    const int n0 = (i >> 1) * p[0] + (j >> 1) * p[1] + (k >> 1) * p[2];
    T v[8][3];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int n = n0 + (q & di) * p[0] + ((q >> 1) & dj) * p[1] + ((q >> 2) & dk) * p[2];
#pragma unroll
        for (int c = 0; c < 3; ++c) v[q][c] = xc[3 * n + c];
    }
    const T w = (di ? T(0.5) : T(1)) * (dj ? T(0.5) : T(1)) * (dk ? T(0.5) : T(1));
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[c] = T(0);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        if (((q & 1) && !di) || ((q & 2) && !dj) || ((q & 4) && !dk)) continue;
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += v[q][c];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[c] *= w;
}

// an owned node of this thread on the current level
template <class T>
struct TailNode {
    int pn;         // node index in slab-major order, -1 for none
    int gn;         // node index on the level's grid
    int nl;         // first value of the node in an iterate buffer
    int nb;         // first value of the padded element above it in every direction
    int i, j, k;
    unsigned m;     // mask
    T g;            // inverse diagonal
    T b[3], d[3], x[3];
    int down, up;   // its copies in the neighbours' halo planes, -1 for none
};

template <class T, int AXIS>
struct Tail {
    static constexpr int TT = TailCfg<T>::TT, NPT = TailCfg<T>::NPT;
    const TailArgs<T>& a;
    T* sm;
    uint32_t bar;                 // this CTA's barriers: [direction][buffer], 8 bytes each
    uint32_t x_down, x_up, b_down, b_up;  // the neighbours' iterate buffers and barriers
    int tid, rank, ctas, slot;
    int cur = 0;                  // the buffer that holds the iterate
    unsigned phase = 0;           // next phase parity of barrier [direction][buffer], one bit each
    unsigned due = 0;             // per direction: 1 + the parity the last exchange's halo plane completes, or 0
    bool lost = false;            // a halo wait of this thread ran out
    TailNode<T> nd[NPT];

    __device__ T* vec(T* p, int l) const { return p + (int64_t)slot * a.lev[l].vs; }

    __device__ int own(const TailGeo& g) const { return rank < g.active ? min(g.per, g.L - rank * g.per) : 0; }
    // element layers the CTA computes: its own and, but for the first CTA, the one below
    __device__ int first_layer(const TailGeo& g) const { return g.active > 1 ? rank * g.per - 1 : 0; }
    __device__ int elems(const TailGeo& g) const {
        const int o = own(g);
        return o > 0 ? (o + (g.active > 1 ? 1 : 0)) * g.A * g.B : 0;
    }

    // the element table of level l and its zeroed forces (once per launch)
    __device__ void table(int l) {
        const TailLevel<T>& lv = a.lev[l];
        const TailGeo& g = lv.g;
        float4* f = reinterpret_cast<float4*>(sm + a.lay.f[l]);
        for (int t = tid; t < a.lay.flen[l] / (16 / (int)sizeof(T)); t += TT) f[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int layer = g.A * g.B, ne = elems(g), first = first_layer(g), q0 = g.active > 1 ? 0 : 1;
        float2* et = reinterpret_cast<float2*>(sm + a.lay.e[l]);
        for (int e = tid; e < ne; e += TT) {
            const int q = e / layer, in = e - q * layer, b = in / g.A, aa = in - b * g.A;
            const int ge = (first + q) * g.es + aa * g.ea + b * g.eb;
            const float Ee = first + q >= 0 && ANL_IN_RANGE(ge, lv.d.ne()) ? __ldg(lv.E + ge) : 0.f;
            // node plane 0 is the halo below; a level in one CTA starts at plane 1
            const int n0 = (q + q0) * g.planeN + aa + g.PA * b, pe = ((q + q0) * (g.B + 1) + b + 1) * g.PA + aa + 1;
            // the top bit: the element has nodes of a halo plane
            const bool halo = g.active > 1 && ((q == 0 && rank > 0) || (first + q + 1 == (rank + 1) * g.per && rank + 1 < g.active));
            et[e] = make_float2(Ee, __int_as_float(n0 | (pe << 16) | (halo ? 0x80000000 : 0)));
        }
    }

    // this thread's nodes of level l
    __device__ void enter(int l) {
        const TailLevel<T>& lv = a.lev[l];
        const TailGeo& g = lv.g;
        const int o = own(g), nown = o > 0 ? o + (rank == g.active - 1 ? 1 : 0) : 0;
#pragma unroll
        for (int r = 0; r < NPT; ++r) {
            TailNode<T>& n = nd[r];
            const int t = tid + r * TT;
            n.pn = -1;
            n.m = 0;
            n.g = T(0);
#pragma unroll
            for (int c = 0; c < 3; ++c) n.b[c] = n.d[c] = n.x[c] = T(0);
            if (t >= nown * g.planeN) continue;
            const int p = 1 + t / g.planeN, in = t - (p - 1) * g.planeN, b = in / g.PA, aa = in - b * g.PA;
            const int s = rank * g.per + p - 1;
            n.gn = s * g.ns + aa * g.na + b * g.nb;
            if (!ANL_IN_RANGE(n.gn, lv.d.nn())) continue;
            n.pn = s * g.planeN + in;
            n.nl = 3 * (p * g.planeN + in);
            n.nb = FW * ((p * (g.B + 1) + b + 1) * g.PA + aa + 1);
            n.i = AXIS == 0 ? s : aa;
            n.j = AXIS == 1 ? s : AXIS == 0 ? aa : b;
            n.k = AXIS == 2 ? s : b;
            n.m = __ldg(lv.nmask + n.gn) & 7u;
            n.g = T(__ldg(lv.diag + n.gn));
            n.down = p == 1 && rank > 0 ? 3 * ((g.per + 1) * g.planeN + in) : -1;
            n.up = p == nown && rank + 1 < g.active ? 3 * in : -1;
        }
    }

    // the nodes' x into the other buffer and the neighbours' halo planes; with EARLY the threads whose
    // elements need the own halo planes wait for them there (wait_halo), otherwise every thread here
    __device__ void exchange(int l) {
        const TailGeo& g = a.lev[l].g;
        cur ^= 1;
        const bool from[2] = {rank > 0 && rank < g.active, rank + 1 < g.active};
        if (tid == 0) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
                if (from[q]) bar_expect(bar + 8u * (2 * q + cur), 3u * (unsigned)sizeof(T) * (unsigned)g.planeN);
        }
        const int o = cur * a.lay.xlen;
#pragma unroll
        for (int r = 0; r < NPT; ++r) {
            const TailNode<T>& n = nd[r];
            if (n.pn < 0) continue;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                // this CTA lies above rank - 1 and below rank + 1
                if (n.down >= 0) st_async(x_down + (unsigned)sizeof(T) * (unsigned)(o + n.down + c), n.x[c], b_down + 8u * (2 + cur));
                if (n.up >= 0) st_async(x_up + (unsigned)sizeof(T) * (unsigned)(o + n.up + c), n.x[c], b_up + 8u * cur);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) sm[o + n.nl + c] = n.x[c];
        }
        due = 0;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (!from[q]) continue;
            const unsigned bit = 2 * q + cur;
            due |= (1u + ((phase >> bit) & 1u)) << (2 * q);
            phase ^= 1u << bit;
        }
        if (!TailCfg<T>::EARLY) wait_halo();
        __syncthreads();
    }

    // This thread's wait for the halo planes of the last exchange. Some thread of the CTA waits in every
    // step (each side's halo plane has elements at it), and all pass a barrier after that, so the
    // next use of an mbarrier finds this phase complete.
    __device__ void wait_halo() {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const unsigned w = (due >> (2 * q)) & 3u;
            if (w != 0 && !lost) lost = !bar_wait(bar + 8u * (2 * q + cur), w - 1u);
        }
    }

    // the corner forces of the CTA's elements (corner pa + 2 pb + 4 ps in slab directions)
    __device__ void elements(int l) {
        const TailGeo& g = a.lev[l].g;
        const int ne = elems(g);
        const T* x = sm + cur * a.lay.xlen;
        const float2* et = reinterpret_cast<const float2*>(sm + a.lay.e[l]);
        T* F = sm + a.lay.f[l];
        const int sx = 3 * g.p[0], sy = 3 * g.p[1], sz = 3 * g.p[2];
        bool waited = false;
        for (int e = tid; e < ne; e += TT) {
            const float2 te = et[e];
            const int tab = __float_as_int(te.y);
            if (TailCfg<T>::EARLY && tab < 0 && !waited) {
                wait_halo();
                waited = true;
            }
            if (te.x == 0.f) continue;  // its forces stay the zeros of table()
            const T* p0 = x + 3 * (tab & 0xffff);
            V3<T> u[2][2][2];
#pragma unroll
            for (int pz = 0; pz < 2; ++pz)
#pragma unroll
                for (int py = 0; py < 2; ++py)
#pragma unroll
                    for (int px = 0; px < 2; ++px) {
                        const T* p = p0 + px * sx + py * sy + pz * sz;
                        u[px][py][pz].xy.x = p[0];
                        u[px][py][pz].xy.y = p[1];
                        u[px][py][pz].z = p[2];
                    }
            V3<T> dxb[2], dxt[2], dyb[2], dyt[2], dz[2][2], f[2][2][2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                dxb[q] = u[1][q][0] - u[0][q][0];
                dxt[q] = u[1][q][1] - u[0][q][1];
                dyb[q] = u[q][1][0] - u[q][0][0];
                dyt[q] = u[q][1][1] - u[q][0][1];
            }
#pragma unroll
            for (int px = 0; px < 2; ++px)
#pragma unroll
                for (int py = 0; py < 2; ++py) dz[px][py] = u[px][py][1] - u[px][py][0];
            modal_element<T>(a.km, T(te.x), dxb, dxt, dyb, dyt, dz, f);
            T* fo = F + FW * ((tab >> 16) & 0x7fff);
#pragma unroll
            for (int pz = 0; pz < 2; ++pz)
#pragma unroll
                for (int py = 0; py < 2; ++py)
#pragma unroll
                    for (int px = 0; px < 2; ++px) {
                        const int pa = AXIS == 0 ? py : px, pb = AXIS == 2 ? py : pz;
                        const int ps = AXIS == 0 ? px : AXIS == 1 ? py : pz;
                        const int q = pa + 2 * pb + 4 * ps;
                        fo[3 * q] = f[px][py][pz].xy.x;
                        fo[3 * q + 1] = f[px][py][pz].xy.y;
                        fo[3 * q + 2] = f[px][py][pz].z;
                    }
        }
        __syncthreads();
    }

    // (K x)(n): the 8 corners that meet at the node, in a fixed order
    __device__ void force(int l, const TailNode<T>& n, T (&y)[3]) const {
        const TailGeo& g = a.lev[l].g;
        const T* F = sm + a.lay.f[l] + n.nb;
        y[0] = y[1] = y[2] = T(0);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const T* p = F - FW * ((q & 1) + ((q >> 1) & 1) * g.PA + (q >> 2) * g.planeN) + 3 * q;
#pragma unroll
            for (int c = 0; c < 3; ++c) y[c] += p[c];
        }
    }

    // one Chebyshev step
    __device__ void step(int l, T c1, T c2) {
        elements(l);
#pragma unroll
        for (int r = 0; r < NPT; ++r) {
            TailNode<T>& n = nd[r];
            if (n.m == 0) continue;
            T y[3];
            force(l, n, y);
            const T gn = c2 * n.g;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T dn = (n.m >> c) & 1 ? c1 * n.d[c] + (n.b[c] - y[c]) * gn : T(0);
                n.d[c] = dn;
                n.x[c] += dn;
            }
        }
        exchange(l);
    }
};

template <class T, int AXIS>
__global__ void __launch_bounds__(TailCfg<T>::TT, 1) k_vtail(const __grid_constant__ TailArgs<T> a) {
    constexpr int TT = TailCfg<T>::TT, NPT = TailCfg<T>::NPT;
    extern __shared__ __align__(16) unsigned char tail_bytes[];
    T* tail_smem = reinterpret_cast<T*>(tail_bytes);
    __shared__ T cf[kTailMaxLevels][2 * kTailMaxDegree];
    __shared__ __align__(8) uint64_t bars[2][2];
    __shared__ int cta_lost;
    const int tid = threadIdx.x, ctas = a.ctas;
    const int rank = blockIdx.x % ctas, slot = blockIdx.x / ctas;
    const int* done = slot_bytes(a.done, slot, a.sc_bytes);
    if (done != nullptr && *done) return;  // the same for the whole cluster
    const int last = a.nlev - 1;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&bars[0][0]);
    if (tid == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8u * q) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        cta_lost = 0;
    }
    for (int q = tid; q < last * 2 * kTailMaxDegree; q += TT) {
        const int l = q / (2 * kTailMaxDegree), k = q - l * 2 * kTailMaxDegree;
        if (k < 2 * a.lev[l].degree) cf[l][k] = T(a.lev[l].cheb[k]);
    }
    __syncthreads();
    Tail<T, AXIS> t{a, tail_smem, bar, 0, 0, 0, 0, tid, rank, ctas, slot};
    {
        const uint32_t xb = (uint32_t)__cvta_generic_to_shared(tail_smem);
        const int below = rank > 0 ? rank - 1 : 0, above = rank + 1 < ctas ? rank + 1 : rank;
        t.x_down = map_rank(xb, below);
        t.x_up = map_rank(xb, above);
        t.b_down = map_rank(bar, below);
        t.b_up = map_rank(bar, above);
    }
    for (int l = 0; l < last; ++l) t.table(l);
    cluster_sync();  // every CTA's barriers are ready before its shared memory is written

    for (int l = 0; l < last; ++l) {  // down: smooth from zero, residual
        const int deg = a.lev[l].degree;
        t.enter(l);
#pragma unroll
        for (int r = 0; r < NPT; ++r) {
            TailNode<T>& n = t.nd[r];
            if (n.pn < 0) continue;
            if (l == 0) {
#pragma unroll
                for (int c = 0; c < 3; ++c) n.b[c] = __ldg(t.vec(a.b0, 0) + 3 * n.gn + c);
            } else {
                restrict_at<3, T>(a.lev[l - 1], t.vec(a.lev[l - 1].r, l - 1), n.i, n.j, n.k, 0, n.b);
            }
            const T gn = cf[l][1] * n.g;  // step 0: x = d = c2_0 D^-1 b
            T* save = t.vec(a.lev[l].b, l) + 3 * n.pn;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (!((n.m >> c) & 1)) n.b[c] = T(0);
                n.x[c] = n.d[c] = gn * n.b[c];
                if (l > 0) save[c] = n.b[c];
            }
        }
        t.exchange(l);
        for (int k = 1; k < deg; ++k) t.step(l, cf[l][2 * k], cf[l][2 * k + 1]);
        t.elements(l);
        T* res = t.vec(a.lev[l].r, l);
        T* save = t.vec(a.lev[l].xt, l);
#pragma unroll
        for (int r = 0; r < NPT; ++r) {
            const TailNode<T>& n = t.nd[r];
            if (n.pn < 0) continue;
            T y[3] = {T(0), T(0), T(0)};
            if (n.m) t.force(l, n, y);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                res[3 * n.pn + c] = (n.m >> c) & 1 ? n.b[c] - y[c] : T(0);
                save[3 * n.pn + c] = n.x[c];
            }
        }
        cluster_sync();
    }

    {  // the coarsest grid: its right-hand side in every CTA, the rows of the inverse shared out
        const Dims d = a.lev[last].d;
        T* bc = tail_smem + a.lay.c;
        const T* rf = t.vec(a.lev[last - 1].r, last - 1);
        for (int q = tid; q < 3 * (int)d.nn(); q += TT) {
            const int N = q / 3, c = q - 3 * N;
            const int K = N / ((d.nx + 1) * (d.ny + 1)), J = N / (d.nx + 1) % (d.ny + 1), I = N % (d.nx + 1);
            const unsigned m = __ldg(a.lev[last].nmask + N);
            T v[1];
            restrict_at<1, T>(a.lev[last - 1], rf, I, J, K, c, v);
            bc[q] = (m >> c) & 1 ? v[0] : T(0);
        }
        __syncthreads();
        const int n = a.nc, lane = tid & 31;
        T* xc = t.vec(a.lev[last].x, last);
        for (int row = rank * (TT / 32) + (tid >> 5); row < n; row += ctas * (TT / 32)) {
            // one warp per row; FP32: compensated sums of the inverse's float pairs, the lanes' pairs
            // added in a fixed tree
            T sum;
            if constexpr (std::is_same<T, double>::value) {
                const double* inv = a.ainv + (int64_t)row * n;
                sum = 0.0;
#pragma unroll 4
                for (int c = lane; c < n; c += 32) sum = fma(__ldg(inv + c), bc[c], sum);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
            } else {
                const float* hi = a.ainv_hi + (int64_t)row * n;
                const float* lo = a.ainv_lo + (int64_t)row * n;
                Acc2 acc;
#pragma unroll 4
                for (int c = lane; c < n; c += 32) {
                    const float h = __ldg(hi + c), q = __ldg(lo + c), b = bc[c];
                    acc.add_prod(h, b);
                    acc.add_prod(q, b);
                }
                float s = acc.s, e = acc.c;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float s2 = __shfl_down_sync(0xffffffffu, s, o), e2 = __shfl_down_sync(0xffffffffu, e, o);
                    float v, f;
                    two_sum(s, s2, v, f);
                    s = v;
                    e += e2 + f;
                }
                sum = s + e;
            }
            if (lane == 0) xc[row] = (__ldg(a.lev[last].nmask + row / 3) >> (row % 3)) & 1 ? sum : T(0);
        }
        cluster_sync();
    }

    for (int l = last - 1; l >= 0; --l) {  // up: add the correction, smooth
        const int deg = a.lev[l].degree;
        t.enter(l);
        const T* xc = t.vec(a.lev[l + 1].x, l + 1);
#pragma unroll
        for (int r = 0; r < NPT; ++r) {
            TailNode<T>& n = t.nd[r];
            if (n.pn < 0) continue;
            // the values this thread left on the way down
            const T* b = l == 0 ? t.vec(a.b0, 0) + 3 * n.gn : t.vec(a.lev[l].b, l) + 3 * n.pn;
            const T* x = t.vec(a.lev[l].xt, l) + 3 * n.pn;
            T p[3];
            prolong_at(a.lev[l + 1].g.p, xc, n.i, n.j, n.k, p);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                n.b[c] = (n.m >> c) & 1 ? b[c] : T(0);
                n.x[c] = x[c] + ((n.m >> c) & 1 ? p[c] : T(0));
            }
        }
        t.exchange(l);
        for (int k = 0; k < deg; ++k) t.step(l, k == 0 ? T(0) : cf[l][2 * k], cf[l][2 * k + 1]);
        if (TailCfg<T>::EARLY) t.wait_halo();  // (nothing reads the last halo planes, but their stores have to be in)
        if (t.lost || (rank == 0 && tid >= a.lose_from)) cta_lost = 1;
        __syncthreads();
        const bool lost = cta_lost != 0;  // a lost halo fails the solve, whichever thread waited for it
        T* xo = t.vec(a.lev[l].x, l);
#pragma unroll
        for (int r = 0; r < NPT; ++r) {
            const TailNode<T>& n = t.nd[r];
            if (n.pn < 0) continue;
#pragma unroll
            for (int c = 0; c < 3; ++c) xo[3 * (l == 0 ? n.gn : n.pn) + c] = lost ? T(NAN) : n.x[c];
        }
        cluster_sync();  // the correction is written; at the end no CTA leaves before its neighbours' stores
    }
    if (t.lost) __nanosleep(1000000);  // ... which it has not seen arrive if a wait ran out
}

int tail_axis(const Dims& d) { return d.nx >= d.ny && d.nx >= d.nz ? 0 : d.ny >= d.nz ? 1 : 2; }

// fills the levels' geometry and the layout; false where they exceed a cluster
template <class T>
bool tail_plan(TailLevel<T>* lev, int nlev, int ctas, int axis, TailLayout* lay) {
    for (int l = 0; l < nlev; ++l) {
        TailGeo& g = lev[l].g;
        if (lev[l].d.nn() > 0xffff) return false;
        if (l == nlev - 1) {  // the coarsest grid: natural order
            g.p[0] = 1;
            g.p[1] = lev[l].d.nx + 1;
            g.p[2] = g.p[1] * (lev[l].d.ny + 1);
            continue;
        }
        g = slab_geo(axis, lev[l].d, ctas, TailCfg<T>::ALONE);
        if (lev[l].degree < 1 || lev[l].degree > kTailMaxDegree) return false;
        if (max_elems(g) > TailCfg<T>::MOST) return false;
        if (max_nodes(g) > TailCfg<T>::TT * TailCfg<T>::NPT || max_padded(g) > 0x7fff || max_nodes(g) + 2 * g.planeN > 0xffff) return false;
    }
    *lay = tail_layout<T>(lev, nlev);
    return sizeof(T) * (size_t)lay->words <= (size_t)kTailMaxSmem;
}

cudaLaunchConfig_t tail_config(int ctas, int threads, int nrhs, size_t bytes, cudaStream_t s, cudaLaunchAttribute* attr) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)ctas;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(ctas * nrhs));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <class T, int AXIS>
int tail_prepare_axis() {
    ANL_CUDA(cudaFuncSetAttribute(k_vtail<T, AXIS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailMaxSmem));
    ANL_CUDA(cudaFuncSetAttribute(k_vtail<T, AXIS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    return ANL_OK;
}

}  // namespace

// CTAs of the tail's cluster: 16 where the device can place such a cluster with the largest
// shared memory, else 8 (the portable size).
template <class T>
int vtail_prepare(int* ctas) {
    static int n = 0;
    if (n == 0) {
        ANL_TRY((tail_prepare_axis<T, 0>()));
        ANL_TRY((tail_prepare_axis<T, 1>()));
        ANL_TRY((tail_prepare_axis<T, 2>()));
        cudaLaunchAttribute attr;
        cudaLaunchConfig_t cfg = tail_config(16, TailCfg<T>::TT, 1, kTailMaxSmem, nullptr, &attr);
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, k_vtail<T, 0>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            fit = 0;
        }
        n = fit >= 1 ? 16 : 8;
    }
    *ctas = n;
    return ANL_OK;
}

template <class T>
bool vtail_fits(TailLevel<T>* lev, int nlev, int ctas) {
    TailLayout lay;
    return tail_plan<T>(lev, nlev, ctas, tail_axis(lev[0].d), &lay);
}

template <class T>
int launch_vtail(const TailArgs<T>& args, cudaStream_t s) {
    TailArgs<T> a = args;
    const int axis = tail_axis(a.lev[0].d);
    if (a.nlev < 2 || a.nlev > kTailMaxLevels || !tail_plan<T>(a.lev, a.nlev, a.ctas, axis, &a.lay)) {
        set_error("V-cycle tail: the levels exceed one cluster of %d CTAs", a.ctas);
        return ANL_ERR_BADARG;
    }
    const size_t bytes = sizeof(T) * (size_t)a.lay.words;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = tail_config(a.ctas, TailCfg<T>::TT, std::max(1, a.nrhs), bytes, s, &attr);
    switch (axis) {
        case 0: ANL_CUDA(cudaLaunchKernelEx(&cfg, k_vtail<T, 0>, a)); break;
        case 1: ANL_CUDA(cudaLaunchKernelEx(&cfg, k_vtail<T, 1>, a)); break;
        default: ANL_CUDA(cudaLaunchKernelEx(&cfg, k_vtail<T, 2>, a)); break;
    }
    ANL_LAUNCH_CHECK();
    return ANL_OK;
}

template int vtail_prepare<float>(int*);
template int vtail_prepare<double>(int*);
template bool vtail_fits<float>(TailLevel<float>*, int, int);
template bool vtail_fits<double>(TailLevel<double>*, int, int);
template int launch_vtail<float>(const TailArgs<float>&, cudaStream_t);
template int launch_vtail<double>(const TailArgs<double>&, cudaStream_t);

ANL_DEBUG_UNIT(vtail)

}  // namespace anl
