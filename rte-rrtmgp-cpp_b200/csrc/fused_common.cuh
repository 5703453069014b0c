// Building blocks shared by the fused FP32 column-forward kernels (longwave and shortwave).
//
// Mapping (both kernels): one CTA per column; lane l of every warp handles g-point
// 32*group + l; warp w owns the layer chunk [w*CL, (w+1)*CL) counted from the top of the
// atmosphere.  Per group of 32 g-points each warp first writes one record per (layer, band)
// of its chunk to shared memory (table offsets and interpolation weights of
// interpolation_kernel, minor scalings, band Planck values, cloud properties); the per
// (layer, g-point) work then reads its record with 128-bit shared loads and the tables with
// 128-bit corner-packed global loads (KdistView::kmaj4 & co.).
#pragma once

#include <cooperative_groups.h>

#include <algorithm>
#include <array>
#include <cfloat>
#include <cmath>
#include <map>
#include <mutex>

#include "common.cuh"
#include "rte_device.cuh"

namespace rrtmgp_b200 {
namespace fused {

// Per-layer state kept in shared memory for the whole kernel (layers counted from the top).
struct __align__(16) LayerState {
    int jt, jp, itropo, pad;
    float ftemp, fpress, p, t;
    float t_top, t_bot, dp, pad2;
};

// Per (layer, band) records.  Their sizes are odd numbers of 16-byte units, so that the 128-bit
// stores of 32 lanes building consecutive records spread over all 32 banks.
//
// Longwave: only what the weights cannot be formed from (the major and the Planck weights are
// products of fm, fpress and col_mix, a dozen multiplies per lane of a kernel whose FMA pipe is a
// quarter used), because shared memory held by records is taken from the L1 that holds the table
// rows.  With the aligned minor rows: 8192 x 128 3.05 -> 2.96 ms, dense tables 2000 x 60 728 -> 631 us;
// but grids that leave an SM with 7 to 10 warps of 16 layers are 1 - 2.5% slower (1000 x 104 359 -> 363 us,
// 600 x 104 261 -> 268, 1000 x 160 620 -> 625).
struct __align__(16) LwRec {
    int4 kb;          // x, y: element offsets (row * ngpt) of the kmp8 rows of (t0, p0, e0) and
                      //       (t1, p0, e1); z, w: kmin4 rows of (a, t0, e0), (a, t1, e1), unit 0
    float4 fm;        // fminor (minor weights)
    float4 mix;       // col_mix at the two temperatures, fpress, surface Planck function (bottom layer only)
    float4 aux;       // pl_lay, pl_top, pl_bot, tau_cloud
    int4 pad;
};
static_assert(sizeof(LwRec) == 80, "LwRec stride");

// Shortwave: the kernel is bound by instruction issue, so the weights are stored as they are used.
struct __align__(16) SwRec {
    int4 kb;               // as LwRec, on the kmaj4 rows
    float4 wmaj0, wmaj1;   // col_mix x fmajor (major absorption weights)
    float4 fm;             // fminor (minor and Rayleigh weights)
    float4 aux;            // col_dry + col_h2o (Rayleigh), cloud tau, tau*ssa, tau*ssa*g
    float aux2;            // cloud absorption optical depth tau_c * (1 - ssa_c)
    int pad[7];
};
static_assert(sizeof(SwRec) == 112, "SwRec stride");

// Reduce-scatter of N per-lane values over 32 lanes: afterwards lane L holds in v[0] the warp
// total of value L >> log2(32 / N) (N <= 32, a power of two).
template <int N, int OFF>
struct ReduceScatter {
    static __device__ __forceinline__ void run(float* v, int lane)
    {
        constexpr int H = N / 2;
        const bool upper = (lane & OFF) != 0;
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const float send = upper ? v[i] : v[i + H];
            const float keep = upper ? v[i + H] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, OFF);
        }
        ReduceScatter<H, OFF / 2>::run(v, lane);
    }
};
template <int OFF>
struct ReduceScatter<1, OFF> {
    static __device__ __forceinline__ void run(float* v, int lane)
    {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], OFF);
        ReduceScatter<1, OFF / 2>::run(v, lane);
    }
};
template <>
struct ReduceScatter<1, 0> {
    static __device__ __forceinline__ void run(float*, int) {}
};

__device__ __forceinline__ float warp_sum(float x)
{
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    return x;
}

// Interpolation of band b at layer state s (interpolation_kernel,
// gas_optics_rrtmgp_kernels.cu:256-291): its weights, and the table rows of a record.  The minor
// scalings are per layer, not per record (layer_minor_scalings).
__device__ __forceinline__ FlavorWeights<float> record_rows(const KdistView<float>& k, int4& kb, const LayerState& s,
                                                            const float* cg, int cgs, int b)
{
    LayerInterp<float> li;
    li.jt = s.jt;
    li.jp = s.jp;
    li.itropo = s.itropo;
    li.ftemp = s.ftemp;
    li.fpress = s.fpress;
    const int a = li.itropo;
    const FlavorWeights<float> fw = flavor_weights(k, k.band_flav[2 * b + a], li, cg, cgs);
    const int ne1 = k.neta - 1, np = k.npres;
    const int p0 = li.jp + a - 1;
    const int mrow = k.nminor_units * k.ngpt;
    kb = make_int4((((li.jt - 1) * np + p0) * ne1 + (fw.j0 - 1)) * k.ngpt,
                   ((li.jt * np + p0) * ne1 + (fw.j1 - 1)) * k.ngpt,
                   ((a * k.ntemp + li.jt - 1) * ne1 + (fw.j0 - 1)) * mrow,
                   ((a * k.ntemp + li.jt) * ne1 + (fw.j1 - 1)) * mrow);
    return fw;
}

__device__ __forceinline__ void record_weights(const KdistView<float>& k, LwRec& R, const LayerState& s,
                                               const float* cg, int cgs, int b, float planck_sfc)
{
    const FlavorWeights<float> fw = record_rows(k, R.kb, s, cg, cgs, b);
    R.fm = make_float4(fw.fm[0], fw.fm[1], fw.fm[2], fw.fm[3]);
    R.mix = make_float4(fw.cm[0], fw.cm[1], s.fpress, planck_sfc);
}

__device__ __forceinline__ void record_weights(const KdistView<float>& k, SwRec& R, const LayerState& s,
                                               const float* cg, int cgs, int b)
{
    const FlavorWeights<float> fw = record_rows(k, R.kb, s, cg, cgs, b);
    R.fm = make_float4(fw.fm[0], fw.fm[1], fw.fm[2], fw.fm[3]);
    const float fp = s.fpress, f1 = 1.f - s.fpress;
    R.wmaj0 = make_float4(fw.cm[0] * (f1 * fw.fm[0]), fw.cm[0] * (f1 * fw.fm[1]), fw.cm[0] * (fp * fw.fm[0]),
                          fw.cm[0] * (fp * fw.fm[1]));
    R.wmaj1 = make_float4(fw.cm[1] * (f1 * fw.fm[2]), fw.cm[1] * (f1 * fw.fm[3]), fw.cm[1] * (fp * fw.fm[2]),
                          fw.cm[1] * (fp * fw.fm[3]));
}

// Minor scaling of scaling kind sid of atmosphere a at a layer (minor_scaling: the same
// arithmetic, gas_optical_depths_minor_kernel :396-417).
__device__ __forceinline__ float kind_scaling(const KdistView<float>& k, int a, int sid, const float* cg, int cgs,
                                              float p, float t)
{
    const int flags = k.scal_flags[a][sid];
    float scaling = cg[k.scal_gas[a][sid] * cgs];
    if (flags & 1) {
        scaling *= 0.01f * p / t;
        const int sg = k.scal_sgas[a][sid];
        if (sg > 0) {
            const float vmr_fact = 1.f / cg[0];
            const float dry_fact = 1.f / (1.f + cg[k.idx_h2o * cgs] * vmr_fact);
            if (flags & 2) scaling *= (1.f - cg[sg * cgs] * vmr_fact * dry_fact);
            else scaling *= cg[sg * cgs] * vmr_fact * dry_fact;
        }
    }
    return scaling;
}

// Scalings of every kind of layers 0 .. nloc - 1 (layer state st[], gas columns cg with
// stride cgs) into sc[jl * k.max_nscal + sid]; threads tid, tid + nthr, ... of the calling
// team take one (layer, kind) each.  Kinds past the layer's atmosphere's count are set to 0.
__device__ __forceinline__ void layer_minor_scalings(const KdistView<float>& k, const LayerState* st, const float* cg,
                                                     int cgs, float* sc, int nloc, int tid, int nthr)
{
    const int ns = k.max_nscal;
    for (int idx = tid; idx < nloc * ns; idx += nthr) {
        const int jl = idx / ns, sid = idx - jl * ns;
        const LayerState& s = st[jl];
        sc[idx] = sid < k.nscal[s.itropo] ? kind_scaling(k, s.itropo, sid, cg + jl, cgs, s.p, s.t) : 0.f;
    }
}

// One 256-bit load of a table row entry (sm_100; p is 32-byte aligned: Tab8).
__device__ __forceinline__ Tab8 ldg8(const Tab8* p)
{
    Tab8 r;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y), "=f"(r.b.z), "=f"(r.b.w)
        : "l"(p));
    return r;
}

// 128-bit load when on, else zeros: one predicated load instead of a branch around it, so that the
// loads of several unrolled layers can be in flight together.  (Without the zeros the
// registers of an unrolled loop's loads are live from its start: 2 KB of spills.)
__device__ __forceinline__ float4 ldg4_if(const float4* p, bool on)
{
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "+f"(r.x), "+f"(r.y), "+f"(r.z), "+f"(r.w)
        : "l"(p), "r"(int(on)));
    return r;
}

__device__ __forceinline__ float dot4(const float4& a, const float4& b)
{
    return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w;
}

// Sum over (eta, p) of one temperature's corners: f0, f1 the fminor weights of the two etas.
__device__ __forceinline__ float corner_sum(float f0, float f1, float fp, const float4& c)
{
    return (1.f - fp) * (f0 * c.x + f1 * c.y) + fp * (f0 * c.z + f1 * c.w);
}

// The minor intervals of a lane's g-point in one atmosphere: the scaling kinds of the pairs of units
// 0 and 1 (a byte each; 0 past the last interval) and the most intervals over the warp's lanes.
struct MinorRef {
    int sid0, sid1, nmax;
};

// The gas tables of one domain, by value for out-of-line callers.
struct GasTab {
    const float4* kmaj4;   // shortwave
    const Tab8* kmp8;      // longwave
    const float4* kmin4;
    const int2* minor_s;
    int ngpt, nunits;
};
__device__ __forceinline__ GasTab gas_tab(const KdistView<float>& k)
{
    return GasTab{k.kmaj4, k.kmp8, k.kmin4, k.minor_s, k.ngpt, k.nminor_units};
}

__device__ __forceinline__ MinorRef minor_ref(const KdistView<float>& k, int a, int g, bool valid)
{
    const int2* const m = k.minor_s + size_t(a) * k.nminor_units * k.ngpt + g;
    const int2 e = valid ? __ldg(m) : make_int2(0, 0);
    return MinorRef{e.x, valid && k.nminor_units > 1 ? __ldg(m + k.ngpt).x : 0, __reduce_max_sync(0xffffffffu, e.y)};
}

// The table values of one (layer, g-point): the two major corner rows, the longwave's
// Planck-fraction rows, the minor rows of units 0 and 1 (shortwave: pair 0 of unit 0 is the
// Rayleigh coefficient), zeros where no lane of the warp needs them.  Loaded together, before any
// of them is used.
struct GasRows {
    float4 c0, c1;   // kmajor corners
    float4 p0, p1;   // LW: Planck fraction corners
    float4 m0, m1;   // minor rows, unit 0
    float4 n0, n1;   // minor rows, unit 1
};
template <bool SW>
__device__ __forceinline__ void load_rows(const GasTab& k, const int4& kb, int g, int nmax, GasRows& r)
{
    if constexpr (SW) {
        r.c0 = __ldg(k.kmaj4 + (kb.x + g));
        r.c1 = __ldg(k.kmaj4 + (kb.y + g));
        r.m0 = __ldg(k.kmin4 + (kb.z + g));
        r.m1 = __ldg(k.kmin4 + (kb.w + g));
    } else {
        const Tab8 t0 = ldg8(k.kmp8 + (kb.x + g)), t1 = ldg8(k.kmp8 + (kb.y + g));
        r.c0 = t0.a; r.p0 = t0.b;
        r.c1 = t1.a; r.p1 = t1.b;
        r.m0 = ldg4_if(k.kmin4 + (kb.z + g), nmax > 0);
        r.m1 = ldg4_if(k.kmin4 + (kb.w + g), nmax > 0);
    }
    if constexpr (SW) {   // one interval in unit 0
        r.n0 = ldg4_if(k.kmin4 + (kb.z + k.ngpt + g), nmax > 1);
        r.n1 = ldg4_if(k.kmin4 + (kb.w + k.ngpt + g), nmax > 1);
    } else {
        // Two in unit 0.  A branch, taken by few warps: with predicated loads the longwave forward was 2 - 4%
        // slower (300 x 104 180 us, 173 now; 1000 x 112 389, 380; 147 x 160 96.5, 94.7; 8192 x 128 2.94 ms,
        // 2.89).  Unit 0, which most warps read, is better predicated (1000 x 128 400 us, 426 with a branch).
        r.n0 = r.n1 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (nmax > 2) {
            r.n0 = __ldg(k.kmin4 + (kb.z + k.ngpt + g));
            r.n1 = __ldg(k.kmin4 + (kb.w + k.ngpt + g));
        }
    }
}

// The (T, eta) corners in fminor order of the first and the second pair of two rows.
__device__ __forceinline__ float4 pair0(const float4& x, const float4& y) { return make_float4(x.x, x.y, y.x, y.y); }
__device__ __forceinline__ float4 pair1(const float4& x, const float4& y) { return make_float4(x.z, x.w, y.z, y.w); }
__device__ __forceinline__ float4 rayleigh_corners(const GasRows& r) { return pair0(r.m0, r.m1); }

// Visits the minor intervals of g-point g: f(corners in fminor order, scaling kind), in their file
// order.  Lanes with fewer intervals than m.nmax (warp-uniform bound) take zero coefficients and
// kind 0, so nothing diverges and no select is needed.  Units 0 and 1 come from r (load_rows).
// DENSE: more than three intervals over some g-point (KdistView::max_minor_per_g > 3); the loop over
// the further units is compiled only then.
template <bool SW, bool DENSE, class F>
__device__ __forceinline__ void for_minors(const GasTab& k, const int4& kb, int a, int g, const GasRows& r,
                                           const MinorRef& m, F&& f)
{
    constexpr int R = SW ? 1 : 0;
    if constexpr (!SW)
        if (m.nmax > 0) f(pair0(r.m0, r.m1), m.sid0 & 255);
    if (m.nmax > 1 - R) f(pair1(r.m0, r.m1), m.sid0 >> 8);
    if (m.nmax > 2 - R) f(pair0(r.n0, r.n1), m.sid1 & 255);
    if (m.nmax > 3 - R) f(pair1(r.n0, r.n1), m.sid1 >> 8);
    if constexpr (DENSE) {
        for (int u = 2; 2 * u - R < m.nmax; ++u) {
            const int w = __ldg(&k.minor_s[(size_t(a) * k.nunits + u) * k.ngpt + g].x);
            const float4 x0 = __ldg(k.kmin4 + (kb.z + u * k.ngpt + g));
            const float4 x1 = __ldg(k.kmin4 + (kb.w + u * k.ngpt + g));
            f(pair0(x0, x1), w & 255);
            f(pair1(x0, x1), w >> 8);
        }
    }
}

// Absorption optical depth of g-point g from a record: major (8 corners) plus the minor
// intervals covering g, as gas_optical_depths_major/minor.  r: load_rows of the record; the rest as
// for_minors.  sc: the layer's scalings, kind sid at sc[sid * sst].
__device__ __forceinline__ float major_tau(const LwRec& R, const GasRows& r)
{
    return R.mix.x * corner_sum(R.fm.x, R.fm.y, R.mix.z, r.c0) + R.mix.y * corner_sum(R.fm.z, R.fm.w, R.mix.z, r.c1);
}
__device__ __forceinline__ float major_tau(const SwRec& R, const GasRows& r)
{
    return dot4(R.wmaj0, r.c0) + dot4(R.wmaj1, r.c1);
}
template <bool SW, bool DENSE, class Rec>
__device__ __forceinline__ float tau_abs(const GasTab& k, const Rec& R, int a, int g, const GasRows& r,
                                         const MinorRef& m, const float* sc, int sst = 1)
{
    float tau = major_tau(R, r);
    for_minors<SW, DENSE>(k, R.kb, a, g, r, m,
                          [&](const float4& c, int sid) { tau += sc[sid * sst] * dot4(R.fm, c); });
    return tau;
}

// Planck fraction (Planck_source_kernel, gas_optics_rrtmgp_kernels.cu:181-190).
__device__ __forceinline__ float planck_fraction(const LwRec& R, const GasRows& r)
{
    return corner_sum(R.fm.x, R.fm.y, R.mix.z, r.p0) + corner_sum(R.fm.z, R.fm.w, R.mix.z, r.p1);
}

// Context of a fused column computation.  Members: icol(); warp() = the chunk this warp owns
// and nwarps() = the chunks of the column; lwarp() = the warp within the CTA (or team) that
// holds its shared memory; tid() / nthreads() of that CTA (team); smem(); sync() = the barrier
// of every warp of the column; layer0() / nloc(nlay) = the layers whose state that shared
// memory holds; put(p, v) stores v at p in the shared memory of every CTA that reads it.
// CtaCtx: the whole CTA computes column blockIdx.x; every value is a special register or a
// launch constant, so none occupies a register across the column.  The batched kernel
// supplies its own context type with the same members.
struct CtaCtx {
    __device__ __forceinline__ int icol() const { return blockIdx.x; }
    __device__ __forceinline__ int warp() const { return threadIdx.x >> 5; }
    __device__ __forceinline__ int nwarps() const { return blockDim.x >> 5; }
    __device__ __forceinline__ int lwarp() const { return threadIdx.x >> 5; }
    __device__ __forceinline__ int tid() const { return threadIdx.x; }
    __device__ __forceinline__ int nthreads() const { return blockDim.x; }
    __device__ __forceinline__ int layer0() const { return 0; }
    __device__ __forceinline__ int nloc(int nlay) const { return nlay; }
    __device__ __forceinline__ unsigned char* smem() const
    {
        extern __shared__ __align__(16) unsigned char smem_raw[];
        return smem_raw;
    }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    template <class T>
    __device__ __forceinline__ void put(T* p, const T& v) const { *p = v; }
    __device__ __forceinline__ int group0(int) const { return 0; }
    __device__ __forceinline__ int group1(int ngroups) const { return ngroups; }
    template <class... A>
    __device__ __forceinline__ bool combine(A&...) const { return true; }
};

// One column on a thread-block cluster of cs CTAs (columns deeper than one CTA holds): CTA r
// of the cluster owns the chunks [r W, (r + 1) W) (W = its warps) and the state of their
// layers [r W CL, (r + 1) W CL); the chunk quantities every warp reads are stored into the
// shared memory of all CTAs of the cluster (distributed shared memory) and the barrier is the
// cluster's.
template <int CL>
struct ClusterCtx {
    int cs;
    __device__ __forceinline__ int rank() const { return int(cooperative_groups::this_cluster().block_rank()); }
    __device__ __forceinline__ int icol() const { return blockIdx.x / cs; }
    __device__ __forceinline__ int warp() const { return rank() * int(blockDim.x >> 5) + int(threadIdx.x >> 5); }
    __device__ __forceinline__ int nwarps() const { return cs * int(blockDim.x >> 5); }
    __device__ __forceinline__ int lwarp() const { return threadIdx.x >> 5; }
    __device__ __forceinline__ int tid() const { return threadIdx.x; }
    __device__ __forceinline__ int nthreads() const { return blockDim.x; }
    __device__ __forceinline__ int layer0() const { return rank() * int(blockDim.x >> 5) * CL; }
    __device__ __forceinline__ int nloc(int nlay) const
    {
        return max(0, min(int(blockDim.x >> 5) * CL, nlay - layer0()));
    }
    __device__ __forceinline__ unsigned char* smem() const
    {
        extern __shared__ __align__(16) unsigned char smem_raw[];
        return smem_raw;
    }
    __device__ __forceinline__ void sync() const { cooperative_groups::this_cluster().sync(); }
    template <class T>
    __device__ __forceinline__ void put(T* p, const T& v) const
    {
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        for (int r = 0; r < cs; ++r) *cl.map_shared_rank(p, r) = v;
    }
    __device__ __forceinline__ int group0(int) const { return 0; }
    __device__ __forceinline__ int group1(int ngroups) const { return ngroups; }
    template <class... A>
    __device__ __forceinline__ bool combine(A&...) const { return true; }
};

// One column on a thread-block cluster of `parts` CTAs that share its g-points (grids of too few
// columns to fill the chip): every CTA holds all layers and computes the groups [rank G / parts,
// (rank + 1) G / parts); the FP64 accumulators are then added in rank order by CTA 0 through
// distributed shared memory (xch: the byte offset of nthreads doubles per accumulator behind the
// column's shared memory).
struct SplitCtx : CtaCtx {
    int parts, xch;
    __device__ __forceinline__ SplitCtx(int p, int x) : parts(p), xch(x) {}
    __device__ __forceinline__ int rank() const { return int(cooperative_groups::this_cluster().block_rank()); }
    __device__ __forceinline__ int icol() const { return blockIdx.x / parts; }
    __device__ __forceinline__ int group0(int ngroups) const { return rank() * ngroups / parts; }
    __device__ __forceinline__ int group1(int ngroups) const { return (rank() + 1) * ngroups / parts; }
    template <class... A>
    __device__ __forceinline__ bool combine(A&... a) const
    {
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        double* const own = reinterpret_cast<double*>(smem() + xch) + tid();
        const int r = rank();
        int i = 0;
        if (r > 0) ((own[nthreads() * i++] = a), ...);
        cl.sync();
        if (r == 0)
            for (int p = 1; p < parts; ++p) {
                const double* const other = cl.map_shared_rank(own, p);
                i = 0;
                ((a += other[nthreads() * i++]), ...);
            }
        cl.sync();   // no CTA leaves while its shared memory may still be read
        return r == 0;
    }
};

// Whether per_sm CTAs of smem bytes of dynamic shared memory fit in `bytes` of an SM (each takes 1 KB
// more than it asks for).
inline bool ctas_fit(int per_sm, size_t smem, size_t bytes = 228 * 1024) { return per_sm * (smem + 1024) <= bytes; }

// CTAs (cluster = 1) or clusters of a kernel that the device holds at once, by the driver; 0 when it has
// no answer.  Clusters do not cross the chip's GPCs: of 444 places for CTAs only 432 or so take clusters
// of three, and a grid of 441 such CTAs needs a second wave (147 x 40 shortwave: 65 us, 42 in
// clusters of two).
template <class K>
int resident(K kernel, int nsm, int threads, size_t smem, int cluster)
{
    int n = 0;
    cudaError_t e;
    if (cluster == 1) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem);
        n *= nsm;
    } else {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cluster);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = unsigned(cluster);
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
    }
    if (e == cudaSuccess) return n;
    cudaGetLastError();
    return 0;
}

// Columns that the device holds at once when s = 1 .. 8 CTAs share the groups of each ([s]; [0] unused).
using AtOnce = std::array<int, 9>;

// The AtOnce of a launch shape (kernel, device, threads, shared memory), asked from the driver once: eight
// questions take longer than a small grid's launch.
class ResidencyTable {
public:
    template <class K, class F>
    AtOnce operator()(K kernel, int device, int threads, size_t smem, F&& ask)
    {
        const std::array<size_t, 4> key{reinterpret_cast<size_t>(kernel), size_t(device), size_t(threads), smem};
        std::lock_guard<std::mutex> lock(mu_);
        const auto it = known_.find(key);
        if (it != known_.end()) return it->second;
        AtOnce a{};
        for (int s = 1; s <= 8; ++s) a[s] = ask(s);
        if (known_.size() >= 1024) known_.clear();   // launch shapes of many handles
        known_[key] = a;
        return a;
    }

private:
    std::mutex mu_;
    std::map<std::array<size_t, 4>, AtOnce> known_;
};
inline ResidencyTable& residency()
{
    static ResidencyTable r;
    return r;
}

// CTAs per column for a grid of ncol columns of G groups, at[s] columns at once (0: not possible; s = 1 in
// the instance that an unsplit grid runs).  A CTA costs its groups and kGroupSetup more for its set-up (layer state,
// scalings, cloud optics, launch); waves of CTAs run one after the other.  The split with the
// least waves x cost is taken when it saves more than a tenth.
constexpr float kGroupSetup = 2.0f;   // measured 1.4 (LW) to 3 (SW) groups at 60 layers
inline int group_parts(int ncol, int G, const AtOnce& at)
{
    if (at[1] < 1) return 1;
    auto cost = [&](int s) {
        return float((ncol + at[s] - 1) / at[s]) * (kGroupSetup + float((G + s - 1) / s));
    };
    float least = 0.9f * cost(1);
    int best = 1;
    for (int s = 2; s <= std::min(G, 8); ++s) {
        if (at[s] < 1 || cost(s) >= least) continue;
        least = cost(s);
        best = s;
    }
    return best;
}

// Fill the per-layer state and col_gas of layers j0 .. j0 + nloc - 1 (counted from the top,
// those below nlay) of column icol into st[j - j0] and cg[(gas) * cg_stride + j - j0]; threads
// tid, tid + nthr, ... of the calling team take one layer each.
__device__ __forceinline__ void setup_layer_range(const KdistView<float>& k, const GasSet<float>& gs, int ncol,
                                                  int nlay, int icol, bool top_at_1, const float* __restrict__ play,
                                                  const float* __restrict__ plev, const float* __restrict__ tlay,
                                                  const float* __restrict__ tlev, const float* __restrict__ col_dry,
                                                  LayerState* st, float* cg, int cg_stride, int j0, int nloc,
                                                  int tid, int nthr)
{
    for (int jl = tid; jl < nloc; jl += nthr) {
        const int j = j0 + jl;
        if (j >= nlay) break;
        const int l = top_at_1 ? j : nlay - 1 - j;
        const size_t cl = icol + size_t(l) * ncol;
        const float p = play[cl], t = tlay[cl];
        fill_col_gas(k, gs, ncol, nlay, icol, l, plev, col_dry, cg + jl, cg_stride);
        const LayerInterp<float> li = layer_interp(k, p, t);
        const int lt = top_at_1 ? j : nlay - j, lb = top_at_1 ? j + 1 : nlay - 1 - j;
        LayerState s;
        s.jt = li.jt;
        s.jp = li.jp;
        s.itropo = li.itropo;
        s.pad = 0;
        s.ftemp = li.ftemp;
        s.fpress = li.fpress;
        s.p = p;
        s.t = t;
        s.t_top = tlev ? tlev[icol + size_t(lt) * ncol] : 0.f;
        s.t_bot = tlev ? tlev[icol + size_t(lb) * ncol] : 0.f;
        s.dp = fabsf(plev[icol + size_t(lb) * ncol] - plev[icol + size_t(lt) * ncol]);
        s.pad2 = 0.f;
        st[jl] = s;
    }
}

// Table layouts the corner-packed FP32 kernels take: minor intervals inside one band (their
// interpolation weights are the band's), at most kMaxScal scaling kinds per atmosphere, and
// a group of 32 g-points touching at most max_bands bands.  Any number of minor intervals per
// band or per g-point is accepted.
inline bool fused_layout_ok(const KdistView<float>& v, bool sw, int max_bands)
{
    return v.minor_in_band && v.nscal[0] <= kMaxScal && v.nscal[1] <= kMaxScal &&
           v.max_group_bands <= max_bands && v.is_lw == !sw;
}

// Shared-memory offsets (bytes) of the fused kernels, all 16-byte aligned.
struct SmemLayout {
    size_t state, cg, scal, cloud, maps, sfc, recs, total;
};

__host__ __device__ __forceinline__ size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// nlay: layers whose state the CTA holds; NW: chunks of the column (maps); NWloc: warps of
// the CTA (records of rec_bytes each).
__host__ __device__ __forceinline__ SmemLayout smem_layout(int nlay, int ngas, int nband, int ncloud_vals, int NW,
                                                           int nmaps, int CL, int nbands_per_group, int nscal,
                                                           size_t rec_bytes, int NWloc = -1)
{
    if (NWloc < 0) NWloc = NW;
    SmemLayout L;
    L.state = 0;
    L.cg = align16(L.state + sizeof(LayerState) * size_t(nlay));
    L.scal = align16(L.cg + sizeof(float) * size_t(ngas + 1) * nlay);
    L.cloud = align16(L.scal + sizeof(float) * size_t(nscal) * nlay);
    L.maps = align16(L.cloud + sizeof(float) * size_t(ncloud_vals) * nband * nlay);
    L.sfc = align16(L.maps + sizeof(float4) * size_t(NW) * 32 * nmaps);
    L.recs = align16(L.sfc + sizeof(float) * 64);
    L.total = align16(L.recs + rec_bytes * size_t(NWloc) * CL * nbands_per_group);
    return L;
}

}  // namespace fused
}  // namespace rrtmgp_b200
