// pagerank_split.cu -- PageRank with FP32 values and compensated gather sums,
// FP64 diagnostics (no counterpart in the reference; its PageRank is FP64
// throughout).
//
// Formula and superstep structure follow benchmarks/pagerank.c:36-66,98-99
// run under the single-broadcast version (combiner_single_broadcast_
// postamble.h:57-89,185-201):
//   superstep 0:       x_v = 1/V
//   superstep s >= 1:  x_v = (1-d)/V + d * sum_{u in row(v), deg u > 0} x_u / deg u
//   a vertex broadcasts x_v / deg v while s < rounds and deg v > 0;
// rounds + 1 supersteps in all.  As in the reference's benchmarks (they load
// with directed = false, pagerank.c:91), the stored rows serve both as the
// gather lists and for the out-degrees; no dangling mass is redistributed.
//
// Precision split: the values x and the broadcast quotients are FP32 (4 bytes
// per vertex, so the gathered array of an R-MAT scale-24 graph, 64 MiB, stays
// in the 126 MB L2), and each gather sum is compensated: every lane keeps a
// (sum, compensation) pair updated with Knuth's TwoSum (the Kahan-Babuska
// refinement of Kahan summation due to Neumaier, 1974), and pairs of lanes,
// warps and hub chunks are merged with the same error-free transformation.
// The diagnostics of every superstep -- the mass sum x, the dangling mass (sum
// of x over vertices without out-edges) and the L1 residual sum |x - x_prev| --
// are reduced in FP64.
//
// One kernel per superstep gathers, updates and sums the diagnostics: the
// hubs' rows in chunks, a warp each (partial pairs to scratch, merged in chunk
// order by the warp whose chunk arrives last), then rows by length with 16, 8
// and 1 lanes each.  Everything is enqueued on one stream without host
// synchronisation or allocation, so a run can be captured into a CUDA graph.
#include "ipregel_b200.h"

#include <cuda_runtime.h>
#include <cub/cub.cuh>

#include <cstdlib>
#include <new>
#include <utility>
#include <vector>

extern "C" int ipg_internal_fail(int code, const char* msg);

#define PR_THREADS 256
#define PR_CHUNK 4096 /* most edges of a hub chunk, and so of a row that is no hub */
#define PR_MID 64     /* rows up to here take PR_GROUP lanes, longer ones PR_LONG */
#ifndef PR_GROUP
#define PR_GROUP 8
#endif
#ifndef PR_SHORT
#define PR_SHORT 1
#endif
#ifndef PR_LONG
#define PR_LONG 16
#endif
#ifndef PR_CTAS
#define PR_CTAS 4 /* resident CTAs per SM the gather is compiled for */
#endif
#define PR_CTAS_PER_SM 8 /* upper bound of the other kernels; the resident count decides */

#define PR_CUDA(call)                                                      \
    do {                                                                   \
        cudaError_t e_ = (call);                                           \
        if (e_ != cudaSuccess) return ipg_internal_fail(IPG_ECUDA, cudaGetErrorString(e_)); \
    } while (0)

#define PR_TRY(call)                       \
    do {                                   \
        int r_ = (call);                   \
        if (r_ != IPG_OK) return r_;       \
    } while (0)

struct ipg_pr_plan {
    ipg_graph* g = nullptr;
    ipg_graph_view gv{};
    ipg_bins bins{};
    float* b[2] = {nullptr, nullptr};  // broadcast quotients, by superstep parity
    float* xs = nullptr;               // values of every other superstep
    // on the graph's degree-ordered copy (ipg_graph_degree_order): the
    // supersteps write xs / xs2 in the copy's numbering, and a last gather
    // writes the values in the caller's (null: the graph's own numbering)
    const uint32_t* new_of_old = nullptr;
    float* xs2 = nullptr;
    ipg_hubs hubs{};                   // rows above hub_min in chunks
    ipg_hold* holds[2] = {nullptr, nullptr};  // of both
    uint64_t hub_min = 0, chunk = 0;
    bool quads = false;                // the gather lists take 128-bit loads
    float2* partial = nullptr;         // (sum, compensation) of every hub chunk
    uint32_t* arrived = nullptr;       // per hub the chunks arrived (0 between supersteps)
    uint32_t* shorts = nullptr;        // the short class: first the vertices with in-edges (null: unsplit)
    uint64_t empty = 0, empty_dangling = 0;  // the rest of it
    uint64_t class_count[3] = {0, 0, 0}, class_edges[3] = {0, 0, 0};
    int sms = 148;
    uint32_t grid = 0, grid_flat = 0;  // resident CTAs of the gather / of the others, all SMs
    std::vector<std::pair<void*, uint64_t>> allocs;
};

namespace {

// ---- compensated FP32 accumulation ----------------------------------------
// The value of a pair is s + c.  TwoSum gives the exact rounding error of
// s + x, which is carried in c.  __fadd_rn/__fsub_rn keep the compiler from
// contracting or reordering the error terms.
template <bool COMP>
__device__ __forceinline__ void pr_add(float& s, float& c, float x)
{
    if constexpr (COMP) {
        const float t = __fadd_rn(s, x);
        const float bp = __fsub_rn(t, s);
        const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(x, bp));
        c = __fadd_rn(c, err);
        s = t;
    } else {
        (void)c;
        s = __fadd_rn(s, x);
    }
}

template <bool COMP>
__device__ __forceinline__ void pr_merge(float& s, float& c, float s2, float c2)
{
    pr_add<COMP>(s, c, s2);
    if constexpr (COMP) c = __fadd_rn(c, c2);
}

template <bool COMP>
__device__ __forceinline__ void pr_warp_merge(float& s, float& c)
{
    for (int o = 16; o > 0; o >>= 1) {
        const float s2 = __shfl_down_sync(0xffffffffu, s, o);
        const float c2 = __shfl_down_sync(0xffffffffu, c, o);
        pr_merge<COMP>(s, c, s2, c2);
    }
}

struct PrStep {
    const uint64_t* __restrict__ row;     // out-rows: the degrees
    const uint64_t* __restrict__ in_row;  // gather lists (the rows themselves
    const uint32_t* __restrict__ in_adj;  // unless the graph is directed)
    // written by the superstep before, which may still run when this one's CTAs
    // come onto the SMs (k_pr_step): ordinary loads, no __restrict__
    const float* b_cur;   // read by the gathers
    float* b_next;        // written for the next superstep
    float* x_out;         // this superstep's values
    const float* x_prev;  // the last superstep's
    double* diag;         // this superstep's mass, dangling mass, residual
    float ratio, damping;
    const uint32_t* __restrict__ list[3];  // short, middle, long rows (hubs among the long)
    uint64_t n[3];
    const uint4* __restrict__ hub;         // {vertex, first chunk, chunks}
    const uint32_t* __restrict__ owner;    // chunk -> hub
    float2* partial;
    uint32_t* arrived;
    uint64_t chunks, chunk, hub_min;
    uint64_t empty, empty_dangling;  // vertices without in-edges; of those, without out-edges
    float x0;                        // superstep 0's value
    bool first;                      // superstep 1
    bool quads;  // 128-bit id loads: an aligned array of whole loads
};

// Sum of the vertex diagnostics over the CTA, added to diag[0..2].
__device__ __forceinline__ void pr_block_diag(double m, double d, double r, double* diag)
{
    __shared__ double sh[3][PR_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) {
        m += __shfl_down_sync(0xffffffffu, m, o);
        d += __shfl_down_sync(0xffffffffu, d, o);
        r += __shfl_down_sync(0xffffffffu, r, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        sh[0][warp] = m;
        sh[1][warp] = d;
        sh[2][warp] = r;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0, c = 0;
        for (int w = 0; w < PR_THREADS / 32; w++) {
            a += sh[0][w];
            b += sh[1][w];
            c += sh[2][w];
        }
        if (a != 0.0) atomicAdd(&diag[0], a);
        if (b != 0.0) atomicAdd(&diag[1], b);
        if (c != 0.0) atomicAdd(&diag[2], c);
    }
}

// Diagnostics of the vertices a thread updated.
struct PrDiag {
    double m = 0, d = 0, r = 0;
};

// Vertex update of pagerank.c:51-52 and the broadcast of :57-63; the values
// are double-buffered.  deg and x_prev were loaded before the gather, so the
// update waits for nothing (read after it, the old value more than doubled
// the superstep on R-MAT scale 24, and a pass of its own took 4 % of the run).
template <bool LAST>
__device__ __forceinline__ void pr_finish(const PrStep& a, uint64_t v, uint64_t deg, float x_prev, float sum, PrDiag& g)
{
    const float xn = __fadd_rn(a.ratio, __fmul_rn(a.damping, sum));
    a.x_out[v] = xn;
    if constexpr (!LAST) a.b_next[v] = deg ? __fdiv_rn(xn, (float)deg) : 0.0f;
    g.m += (double)xn;
    if (!deg) g.d += (double)xn;
    g.r += fabs((double)xn - (double)x_prev);
}

// The aligned four ids at position rel (a multiple of 4) from row start r0
// rounded down to one; which of them belong to the row of deg edges is
// decided when they are used, so that nothing waits for the load before.
__device__ __forceinline__ uint4 pr_ld_quad(const PrStep& a, uint64_t r0, uint32_t deg, uint32_t rel)
{
    const uint32_t off = (uint32_t)r0 & 3u;
    return __ldcs(reinterpret_cast<const uint4*>(a.in_adj + (rel < off + deg ? r0 - off + rel : 0)));
}

// Adds the quotients of the row's edges among them, in order.
template <bool COMP>
__device__ __forceinline__ void pr_add_quad(const PrStep& a, const uint4& q, uint64_t r0, uint32_t deg, uint32_t rel,
                                            float& s, float& c)
{
    const uint32_t t = rel - ((uint32_t)r0 & 3u);  // edge of the row; before its first: wraps
    const uint32_t id[4] = {q.x, q.y, q.z, q.w};
    float w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = t + k < deg ? a.b_cur[id[k]] : 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++) pr_add<COMP>(s, c, w[k]);  // 0 leaves the pair as it is
}

// Lane-strided sum over in_adj[e0, e1) for arrays without 128-bit loads.
template <bool COMP>
__device__ __forceinline__ void pr_gather(const PrStep& a, uint64_t e0, uint64_t e1, uint64_t lane, uint64_t lanes,
                                          float& s, float& c)
{
    for (uint64_t e = e0 + lane; e < e1; e += lanes) pr_add<COMP>(s, c, a.b_cur[a.in_adj[e]]);
}

// Out-degree of v whose gather list holds n ids.
__device__ __forceinline__ uint64_t pr_deg(const PrStep& a, uint64_t v, uint64_t n)
{
    return a.row == a.in_row ? n : a.row[v + 1] - a.row[v];
}

// Superstep 0: x = 1/V, broadcast x/deg, and its diagnostics {sum x, sum of x
// over vertices without out-edges, 0}.
__global__ void __launch_bounds__(PR_THREADS) k_pr_init(const PrStep a, uint64_t V, float x0)
{
    double m = 0, d = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t deg = a.row[v + 1] - a.row[v];
        a.x_out[v] = x0;
        a.b_next[v] = deg ? __fdiv_rn(x0, (float)deg) : 0.0f;
        m += (double)x0;
        if (!deg) d += (double)x0;
    }
    pr_block_diag(m, d, 0.0, a.diag);
}

// out[i] = x[new_of_old[i]]: the values in the caller's numbering.
__global__ void k_pr_by_id(const float* __restrict__ x, const uint32_t* __restrict__ new_of_old, uint64_t V,
                           float* __restrict__ out)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < V; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = x[new_of_old[i]];
}

// Edges of a row; no row but a hub's comes near the limit.
__device__ __forceinline__ uint32_t pr_edges(uint64_t r0, uint64_t r1)
{
    return r1 - r0 < 0x7fffffffull ? (uint32_t)(r1 - r0) : 0x7fffffffu;
}

// The list's vertices, G lanes each; SKIP: hubs are passed over.  What bounds
// a row is the chain list entry -> row bounds -> ids -> quotients, so it is
// pipelined over the group's next rows as in the FP64 engine's gather: while
// a row's quotients are in flight, the next row's ids, the bounds of the one
// after it and the list entry of the one after that are loaded.  Directed
// R-MAT scale 25, 30 rounds: 63.0 ms with a launch per class, unpipelined, and
// a diagnostics pass; 60.6 ms now, of which rows of 17 to 4,096 edges 32.5
// (345 G edges/s, where the same ids gathered flat reach 354), hubs 16 (245
// G/s: their ids hit the L1 least), short rows 10.  16 lanes for all longer
// rows 63.1, 2 or 4 lanes for the short ones 62.3 / 67.6, 5 CTAs per SM (it
// spills) 65.5, 3 CTAs 62.5 ms.
template <int G, bool SKIP, bool COMP, bool LAST>
__device__ __forceinline__ void pr_rows(const PrStep& a, const uint32_t* __restrict__ list, uint64_t n, PrDiag& g)
{
    const int lane = threadIdx.x & 31, gl = lane & (G - 1);
    const unsigned mask = (((1u << G) - 1u) << (lane & ~(G - 1)));
    const uint64_t step = ((uint64_t)gridDim.x * blockDim.x) / G;
    uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / G;
    if (i >= n) return;
    const bool quads = a.quads;
    // v: the row being summed, u: the next, t: the one after it.  Past the
    // list's end vertex 0 stands in: loaded, never summed.
    uint32_t v = list[i], u = i + step < n ? list[i + step] : 0u, t = i + 2 * step < n ? list[i + 2 * step] : 0u;
    uint64_t v0 = a.in_row[v], u0 = a.in_row[u];
    uint32_t vd = pr_edges(v0, a.in_row[v + 1]), ud = pr_edges(u0, a.in_row[u + 1]);
    uint4 qv = make_uint4(0, 0, 0, 0);
    if (quads) qv = pr_ld_quad(a, v0, vd, 4 * gl);
    for (; i < n; i += step) {
        const float xp = gl == 0 ? a.x_prev[v] : 0.0f;
        const uint64_t deg = gl == 0 ? pr_deg(a, v, vd) : 0;
        const uint32_t w = i + 3 * step < n ? list[i + 3 * step] : 0u;
        const uint64_t t0 = a.in_row[t], t1 = a.in_row[t + 1];
        uint4 qu = make_uint4(0, 0, 0, 0);
        if (quads) qu = pr_ld_quad(a, u0, ud, 4 * gl);
        float s = 0.0f, c = 0.0f;
        const bool skip = SKIP && vd > a.hub_min;
        if (skip) vd = 0;
        if (quads) {
            pr_add_quad<COMP>(a, qv, v0, vd, 4 * gl, s, c);
            const uint32_t len = ((uint32_t)v0 & 3u) + vd;
            for (uint32_t rel = 4 * gl + 4 * G; rel < len; rel += 4 * G)
                pr_add_quad<COMP>(a, pr_ld_quad(a, v0, vd, rel), v0, vd, rel, s, c);
        } else {
            pr_gather<COMP>(a, v0, v0 + vd, gl, G, s, c);
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            const float s2 = __shfl_down_sync(mask, s, o, G);
            const float c2 = __shfl_down_sync(mask, c, o, G);
            pr_merge<COMP>(s, c, s2, c2);
        }
        if (gl == 0 && !skip) pr_finish<LAST>(a, v, deg, xp, __fadd_rn(s, c), g);
        v = u;
        u = t;
        t = w;
        v0 = u0;
        vd = ud;
        u0 = t0;
        ud = pr_edges(t0, t1);
        qv = qu;
    }
}

// Hubs, a warp per chunk: the chunk's pair is stored, and the warp whose chunk
// arrives last merges the hub's pairs in chunk order and updates the vertex;
// no warp waits for another.
template <bool COMP, bool LAST>
__device__ __forceinline__ void pr_hubs(const PrStep& a, PrDiag& g)
{
    const int lane = threadIdx.x & 31;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t ch = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; ch < a.chunks; ch += warps) {
        const uint32_t i = a.owner[ch];
        const uint4 hub = a.hub[i];
        const uint64_t v = hub.x, row0 = a.in_row[v], end = a.in_row[v + 1];
        const uint64_t e0 = row0 + (ch - hub.y) * a.chunk, e1 = e0 + a.chunk < end ? e0 + a.chunk : end;
        float s = 0.0f, c = 0.0f;
        if (a.quads) {
            const uint32_t deg = (uint32_t)(e1 - e0), len = ((uint32_t)e0 & 3u) + deg;
            uint4 q = pr_ld_quad(a, e0, deg, 4 * lane);
            for (uint32_t rel = 4 * lane; rel < len; rel += 128) {
                const uint4 next = pr_ld_quad(a, e0, deg, rel + 128);
                pr_add_quad<COMP>(a, q, e0, deg, rel, s, c);
                q = next;
            }
        } else {
            pr_gather<COMP>(a, e0, e1, lane, 32, s, c);
        }
        pr_warp_merge<COMP>(s, c);
        int last = hub.z == 1 ? 1 : 0;
        if (lane == 0 && hub.z != 1) {
            a.partial[ch] = make_float2(s, c);
            __threadfence();
            last = atomicAdd(&a.arrived[i], 1u) == hub.z - 1 ? 1 : 0;
        }
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last && hub.z != 1) {
            __threadfence();
            s = c = 0.0f;
            for (uint32_t k = lane; k < hub.z; k += 32) {
                const float2 p = __ldcg(&a.partial[hub.y + k]);
                pr_merge<COMP>(s, c, p.x, p.y);
            }
            pr_warp_merge<COMP>(s, c);
            if (lane == 0) a.arrived[i] = 0;  // every chunk of the hub has arrived
        }
        if (lane == 0 && last) pr_finish<LAST>(a, v, pr_deg(a, v, end - row0), a.x_prev[v], __fadd_rn(s, c), g);
    }
}

// A vertex without in-edges has the value ratio from superstep 1 on.  Its
// value and quotient are written in supersteps 1 and 2, once into each buffer,
// and stand there for the rest of the run; k_pr_step adds its diagnostics.
// About half of an R-MAT graph's vertices are such.
__global__ void __launch_bounds__(PR_THREADS) k_pr_empty(const PrStep a, const uint32_t* __restrict__ list)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < a.empty; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = list[i], deg = a.row[v + 1] - a.row[v];
        a.x_out[v] = a.ratio;
        a.b_next[v] = deg ? __fdiv_rn(a.ratio, (float)deg) : 0.0f;
    }
}

struct PrHasEdges {
    const uint64_t* row;
    __device__ bool operator()(uint32_t v) const { return row[v + 1] > row[v]; }
};

// cnt += vertices of the list without out-edges
__global__ void k_pr_count_dangling(const uint32_t* __restrict__ list, uint64_t n, const uint64_t* __restrict__ row,
                                    unsigned long long* __restrict__ cnt)
{
    unsigned long long c = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        c += row[list[i] + 1] == row[list[i]];
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(cnt, c);
}

template <bool COMP, bool LAST>
__global__ void __launch_bounds__(PR_THREADS, PR_CTAS) k_pr_step(const PrStep a)
{
    // lets the next superstep's CTAs onto the SMs as this one's leave them, and
    // waits for the one before (neither does anything in a plain launch)
    asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
    PrDiag g;
    pr_hubs<COMP, LAST>(a, g);  // the longest work items first
    pr_rows<PR_LONG, true, COMP, LAST>(a, a.list[2], a.n[2], g);
    pr_rows<PR_GROUP, false, COMP, LAST>(a, a.list[1], a.n[1], g);
    pr_rows<PR_SHORT, false, COMP, LAST>(a, a.list[0], a.n[0], g);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // the vertices without in-edges: a.ratio each
        const double x = (double)a.ratio;
        g.m += (double)a.empty * x;
        g.d += (double)a.empty_dangling * x;
        if (a.first) g.r += (double)a.empty * fabs(x - (double)a.x0);
    }
    pr_block_diag(g.m, g.d, g.r, a.diag);
}

// Edges below which a superstep starts while the one before drains
// (programmatic dependent launch): the gap between them is a fifth of a
// superstep on a small graph.  20 rounds on R-MAT, started early / not, us: 1,024
// vertices 233 / 281, 65,536 vertices 269 / 316, 262,144 (8 M edges) 936 / 976,
// 1 M (31 M edges) 2,345 / 2,450, 2 M (62 M edges) 3,488 / 3,486 (not started early).
#define PR_EARLY (1ULL << 25)

// Grid-stride kernels get exactly the CTAs that are resident at once: more
// would run as a second wave after the first finished its static share.
template <class K>
int pr_occupancy(K kernel)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, PR_THREADS, 0) != cudaSuccess || n <= 0) n = 1;
    return n < PR_CTAS_PER_SM ? n : PR_CTAS_PER_SM;
}

int pr_min_occupancy()
{
    int n = PR_CTAS_PER_SM;
    auto low = [&](int k) { n = k < n ? k : n; };
    low(pr_occupancy(k_pr_step<true, false>));
    low(pr_occupancy(k_pr_step<true, true>));
    low(pr_occupancy(k_pr_step<false, false>));
    low(pr_occupancy(k_pr_step<false, true>));
    return n;
}

template <class T>
int pr_alloc(ipg_pr_plan* p, T** out, uint64_t n)
{
    void* d = nullptr;
    const uint64_t bytes = (n ? n : 1) * sizeof(T);
    PR_TRY(ipg_dev_alloc(&d, bytes));
    p->allocs.push_back({d, bytes});
    *out = (T*)d;
    return IPG_OK;
}

// The short class again, vertices without in-edges behind the others.  Where
// there is no room for it, the class serves as it is, every vertex a row.
int pr_split_shorts(ipg_pr_plan* p)
{
    const uint64_t ns = p->bins.count[0];
    if (!ns) return IPG_OK;
    const PrHasEdges has{p->gv.d_in_row};
    const uint32_t* list = p->bins.d_list[0];
    size_t tb = 0;
    void* mem[2] = {nullptr, nullptr};  // the list; scratch and {with in-edges, dangling}
    cudaError_t e = cub::DevicePartition::If(nullptr, tb, list, (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)ns, has);
    const uint64_t bytes[2] = {ns * 4, ((uint64_t)tb + 15) / 16 * 16 + 16};
    int r = IPG_OK;
    for (int k = 0; k < 2 && e == cudaSuccess && r == IPG_OK; k++) r = ipg_dev_alloc(&mem[k], bytes[k]);
    unsigned long long h[2] = {0, 0};
    if (e == cudaSuccess && r == IPG_OK) {
        uint32_t* shorts = (uint32_t*)mem[0];
        unsigned long long* cnt = (unsigned long long*)((char*)mem[1] + bytes[1] - 16);
        e = cudaMemset(cnt, 0, 16);
        if (e == cudaSuccess) e = cub::DevicePartition::If(mem[1], tb, list, shorts, (uint32_t*)cnt, (int64_t)ns, has);
        if (e == cudaSuccess) e = cudaMemcpy(h, cnt, 16, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && h[0] < ns) {
            k_pr_count_dangling<<<p->grid_flat, PR_THREADS>>>(shorts + h[0], ns - h[0], p->gv.d_row, cnt + 1);
            e = cudaMemcpy(h, cnt, 16, cudaMemcpyDeviceToHost);
        }
    }
    ipg_dev_free(mem[1], bytes[1]);
    if (e != cudaSuccess || r != IPG_OK) {
        ipg_dev_free(mem[0], bytes[0]);
        if (e != cudaSuccess) return ipg_internal_fail(IPG_ECUDA, cudaGetErrorString(e));
        return r == IPG_EBUDGET || r == IPG_ENOMEM ? IPG_OK : r;
    }
    p->allocs.push_back({mem[0], bytes[0]});
    p->shorts = (uint32_t*)mem[0];
    p->empty = ns - h[0];
    p->empty_dangling = h[1];
    return IPG_OK;
}

// Error of an FP32 vector against an FP64 one: out[0] = max abs, out[1] =
// max rel (abs where the reference is 0), out[2] = sum of abs, as doubles.
// Non-negative doubles order as their bit patterns, so the maxima use integer
// atomics.
__global__ void k_err_f32_f64(const float* __restrict__ a, const double* __restrict__ ref, uint64_t n,
                              unsigned long long* __restrict__ out)
{
    double mabs = 0, mrel = 0, sabs = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const double e = fabs((double)a[i] - ref[i]);
        const double r = ref[i] != 0.0 ? e / fabs(ref[i]) : e;
        mabs = e > mabs ? e : mabs;
        mrel = r > mrel ? r : mrel;
        sabs += e;
    }
    atomicMax(&out[0], (unsigned long long)__double_as_longlong(mabs));
    atomicMax(&out[1], (unsigned long long)__double_as_longlong(mrel));
    atomicAdd((double*)&out[2], sabs);
}

// out[3] = smallest index whose abs error equals the maximum.
__global__ void k_err_argmax(const float* __restrict__ a, const double* __restrict__ ref, uint64_t n,
                             unsigned long long* __restrict__ out)
{
    const double mabs = __longlong_as_double((long long)out[0]);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (fabs((double)a[i] - ref[i]) == mabs) atomicMin(&out[3], (unsigned long long)i);
}

}  // namespace

extern "C" int ipg_pr_plan_create(ipg_graph* g, ipg_pr_plan** out)
{
    if (!g || !out) return ipg_internal_fail(IPG_EINVAL, "ipg_pr_plan_create: null argument");
    *out = nullptr;
    ipg_pr_plan* p = new (std::nothrow) ipg_pr_plan();
    if (!p) return ipg_internal_fail(IPG_ENOMEM, "ipg_pr_plan_create: out of host memory");
    int r = IPG_OK;
    do {
        p->g = g;
        if ((r = ipg_graph_view_get(g, &p->gv)) != IPG_OK) break;
        if (p->gv.id_bytes != 4) {
            r = ipg_internal_fail(IPG_EINVAL, "ipg_pr_plan_create: the FP32 PageRank takes 32-bit vertex ids");
            break;
        }
        if (p->gv.V >= (1ULL << 32)) {
            r = ipg_internal_fail(IPG_EINVAL, "ipg_pr_plan_create: more than 2^32 - 1 vertices");
            break;
        }
        p->sms = ipg_sm_count();
        const char* t0s = getenv("IPG_PR_T0");
        const char* t1s = getenv("IPG_PR_T1");
        const uint64_t t0 = (t0s && *t0s) ? strtoull(t0s, nullptr, 10) : 16;
        const uint64_t t1 = (t1s && *t1s) ? strtoull(t1s, nullptr, 10) : 4096;
        // the gathers run on the degree-ordered copy unless IPG_ORDER=0 (or
        // the copy does not fit the HBM budget): the most gathered
        // quotients share cache lines
        ipg_graph* gw = g;
        const char* ord = getenv("IPG_ORDER");
        if (!(ord && *ord && strtoull(ord, nullptr, 10) == 0) && p->gv.V < (1ULL << 31)) {
            ipg_order o;
            const int ro = ipg_graph_degree_order(g, 1, &o);
            if (ro == IPG_OK) {
                gw = o.graph;
                p->new_of_old = o.d_new_of_old;
            } else if (ro != IPG_EBUDGET && ro != IPG_ENOMEM) {
                r = ro;
                break;
            }
        }
        if ((r = ipg_graph_view_get(gw, &p->gv)) != IPG_OK) break;
        p->grid = (uint32_t)p->sms * (uint32_t)pr_min_occupancy();
        p->grid_flat = (uint32_t)p->sms * (uint32_t)pr_occupancy(k_pr_init);
        // hub chunks: at most PR_CHUNK edges, fewer on a small graph so that
        // every resident warp gets several (a quarter of its share); rows
        // above a chunk (or t1) are hubs
        const uint64_t share = p->gv.E / ((uint64_t)p->grid * (PR_THREADS / 32) * 4);
        p->chunk = 256;
        while (p->chunk < PR_CHUNK && p->chunk * 2 <= share) p->chunk *= 2;
        p->hub_min = t1 < p->chunk ? t1 : p->chunk;
        const uint64_t ts = t0 < p->hub_min ? t0 : p->hub_min;
        const uint64_t mid = PR_MID < p->hub_min ? PR_MID : p->hub_min;
        // classes over the gather lists (builds the in-lists of a directed graph)
        if ((r = ipg_graph_bins(gw, 1, ts, mid > ts ? mid : ts, &p->bins)) != IPG_OK) break;
        if ((r = ipg_graph_hold(gw, p->bins.d_list[0], &p->holds[0])) != IPG_OK) break;
        if ((r = ipg_graph_hubs(gw, 1, p->hub_min, p->chunk, &p->hubs)) != IPG_OK) break;
        if ((r = ipg_graph_hold(gw, p->hubs.d_hub, &p->holds[1])) != IPG_OK) break;
        if ((r = ipg_graph_view_get(gw, &p->gv)) != IPG_OK) break;
        int quads = 0;
        if ((r = ipg_graph_quads(gw, 1, &quads)) != IPG_OK) break;
        p->quads = quads != 0;
        const uint64_t V = p->gv.V;
        if ((r = pr_alloc(p, &p->b[0], V)) != IPG_OK) break;
        if ((r = pr_alloc(p, &p->b[1], V)) != IPG_OK) break;
        if ((r = pr_alloc(p, &p->xs, V)) != IPG_OK) break;
        if (p->new_of_old && (r = pr_alloc(p, &p->xs2, V)) != IPG_OK) break;
        if ((r = pr_alloc(p, &p->partial, p->hubs.chunks)) != IPG_OK) break;
        if ((r = pr_alloc(p, &p->arrived, p->hubs.hubs)) != IPG_OK) break;
        cudaError_t e = cudaMemset(p->arrived, 0, (p->hubs.hubs ? p->hubs.hubs : 1) * 4);
        if (e != cudaSuccess) {
            r = ipg_internal_fail(IPG_ECUDA, cudaGetErrorString(e));
            break;
        }
        if ((r = pr_split_shorts(p)) != IPG_OK) break;
        // the classes as the plan's user knows them: thread, lanes, hubs
        p->class_count[0] = p->bins.count[0];
        p->class_edges[0] = p->bins.edges[0];
        p->class_count[2] = p->hubs.hubs;
        p->class_edges[2] = p->hubs.edges;
        p->class_count[1] = p->bins.count[1] + p->bins.count[2] - p->hubs.hubs;
        p->class_edges[1] = p->bins.edges[1] + p->bins.edges[2] - p->hubs.edges;
    } while (0);
    if (r != IPG_OK) {
        ipg_pr_plan_free(p);
        return r;
    }
    *out = p;
    return IPG_OK;
}

extern "C" void ipg_pr_plan_free(ipg_pr_plan* p)
{
    if (!p) return;
    for (auto& a : p->allocs) ipg_dev_free(a.first, a.second);
    for (ipg_hold* h : p->holds) ipg_hold_release(h);
    delete p;
}

extern "C" int ipg_pr_run_f32(ipg_pr_plan* p, uint32_t rounds, double damping, int compensated, float* d_values,
                              double* d_diag, void* stream)
{
    if (!p || !d_values || !d_diag) return ipg_internal_fail(IPG_EINVAL, "ipg_pr_run_f32: null argument");
    if (!(damping >= 0.0 && damping <= 1.0)) return ipg_internal_fail(IPG_EINVAL, "ipg_pr_run_f32: damping outside [0, 1]");
    cudaStream_t st = (cudaStream_t)stream;
    const uint64_t V = p->gv.V;
    PR_CUDA(cudaMemsetAsync(d_diag, 0, (uint64_t)(rounds + 1) * 3 * sizeof(double), st));
    if (V == 0) return IPG_OK;
    PrStep a;
    a.row = p->gv.d_row;
    a.in_row = p->gv.d_in_row;
    a.in_adj = (const uint32_t*)p->gv.d_in_adj;
    a.quads = p->quads;
    for (int k = 0; k < 3; k++) {
        a.list[k] = p->bins.d_list[k];
        a.n[k] = p->bins.count[k];
    }
    if (p->shorts) a.list[0] = p->shorts;
    a.n[0] -= p->empty;
    a.empty = p->empty;
    a.empty_dangling = p->empty_dangling;
    a.hub = (const uint4*)p->hubs.d_hub;
    a.owner = p->hubs.d_owner;
    a.partial = p->partial;
    a.arrived = p->arrived;
    a.chunks = p->hubs.chunks;
    a.chunk = p->chunk;
    a.hub_min = p->hub_min;
    // superstep s writes its values to xbuf(s), so that the last one lands in
    // d_values (on the renamed copy: in xs2, gathered into d_values at the end)
    float* last = p->new_of_old ? p->xs2 : d_values;
    auto xbuf = [&](uint32_t s) { return ((rounds - s) & 1) ? p->xs : last; };
    a.ratio = (float)((1.0 - damping) / (double)V);  // pagerank.c:98 (0.15 / V)
    a.damping = (float)damping;
    a.b_cur = nullptr;
    a.b_next = p->b[0];
    a.x_out = xbuf(0);
    a.x_prev = nullptr;
    a.diag = d_diag;
    a.x0 = (float)(1.0 / (double)V);  // pagerank.c:99
    // no more CTAs than the graph has rows and pairs of edges for
    const uint64_t ctas = (V + p->gv.E / 2 + PR_THREADS - 1) / PR_THREADS;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    PR_CUDA(cudaStreamIsCapturing(st, &capture));
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((uint32_t)(ctas < p->grid ? ctas : p->grid));
    cfg.blockDim = dim3(PR_THREADS);
    cfg.stream = st;
    cfg.attrs = &early;
    cfg.numAttrs = p->gv.E < PR_EARLY && capture == cudaStreamCaptureStatusNone ? 1 : 0;
    k_pr_init<<<p->grid_flat, PR_THREADS, 0, st>>>(a, V, a.x0);
    PR_CUDA(cudaGetLastError());
    for (uint32_t s = 1; s <= rounds; s++) {
        a.b_cur = p->b[(s - 1) & 1];
        a.b_next = p->b[s & 1];
        a.x_prev = xbuf(s - 1);
        a.x_out = xbuf(s);
        a.diag = d_diag + (uint64_t)s * 3;
        a.first = s == 1;
        if (s <= 2 && a.empty) k_pr_empty<<<p->grid_flat, PR_THREADS, 0, st>>>(a, p->shorts + a.n[0]);
        const bool last = s == rounds;
        PR_CUDA(cudaLaunchKernelEx(&cfg,
                                   compensated ? (last ? k_pr_step<true, true> : k_pr_step<true, false>)
                                               : (last ? k_pr_step<false, true> : k_pr_step<false, false>),
                                   a));
    }
    if (p->new_of_old) {
        k_pr_by_id<<<p->grid_flat, PR_THREADS, 0, st>>>(last, p->new_of_old, V, d_values);
        PR_CUDA(cudaGetLastError());
    }
    return IPG_OK;
}

extern "C" int ipg_pr_plan_info(const ipg_pr_plan* p, uint64_t* class_counts, uint64_t* class_edges,
                                uint64_t* hub_chunks)
{
    if (!p) return ipg_internal_fail(IPG_EINVAL, "ipg_pr_plan_info: null plan");
    for (int k = 0; k < 3; k++) {
        if (class_counts) class_counts[k] = p->class_count[k];
        if (class_edges) class_edges[k] = p->class_edges[k];
    }
    if (hub_chunks) *hub_chunks = p->hubs.chunks;
    return IPG_OK;
}

extern "C" int ipg_error_f32_f64(const float* d_a, const double* d_ref, uint64_t n, double* max_abs, double* max_rel,
                                 double* mean_abs, uint64_t* argmax_abs, void* stream)
{
    if ((!d_a || !d_ref) && n) return ipg_internal_fail(IPG_EINVAL, "ipg_error_f32_f64: null argument");
    cudaStream_t st = (cudaStream_t)stream;
    unsigned long long* d_out = nullptr;
    PR_TRY(ipg_dev_alloc((void**)&d_out, 4 * sizeof(unsigned long long)));
    unsigned long long h[4] = {0, 0, 0, ~0ULL};
    cudaError_t e = cudaMemcpyAsync(d_out, h, sizeof h, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && n) {
        const uint64_t blocks = (n + 255) / 256;
        const uint32_t grid = (uint32_t)(blocks < 1184 ? blocks : 1184);
        k_err_f32_f64<<<grid, 256, 0, st>>>(d_a, d_ref, n, d_out);
        k_err_argmax<<<grid, 256, 0, st>>>(d_a, d_ref, n, d_out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, d_out, sizeof h, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    ipg_dev_free(d_out, 4 * sizeof(unsigned long long));
    if (e != cudaSuccess) return ipg_internal_fail(IPG_ECUDA, cudaGetErrorString(e));
    double v[3];
    for (int k = 0; k < 3; k++) {
        long long bits = (long long)h[k];
        v[k] = *reinterpret_cast<double*>(&bits);
    }
    if (max_abs) *max_abs = v[0];
    if (max_rel) *max_rel = v[1];
    if (mean_abs) *mean_abs = n ? v[2] / (double)n : 0.0;
    if (argmax_abs) *argmax_abs = n ? h[3] : 0;
    return IPG_OK;
}
