// g5_batch.cu -- batched BFS: up to 64 roots per graph, any number of graphs
// of uneven scale, all together: g5_batch_run as one launch (k_bsearch), the
// asynchronous and serving forms in a device-resident level loop.
//
// Each vertex carries three 64-bit words (one bit per root of its graph):
// visited, frontier and next-frontier.  One read of a vertex's adjacency
// serves every root whose frontier touches it, which is where the batched
// form beats 64 one-root searches.  The reference has no batched search (it
// runs runBFS once per root, cpu_2d/main.cpp:419-462); this is the
// multi-source form of the same level-synchronous BFS.
//
// Per level and per graph the direction is chosen as in the plain search
// (Beamer's alpha/beta on the union frontier):
//   top-down   edge-balanced tiles over the active-vertex queue; for an edge
//              (u, v) the roots new to v, front[u] & ~visited[v], are OR-ed
//              into next[v] and each such root's parent slot takes an
//              atomicMin with u (skipped when the slot is already <= u)
//   bottom-up  each vertex not yet visited by every root scans its ascending
//              adjacency: hit = front[u] & still-needed roots; the first hit
//              of a root is its parent; the scan stops once no root is needed
// Both give every root the smallest previous-level neighbour as parent, the
// same parent as the plain search and the reference CPU BFS.
//
// The search runs on a copy of each graph whose vertices are numbered by
// descending degree: the few high-degree vertices, which most adjacency
// entries point at, then share a small range of the frontier array that stays
// in L2 while the bottom-up levels probe it at random.  Each row keeps its
// neighbours in original-id order, so the first hit along a row is still the
// smallest original id; parents and roots are translated at the boundary and
// the output is indexed by original ids.  The bottom-up sweep itself walks
// the vertices in original-id order, which spreads the long rows over the
// warps.
//
// Vertex ranges of the graphs are padded to whole compaction chunks so every
// chunk belongs to one graph; the level loop is one CUDA graph (conditional
// while node).
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <vector>

#include "g5_common.cuh"
#include "g5_internal.h"

namespace {

constexpr int kB = 256;
constexpr int kW = kB / 32;
constexpr int kChunk = 2048;           // vertices per compaction chunk
constexpr uint64_t kTile = 256;        // edges per top-down warp tile
constexpr int kSerial = 4;             // bottom-up entries scanned per lane first
constexpr int kMaxGraphs = 64;
constexpr uint64_t kBuMinFrac = 16;    // bottom-up only when frontier entries > n / kBuMinFrac
constexpr int kMaxLevels = 1024;

enum : int32_t { TD = 0, BU = 1 };

constexpr int kListDegBits = 24;
constexpr uint32_t kListDeg = (1u << kListDegBits) - 1;

struct GraphDesc {
    const int64_t *row_off;  // degree-ordered copy: rows by new id
    const uint32_t *col;     // new ids, each row in original-id order
    const uint32_t *orig;    // new id -> original id
    const uint32_t *perm;    // original id -> new id
    const uint4 *blist;      // the vertices with edges, by ascending original id (k_rl_list)
    uint64_t nblist;         // their count
    uint64_t step0;          // first bottom-up warp step of this graph
    int64_t n;
    int64_t nnz;
    uint64_t vbase;      // first global vertex id
    uint64_t pred_base;  // offset of vertex 0's parents in pred_out (nroots per vertex)
    uint64_t mask;       // one bit per root
    int32_t nroots;
    int32_t dir;         // direction for the current level
    uint64_t nf, mf;     // active vertices and their adjacency entries
    uint64_t mu;         // adjacency entries of not fully visited vertices
    uint64_t examined;
    uint64_t amask;      // roots whose frontier is not empty (this level)
    uint64_t amask_next; // being collected by k_bcount for the next level
};

struct BState {
    int32_t level;
    uint32_t err;
    uint64_t active;     // active vertices over all graphs (this level)
    uint64_t qlen;       // queue length (top-down graphs only)
    uint64_t qedges;     // its adjacency entries
    uint64_t examined;   // adjacency entries examined, all levels
    uint32_t dirs;       // this level: bit 0 a graph expands top-down, bit 1 bottom-up
};

struct BArgs {
    GraphDesc *gd;
    int ngraphs;
    const uint8_t *chunk_graph;
    uint32_t nchunks;
    uint64_t ntot;          // padded global vertex count
    const uint32_t *deg;    // per global vertex
    const uint32_t *iso;    // one bit per global vertex of degree 0
    uint64_t *vis, *front, *next;
    uint32_t *pred;         // output parents, vertex-major per graph: [v][nroots]
    uint32_t *queue;
    uint64_t *qoff;
    int64_t *qbase;
    uint32_t *tile_start;
    uint64_t max_tiles;
    uint64_t *chunk_n, *chunk_m;
    uint8_t *chunk_live;    // per chunk: bit 0 next frontier not empty, bit 1 nothing for k_bwrite
    const uint8_t *step_graph; // graph of each bottom-up warp step (32 list entries)
    uint64_t nsteps;
    BState *st;
    const int64_t *roots;   // device copy of the roots (graph-major)
    const int32_t *root_off;
    double alpha, beta;
    cudaGraphConditionalHandle cond;
    int use_cond;
    uint64_t *level_log;    // per level: active vertices
    int serving;            // continuous batching: no level cap, fixed m_u
};

__device__ __forceinline__ uint64_t wsum(uint64_t v) { return warp_sum_u64(v); }

__device__ __forceinline__ int graph_of(const BArgs &a, uint64_t v) { return a.chunk_graph[v / kChunk]; }

// 4-byte asynchronous copy global -> shared (cp.async): the issuing thread
// goes on at once; cp_async_wait_all() waits for all of its copies.
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    const size_t ga = __cvta_generic_to_global(gmem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(ga) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// ---- init: roots into next, parents of roots -------------------------------------

__global__ void k_binit(BArgs a)
{
    for (int g = blockIdx.x; g < a.ngraphs; g += gridDim.x) {
        GraphDesc &d = a.gd[g];
        for (int r = threadIdx.x; r < d.nroots; r += blockDim.x) {
            const int64_t root = a.roots[a.root_off[g] + r];
            if (root < 0 || root >= d.n) {
                atomicOr(&a.st->err, 1u);
                continue;
            }
            atomicOr((unsigned long long *)&a.next[d.vbase + d.perm[root]], 1ull << r);
            a.pred[d.pred_base + (uint64_t)root * d.nroots + r] = (uint32_t)root;
        }
        if (threadIdx.x == 0) {
            d.dir = TD;
            d.mu = (uint64_t)d.nnz;
            d.examined = 0;
            d.amask = 0;
            d.amask_next = 0;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.st->level = -1;
        a.st->err = 0;
        a.st->examined = 0;
    }
}

// ---- expansion ------------------------------------------------------------------------

__device__ void bexp_td(const BArgs &a, uint64_t &examined)
{
    __shared__ uint64_t s_q[kW][32];
    const int lane = g5_lane(), wib = threadIdx.x >> 5;
    const uint64_t gw = (uint64_t)blockIdx.x * kW + wib, nw = (uint64_t)gridDim.x * kW;
    const uint64_t mf = a.st->qedges, nf = a.st->qlen;
    const uint64_t ntiles = (mf + kTile - 1) / kTile;
    if (ntiles > a.max_tiles) {
        if (threadIdx.x == 0) atomicOr(&a.st->err, 2u);
        return;
    }
    for (uint64_t t = gw; t < ntiles; t += nw) {
        const uint64_t e0 = t * kTile, e1 = min(e0 + kTile, mf);
        uint64_t cur = a.tile_start[t];
        for (uint64_t gb = e0; gb < e1; gb += 32) {
            const uint64_t idx = cur + 1 + lane;
            s_q[wib][lane] = idx <= nf ? a.qoff[idx] : ~0ull;
            __syncwarp();
            const uint64_t e = gb + lane;
            int lo = 0, hi = 32;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (s_q[wib][mid] <= e) lo = mid + 1;
                else hi = mid;
            }
            const uint64_t i = cur + lo;
            bool in_range = true;
            if (lo == 32 && e < e1) in_range = (i + 1 > nf) ? false : (a.qoff[i + 1] > e);
            if (e < e1) {
                if (!in_range) {
                    atomicOr(&a.st->err, 4u);
                } else {
                    const uint32_t ug = a.queue[i];
                    const GraphDesc &d = a.gd[graph_of(a, ug)];
                    const uint32_t vl = __ldg(d.col + (a.qbase[i] + (int64_t)e));
                    const uint64_t vg = d.vbase + vl;
                    // roots new to v: the smallest frontier neighbour is the
                    // parent (atomicMin, after a plain read to skip most)
                    const uint64_t nb = a.front[ug] & ~a.vis[vg];
                    if (nb) {
                        const uint32_t ul = __ldg(d.orig + (ug - d.vbase));
                        uint32_t *pv = a.pred + d.pred_base + (uint64_t)__ldg(d.orig + vl) * d.nroots;
                        uint64_t x = nb;
                        while (x) {
                            const int r = __ffsll((long long)x) - 1;
                            x &= x - 1;
                            uint32_t *slot = pv + r;
                            if (*slot > ul) atomicMin(slot, ul);
                        }
                        if (nb & ~a.next[vg]) atomicOr((unsigned long long *)&a.next[vg], (unsigned long long)nb);
                    }
                }
            }
            cur = __shfl_sync(0xFFFFFFFFu, i, 31);
            __syncwarp();
        }
        if (lane == 0) examined += e1 - e0;
    }
}

__device__ __forceinline__ uint64_t warp_or_u64(uint64_t x)
{
    const uint32_t lo = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)x), hi = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(x >> 32));
    return lo | (uint64_t)hi << 32;
}

// Bottom-up: the candidates of v are the roots that have not visited it;
// the first frontier hit of each root along v's ascending adjacency is its
// parent.  A warp takes 32 consecutive vertices (never two graphs: graphs
// are chunk aligned).  Each lane first probes v's first kSerial entries with
// independent loads and keeps the hits as (parent, roots) events in shared
// memory (in the one-launch form again and again while many lanes are short of
// roots); vertices still missing roots are then scanned by the whole warp,
// 64 entries per step, whose first hits per root (an exclusive prefix OR over
// the lanes) are written at once.  The serial hits are written last, lane r
// taking root r of each vertex: each vertex's parents are one contiguous run
// of nroots words, so those stores are contiguous.
struct BuScratch {  // one warp's serial hits
    uint64_t evm[kSerial][32];
    uint32_t evu[kSerial][32];
};

// A row of which more than kLongRow entries are left after its warp has
// scanned kLongRow goes to `longs` in pieces of that many (SPLIT; bexp_long
// scans them afterwards): a hub's row of a million entries held its warp as
// long as all the others together needed for the level.  The owner's share keeps
// the early end of rows whose roots are soon found: with none of it, scale 24
// took 10958 us a batch instead of 8160, and without pieces 9593 (eight mixed
// graphs 1324, 1252 and 1432; before the roots that lag were split off).  Pieces of 128, 256, 512, 1024 and 2048 entries:
// 8598, 8266, 8154, 8152, 8222 (mixed 1325, 1280, 1257, 1235, 1306; scale 16 211,
// 220, 242, 244, 244).
constexpr uint32_t kLongRow = 512;

// While this many lanes are still short of roots they go on by themselves for
// another kSerial entries: a window of 64 entries takes the warp as long as a
// round of the lanes, 4 entries each.  us per batch, from 6, 10, 16, 24 and never:
// scale 24 6511, 6482, 6597, 6713, 6670; scale 20 660, 650, 649, 664, 666; the
// eight mixed graphs 1125, 1078, 1071, 1078, 1078.
constexpr int kMany = 12;

// Entries [start, start + cnt) of global vertex u's row, and the roots it is
// still to be searched for.
struct __align__(32) LongItem {
    int64_t start;  // in the graph's col
    uint64_t need;
    uint32_t u;
    uint32_t cnt;   // | graph << 16
    uint64_t pad;
};

struct LongRows {
    LongItem *items;
    unsigned long long *alloc;
    uint32_t *steps;  // shared: steps the block has given out
};

// Writes the warp's serial hits: the parents of (vertex, roots) events, two at a
// time over the warp: lane k writes roots k and k + 32.  Empty events cost
// nothing, and the events' root sets are disjoint, so each parent is written once.
__device__ __forceinline__ void put_events(const BArgs &a, const GraphDesc &d, BuScratch &ws, uint32_t vo)
{
    const int lane = g5_lane();
    const uint32_t R = (uint32_t)d.nroots;
    cp_async_wait_all();
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kSerial; ++k) {
        unsigned em = __ballot_sync(0xFFFFFFFFu, ws.evm[k][lane] != 0ull);
        while (em) {
            // two events together: their loads overlap
            const int v0 = __ffs(em) - 1;
            em &= em - 1;
            const int v1 = em ? __ffs(em) - 1 : v0;
            const uint64_t m0 = ws.evm[k][v0], m1 = em ? ws.evm[k][v1] : 0ull;
            const uint32_t u0 = ws.evu[k][v0], u1 = ws.evu[k][v1];
            uint32_t *p0 = a.pred + d.pred_base + (uint64_t)__shfl_sync(0xFFFFFFFFu, vo, v0) * R;
            uint32_t *p1 = a.pred + d.pred_base + (uint64_t)__shfl_sync(0xFFFFFFFFu, vo, v1) * R;
            em &= em - 1;
            if ((m0 >> lane) & 1ull) p0[lane] = u0;
            if ((m0 >> (lane + 32)) & 1ull) p0[lane + 32] = u0;
            if ((m1 >> lane) & 1ull) p1[lane] = u1;
            if ((m1 >> (lane + 32)) & 1ull) p1[lane + 32] = u1;
        }
    }
    __syncwarp();
}

// vps_shift: log2 of the vertices per warp step (32, less on graphs with fewer
// steps of 32 than there are warps: scale 8 took 84 us at 32 and takes 76).
template <bool SPLIT>
__device__ __forceinline__ void bexp_bu(const BArgs &a, const GraphDesc *gd, BuScratch &ws, uint64_t gw, uint64_t nw,
                                        int vps_shift, LongRows longs, uint64_t &examined)
{
    const int lane = g5_lane();
    const uint64_t steps = a.nsteps << (5 - vps_shift);
    uint64_t w = gw;
    while (w < steps) {
        // the graph's vertices with edges in original-id order, 32 per warp
        // step (vertices without edges are never reached, and half the
        // vertices of a Kronecker graph have none): high-degree vertices,
        // which have the lowest new ids, spread over the warps
        const int gi = a.step_graph[w >> (5 - vps_shift)];
        const GraphDesc &d = gd[gi];
        const uint64_t li = lane < 1 << vps_shift ? ((w - (d.step0 << (5 - vps_shift))) << vps_shift) + lane : d.nblist;
        const bool sweep = d.dir == BU && d.nf && d.amask;
        uint4 rec = make_uint4(0, 0, 0, 0);
        if (sweep && li < d.nblist) rec = __ldg(d.blist + li);
        if (SPLIT) {
            // the block's next step goes to its first free warp (fixed shares
            // left a sixth of the warps' time to waiting; steps claimed over the
            // whole grid, 2 ns each at one counter, cost the light levels of
            // scale 24 twice their time)
            uint32_t x = 0;
            if (lane == 0) x = atomicAdd(longs.steps, 1u);
            w = (uint64_t)__shfl_sync(0xFFFFFFFFu, x, 0) * gridDim.x + blockIdx.x;
        } else {
            w += nw;
        }
        if (!sweep) continue;
        const uint32_t R = (uint32_t)d.nroots;
        const uint32_t vo = rec.x, vl = rec.y;  // original id (its parents' row) and new
        const int64_t s = (int64_t)(rec.z | (uint64_t)(rec.w >> kListDegBits) << 32);
        uint32_t dg = rec.w & kListDeg;
        if (dg == kListDeg) dg = (uint32_t)(__ldg(d.row_off + vl + 1) - s);
        const int64_t e = s + dg;
        const uint64_t v = d.vbase + vl;
        // roots with an empty frontier cannot reach v
        uint64_t need = dg ? (~a.vis[v] & d.amask) : 0;
        uint64_t found = 0;
        int64_t j = s;
        uint64_t ex = 0;
        for (;;) {
            // serial probes: all loads first, then the hits in adjacency order
            uint32_t u[kSerial];
            uint64_t f[kSerial];
#pragma unroll
            for (int k = 0; k < kSerial; ++k) u[k] = (need && j + k < e) ? __ldg(d.col + j + k) : 0xFFFFFFFFu;
#pragma unroll
            for (int k = 0; k < kSerial; ++k) f[k] = u[k] != 0xFFFFFFFFu ? a.front[d.vbase + u[k]] : 0ull;
            uint32_t n = 0;  // entries examined
#pragma unroll
            for (int k = 0; k < kSerial; ++k) {
                const uint64_t hit = f[k] & need;
                ws.evm[k][lane] = hit;
                // the parent's original id lands in shared memory while the
                // rest of the row is scanned (read at the write-out below)
                if (hit) cp_async4(&ws.evu[k][lane], d.orig + u[k]);
                need &= ~hit;
                found |= hit;
                if (u[k] != 0xFFFFFFFFu && (need | hit)) n = k + 1;
            }
            j += n;
            ex += n;
            if (!SPLIT || __popc(__ballot_sync(0xFFFFFFFFu, need && j < e)) < kMany) break;
            put_events(a, d, ws, vo);
        }
        // short rows: pending vertices with at most 64 entries left are
        // packed whole, in lane order, into windows of 64 slots (slots lane
        // and lane + 32); each root's first hit in a row is found with a
        // segmented prefix OR over the slots
        while (true) {
            const bool sh = need && j < e && e - j <= 64;
            if (!__ballot_sync(0xFFFFFFFFu, sh)) break;
            const uint32_t r = sh ? (uint32_t)(e - j) : 0u;
            uint32_t inc = r;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += y;
            }
            const uint32_t start = inc - r;
            const bool in = sh && inc <= 64;  // row fits in this window
            uint32_t uq[2], s0q[2];
            uint64_t hq[2], vq[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint32_t k = (uint32_t)lane + 32u * q;
                // owner of slot k: the last lane whose row starts at or before k
                int ow = 0;
#pragma unroll
                for (int step = 16; step; step >>= 1) {
                    const uint32_t sv = __shfl_sync(0xFFFFFFFFu, start, ow + step);
                    if (sv <= k) ow += step;
                }
                const uint32_t s0 = __shfl_sync(0xFFFFFFFFu, start, ow);
                const uint32_t ro = __shfl_sync(0xFFFFFFFFu, in ? r : 0u, ow);
                const int64_t jo = __shfl_sync(0xFFFFFFFFu, j, ow);
                const uint64_t no = __shfl_sync(0xFFFFFFFFu, need, ow);
                vq[q] = __shfl_sync(0xFFFFFFFFu, (uint64_t)vo, ow);
                s0q[q] = s0;
                const bool live = k < s0 + ro;
                uq[q] = live ? __ldg(d.col + jo + (int64_t)(k - s0)) : 0xFFFFFFFFu;
                hq[q] = no;
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) hq[q] = uq[q] != 0xFFFFFFFFu ? (a.front[d.vbase + uq[q]] & hq[q]) : 0ull;
            // the parent's original id, loaded for every hit before the scans
            // below, so its latency overlaps them
            uint32_t oq[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) oq[q] = hq[q] ? __ldg(d.orig + uq[q]) : 0u;
            // segmented inclusive prefix OR: slots 0..31, then 32..63 with
            // the carry of a row that crosses slot 32
            uint64_t ia = hq[0], ib = hq[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t ya = __shfl_up_sync(0xFFFFFFFFu, ia, o);
                const uint64_t yb = __shfl_up_sync(0xFFFFFFFFu, ib, o);
                if (lane >= o && (uint32_t)lane - o >= s0q[0]) ia |= ya;
                if (lane >= o && (uint32_t)lane + 32u - o >= s0q[1]) ib |= yb;
            }
            const uint64_t ca = __shfl_sync(0xFFFFFFFFu, ia, 31);
            if (s0q[1] < 32) ib |= ca;
            const uint64_t pa = __shfl_up_sync(0xFFFFFFFFu, ia, 1);
            const uint64_t pb = __shfl_up_sync(0xFFFFFFFFu, ib, 1);
            const uint64_t ea = (uint32_t)lane > s0q[0] ? pa : 0ull;
            const uint64_t eb = (uint32_t)lane + 32u > s0q[1] ? (lane ? pb : ca) : 0ull;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                uint64_t x = hq[q] & ~(q ? eb : ea);
                if (x) {
                    uint32_t *pv = a.pred + d.pred_base + vq[q] * R;
                    const uint32_t uo = oq[q];
                    while (x) {
                        const int rr = __ffsll((long long)x) - 1;
                        x &= x - 1;
                        pv[rr] = uo;
                    }
                }
            }
            // each packed row takes its total from its last slot
            const uint32_t lk = in ? start + r - 1 : 0u;
            const uint64_t ta = __shfl_sync(0xFFFFFFFFu, ia, (int)(lk & 31));
            const uint64_t tb = __shfl_sync(0xFFFFFFFFu, ib, (int)(lk & 31));
            if (in) {
                const uint64_t seg = lk < 32 ? ta : tb;
                need &= ~seg;
                found |= seg;
                ex += r;
                j = e;
            }
        }
        // long rows: one vertex at a time, four windows of 32 entries per step
        unsigned pend = __ballot_sync(0xFFFFFFFFu, need && j < e);
        while (pend) {
            const int l = __ffs(pend) - 1;
            pend &= pend - 1;
            int64_t jj = __shfl_sync(0xFFFFFFFFu, j, l);
            const int64_t ee = __shfl_sync(0xFFFFFFFFu, e, l);
            uint64_t nd = __shfl_sync(0xFFFFFFFFu, need, l);
            uint32_t *pv = a.pred + d.pred_base + (uint64_t)__shfl_sync(0xFFFFFFFFu, vo, l) * R;
            const int64_t st = jj;
            uint64_t fnd = 0;
            // what is left of a long row after its first entries goes to
            // `longs`, with the roots it is still to be searched for
            const int64_t own = SPLIT && ee - jj > 2 * kLongRow ? jj + kLongRow : ee;
            while (jj < own && nd) {
                uint32_t uw[4];
                uint64_t hw[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int64_t i = jj + 32 * q + lane;
                    uw[q] = i < own ? __ldg(d.col + i) : 0xFFFFFFFFu;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) hw[q] = uw[q] != 0xFFFFFFFFu ? a.front[d.vbase + uw[q]] : 0ull;
                // one OR over the four windows; the first hits are located
                // only when the step holds a root not found before
                uint64_t lo = (hw[0] | hw[1] | hw[2] | hw[3]) & nd;
                lo = warp_or_u64(lo);
                if (!lo) {
                    jj += 128;
                    continue;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (!nd) break;
                    const uint64_t hit = hw[q] & nd;
                    if (!__ballot_sync(0xFFFFFFFFu, hit != 0)) {
                        jj += 32;
                        continue;
                    }
                    const uint32_t uo = hit ? __ldg(d.orig + uw[q]) : 0u;  // overlaps the scan
                    // first lane of each root: exclusive prefix OR over the lanes
                    uint64_t incl = hit;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                        if (lane >= o) incl |= y;
                    }
                    uint64_t excl = __shfl_up_sync(0xFFFFFFFFu, incl, 1);
                    if (lane == 0) excl = 0;
                    uint64_t x = hit & ~excl;
                    if (x) {
                        while (x) {
                            const int rr = __ffsll((long long)x) - 1;
                            x &= x - 1;
                            pv[rr] = uo;
                        }
                    }
                    const uint64_t all = __shfl_sync(0xFFFFFFFFu, incl, 31);
                    const unsigned cov = __ballot_sync(0xFFFFFFFFu, (incl & nd) == nd);
                    fnd |= all;
                    nd &= ~all;
                    jj += nd ? 32 : __ffs(cov);
                }
            }
            jj = min(jj, own);
            if (SPLIT && nd && own < ee) {
                const uint32_t pieces = (uint32_t)((ee - own + kLongRow - 1) / kLongRow);
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(longs.alloc, (unsigned long long)pieces);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                const uint32_t vv = __shfl_sync(0xFFFFFFFFu, (uint32_t)v, l);
                for (uint32_t k = lane; k < pieces; k += 32) {
                    LongItem it;
                    it.start = own + (int64_t)k * kLongRow;
                    it.u = vv;
                    it.cnt = (uint32_t)min(ee - it.start, (int64_t)kLongRow) | (uint32_t)gi << 16;
                    it.need = nd;
                    longs.items[base + k] = it;
                }
            }
            if (lane == l) {
                found |= fnd;
                need = nd;
                ex += (uint64_t)(jj - st);
            }
        }
        put_events(a, d, ws, vo);
        // (only this lane writes v in a bottom-up level, unless some roots go top-down)
        if (found) {
            if (SPLIT) atomicOr((unsigned long long *)&a.next[v], (unsigned long long)found);
            else a.next[v] |= found;
        }
        examined += ex;
    }
}

// The pieces of long rows, a warp each: as the long rows of bexp_bu, but each
// root's first hit in the piece takes its parent slot by atomicMin (rows are in
// original-id order, so the first hit of the whole row is the smallest id).
__device__ __forceinline__ void bexp_long(const BArgs &a, const GraphDesc *gd, const LongItem *items, uint64_t nitems,
                                          uint64_t gw, uint64_t nw)
{
    const int lane = g5_lane();
    for (uint64_t t = gw; t < nitems; t += nw) {
        const ulonglong2 x0 = __ldcg(reinterpret_cast<const ulonglong2 *>(items + t));
        const ulonglong2 x1 = __ldcg(reinterpret_cast<const ulonglong2 *>(items + t) + 1);
        const uint64_t v = (uint32_t)x1.x;
        const uint32_t cnt = (uint32_t)(x1.x >> 32);
        const GraphDesc &d = gd[cnt >> 16];
        int64_t jj = (int64_t)x0.x;
        const int64_t ee = jj + (cnt & 0xFFFFu);
        uint64_t nd = x0.y;
        uint32_t *pv = a.pred + d.pred_base + (uint64_t)__ldg(d.orig + (v - d.vbase)) * (uint32_t)d.nroots;
        uint64_t fnd = 0;
        while (jj < ee && nd) {
            uint32_t uw[4];
            uint64_t hw[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int64_t i = jj + 32 * q + lane;
                uw[q] = i < ee ? __ldg(d.col + i) : 0xFFFFFFFFu;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) hw[q] = uw[q] != 0xFFFFFFFFu ? a.front[d.vbase + uw[q]] & nd : 0ull;
            const uint64_t any = hw[0] | hw[1] | hw[2] | hw[3];
            const uint32_t lo = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)any), hi = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(any >> 32));
            jj += 128;
            uint64_t left = (uint64_t)hi << 32 | lo;
            if (!left) continue;
            fnd |= left;
            nd &= ~left;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint64_t hit = hw[q] & left;
                if (!__any_sync(0xFFFFFFFFu, hit != 0)) continue;
                const uint32_t uo = hit ? __ldg(d.orig + uw[q]) : 0u;
                uint64_t incl = hit;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl |= y;
                }
                uint64_t excl = __shfl_up_sync(0xFFFFFFFFu, incl, 1);
                if (lane == 0) excl = 0;
                for (uint64_t x = hit & ~excl; x; x &= x - 1) {
                    uint32_t *slot = pv + (__ffsll((long long)x) - 1);
                    if (*slot > uo) atomicMin(slot, uo);
                }
                left &= ~__shfl_sync(0xFFFFFFFFu, incl, 31);
            }
        }
        if (lane == 0 && (fnd & ~a.next[v])) atomicOr((unsigned long long *)&a.next[v], (unsigned long long)fnd);
    }
}

__global__ void __launch_bounds__(kB, 4) k_bbu(BArgs a)
{
    __shared__ BuScratch s_ws[kW];
    // no graph expands bottom-up this level
    if (a.st->err || a.st->level < 0 || a.st->active == 0 || !(a.st->dirs & 2u)) return;
    const uint64_t gw = ((uint64_t)blockIdx.x * kB + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * kB) >> 5;
    uint64_t examined = 0;
    bexp_bu<false>(a, a.gd, s_ws[threadIdx.x >> 5], gw, nw, 5, LongRows(), examined);
    examined = wsum(examined);
    if (g5_lane() == 0 && examined) atomicAdd((unsigned long long *)&a.st->examined, (unsigned long long)examined);
}

// Top-down part of a level (graphs expanding top-down).
__global__ void __launch_bounds__(kB, 8) k_btd(BArgs a)
{
    if (a.st->err || a.st->level < 0 || a.st->active == 0 || a.st->qedges == 0) return;
    uint64_t ex = 0;
    bexp_td(a, ex);
    ex = wsum(ex);
    if (g5_lane() == 0 && ex) atomicAdd((unsigned long long *)&a.st->examined, (unsigned long long)ex);
}

// ---- compaction ---------------------------------------------------------------------------

// One warp per chunk over a persistent grid: the chunk's 2048 next words in
// coalesced 256-byte loads, 16 in flight per lane, then the degrees of the
// non-empty ones (no per-chunk block, barrier or serial tail).
__global__ void __launch_bounds__(kB) k_bcount(BArgs a)
{
    constexpr int kBatch = 16;
    const int lane = g5_lane();
    const uint64_t gw = ((uint64_t)blockIdx.x * kB + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * kB) >> 5;
    for (uint64_t c = gw; c < a.nchunks; c += nw) {
        const uint64_t v0 = c * kChunk;
        const uint8_t live = a.chunk_live[c];
        uint64_t cn = 0, cm = 0, act = 0;
        for (int i0 = 0; i0 < kChunk / 32; i0 += kBatch) {
            uint64_t x[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) x[k] = __ldg(a.next + v0 + (uint64_t)(i0 + k) * 32 + lane);
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                if (x[k]) {
                    ++cn;
                    cm += __ldg(a.deg + v0 + (uint64_t)(i0 + k) * 32 + lane);
                    act |= x[k];
                }
            }
        }
        cn = wsum(cn);
        cm = wsum(cm);
        // roots present in the next frontier of this chunk's graph
#pragma unroll
        for (int o = 16; o; o >>= 1) act |= __shfl_xor_sync(0xFFFFFFFFu, act, o);
        if (lane == 0) {
            a.chunk_n[c] = cn;
            a.chunk_m[c] = cm;
            // all chunks of a graph OR into one word: an atomic only for
            // roots not already recorded
            if (act) {
                unsigned long long *am = (unsigned long long *)&a.gd[a.chunk_graph[c]].amask_next;
                if (act & ~*(volatile unsigned long long *)am) atomicOr(am, (unsigned long long)act);
            }
            // no frontier this level nor the last: visited, front and next of
            // the chunk stay as they are, so the write pass skips it
            const bool prev = live & 1u, cur = cn != 0;
            a.chunk_live[c] = (uint8_t)(cur ? 1u : (prev ? 0u : 2u));
        }
    }
}

// Single block: per-graph totals and directions, then prefix sums over the
// chunks of top-down graphs (their vertices form the next queue).
__global__ void __launch_bounds__(1024) k_bscan(BArgs a)
{
    __shared__ uint64_t s_gn[kMaxGraphs], s_gm[kMaxGraphs];
    __shared__ int s_gdir[kMaxGraphs];
    for (int g = threadIdx.x; g < a.ngraphs; g += blockDim.x) {
        s_gn[g] = 0;
        s_gm[g] = 0;
    }
    if (threadIdx.x == 0) a.st->dirs = 0;
    __syncthreads();
    const uint32_t C = a.nchunks;
    // each warp owns a contiguous range of chunks and reads it 32 chunks at a
    // time (coalesced); a step inside one graph is summed with a warp
    // reduction and kept in registers until the graph changes
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t per_w = (C + 31) / 32;
    const uint32_t w0 = min(C, wid * per_w), w1 = min(C, w0 + per_w);
    {
        int cur = -1;
        uint64_t an = 0, am = 0;
        for (uint32_t c0 = w0; c0 < w1; c0 += 32) {
            const uint32_t c = c0 + lane;
            const bool ok = c < w1;
            const uint64_t xn = ok ? a.chunk_n[c] : 0, xm = ok ? a.chunk_m[c] : 0;
            const int g = ok ? a.chunk_graph[c] : -1;
            const int g0 = __shfl_sync(0xFFFFFFFFu, g, 0);
            if (__all_sync(0xFFFFFFFFu, !ok || g == g0)) {
                const uint64_t sn = wsum(xn), sm = wsum(xm);
                if (g0 != cur) {
                    if (lane == 0 && cur >= 0 && (an | am)) {
                        atomicAdd((unsigned long long *)&s_gn[cur], (unsigned long long)an);
                        atomicAdd((unsigned long long *)&s_gm[cur], (unsigned long long)am);
                    }
                    cur = g0;
                    an = am = 0;
                }
                an += sn;
                am += sm;
            } else if (ok && (xn | xm)) {  // a graph boundary inside the step
                atomicAdd((unsigned long long *)&s_gn[g], (unsigned long long)xn);
                atomicAdd((unsigned long long *)&s_gm[g], (unsigned long long)xm);
            }
        }
        if (lane == 0 && cur >= 0 && (an | am)) {
            atomicAdd((unsigned long long *)&s_gn[cur], (unsigned long long)an);
            atomicAdd((unsigned long long *)&s_gm[cur], (unsigned long long)am);
        }
    }
    __syncthreads();
    if (threadIdx.x < a.ngraphs) {
        GraphDesc &d = a.gd[threadIdx.x];
        const uint64_t tn = s_gn[threadIdx.x], tm = s_gm[threadIdx.x];
        int nd = d.dir;
        // Beamer's switch on the union frontier of the graph's roots (when
        // serving, roots come and go, so m_u stays the whole graph)
        const uint64_t mu_after = a.serving ? (uint64_t)d.nnz : (d.mu >= tm ? d.mu - tm : 0);
        if (a.st->level >= 0) {
            if (d.dir == TD) {
                // Beamer's test, and a frontier large enough to pay for a
                // sweep over all of the graph's vertices
                if ((double)tm > (double)mu_after / a.alpha && tm > (uint64_t)d.n / kBuMinFrac) nd = BU;
            } else if ((double)tn < (double)d.n / a.beta && tn < d.nf) {
                nd = TD;
            }
        }
        d.mu = mu_after;
        d.dir = nd;
        d.nf = tn;
        d.mf = tm;
        d.amask = d.amask_next & d.mask;
        d.amask_next = 0;
        s_gdir[threadIdx.x] = nd;
        if (tn) atomicOr(&a.st->dirs, nd == TD ? 1u : 2u);
    }
    __syncthreads();
    // exclusive prefix over the chunks of top-down graphs: warp totals, a
    // scan of the 32 totals, then each warp writes its range's offsets
    uint64_t tn_w = 0, tm_w = 0;
    for (uint32_t c0 = w0; c0 < w1; c0 += 32) {
        const uint32_t c = c0 + lane;
        if (c < w1 && s_gdir[a.chunk_graph[c]] == TD) {
            tn_w += a.chunk_n[c];
            tm_w += a.chunk_m[c];
        }
    }
    tn_w = wsum(tn_w);
    tm_w = wsum(tm_w);
    __shared__ uint64_t s_wn[32], s_wm[32];
    if (lane == 0) {
        s_wn[wid] = tn_w;
        s_wm[wid] = tm_w;
    }
    __syncthreads();
    uint64_t tot_n = 0, tot_m = 0, on = 0, om = 0;
    for (int i = 0; i < 32; ++i) {
        if (i == wid) {
            on = tot_n;
            om = tot_m;
        }
        tot_n += s_wn[i];
        tot_m += s_wm[i];
    }
    for (uint32_t c0 = w0; c0 < w1; c0 += 32) {
        const uint32_t c = c0 + lane;
        const bool ok = c < w1;
        const bool td = ok && s_gdir[a.chunk_graph[c]] == TD;
        const uint64_t xn = td ? a.chunk_n[c] : 0, xm = td ? a.chunk_m[c] : 0;
        uint64_t in = xn, im = xm;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t yn = __shfl_up_sync(0xFFFFFFFFu, in, o), ym = __shfl_up_sync(0xFFFFFFFFu, im, o);
            if (lane >= o) {
                in += yn;
                im += ym;
            }
        }
        if (ok) {
            a.chunk_n[c] = td ? on + in - xn : ~0ull;  // ~0: chunk not queued
            a.chunk_m[c] = om + im - xm;
        }
        on += __shfl_sync(0xFFFFFFFFu, in, 31);
        om += __shfl_sync(0xFFFFFFFFu, im, 31);
    }
    if (threadIdx.x == 0) {
        uint64_t act = 0;
        for (int g = 0; g < a.ngraphs; ++g) act += s_gn[g];
        BState *st = a.st;
        st->level += 1;
        st->active = act;
        st->qlen = tot_n;
        st->qedges = tot_m;
        a.qoff[tot_n] = tot_m;
        if (st->level < kMaxLevels) a.level_log[st->level] = act;
        bool cont = act > 0 && st->err == 0;
        if (cont && !a.serving && st->level + 1 >= kMaxLevels) {
            st->err |= 8u;
            cont = false;
        }
        if (a.use_cond) cudaGraphSetConditional(a.cond, cont ? 1u : 0u);
    }
}

// One warp per live chunk over a persistent grid: visited |= next, next ->
// front, and for chunks of top-down graphs the queue entries in ascending
// vertex order (a ballot per 32 words gives the positions, a warp scan the
// edge offsets).  All loads of a step come before its stores.
__global__ void __launch_bounds__(kB, 4) k_bwrite(BArgs a)
{
    constexpr int kBatch = 8;
    const int lane = g5_lane();
    const uint64_t gw = ((uint64_t)blockIdx.x * kB + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * kB) >> 5;
    for (uint64_t c = gw; c < a.nchunks; c += nw) {
        if (a.chunk_live[c] & 2u) continue;
        const uint64_t v0 = c * kChunk;
        uint64_t pos = a.chunk_n[c], mpos = a.chunk_m[c];
        const bool queued = pos != ~0ull;
        const GraphDesc &d = a.gd[a.chunk_graph[c]];
        for (int i0 = 0; i0 < kChunk / 32; i0 += kBatch) {
            uint64_t nx[kBatch], vs[kBatch];
            uint32_t dg[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) nx[k] = a.next[v0 + (uint64_t)(i0 + k) * 32 + lane];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                const uint64_t v = v0 + (uint64_t)(i0 + k) * 32 + lane;
                vs[k] = nx[k] ? a.vis[v] : 0ull;
                dg[k] = (nx[k] && queued) ? a.deg[v] : 0u;
            }
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                const uint64_t v = v0 + (uint64_t)(i0 + k) * 32 + lane;
                if (nx[k]) {
                    a.vis[v] = vs[k] | nx[k];
                    a.next[v] = 0;
                }
                a.front[v] = nx[k];
            }
            if (!queued) continue;
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                const unsigned bal = __ballot_sync(0xFFFFFFFFu, nx[k] != 0ull);
                if (!bal) continue;
                const uint64_t v = v0 + (uint64_t)(i0 + k) * 32 + lane;
                const uint64_t dv = dg[k];
                uint64_t incl = dv;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += y;
                }
                if (nx[k]) {
                    const uint64_t p = pos + __popc(bal & g5_lanemask_lt());
                    const uint64_t mp = mpos + incl - dv;
                    a.queue[p] = (uint32_t)v;
                    a.qoff[p] = mp;
                    a.qbase[p] = d.row_off[v - d.vbase] - (int64_t)mp;
                    uint64_t t = (mp + kTile - 1) / kTile;
                    const uint64_t tend = (mp + dv + kTile - 1) / kTile;
                    for (; t < tend && t < a.max_tiles; ++t) a.tile_start[t] = (uint32_t)p;
                }
                pos += __popc(bal);
                mpos += __shfl_sync(0xFFFFFFFFu, incl, 31);
            }
        }
    }
}

// ---- the whole batch as one launch -----------------------------------------------------
//
// g5_batch_run's form (the asynchronous and serving forms keep the level graph
// above, whose kernels other work on the GPU runs between): one cooperative
// grid of a block per SM but two, whose blocks meet twice a level.
//   expand  top-down graphs by work items of up to kItemEntries entries,
//           bottom-up ones as in k_bbu
//   commit  visited |= next, next -> front, the next frontier's sums per graph
//   decide  every block computes each graph's direction from the sums, and
//           which roots go top-down in its first bottom-up level all the same
// A top-down level of at most kClaimMax entries appends the rows it reaches
// first to the items of the next level; otherwise, and for graphs that come back
// from bottom-up, the items are built from the frontier words.
//
// Five launches and a while node a level cost about 35 us whatever the level
// held; a level now costs its work and 6-8 us.  Device us per batch of Kronecker
// graphs, 16 edges a vertex, before and after: scale 8, 4 roots, 230 and 71;
// scale 13, 64 roots, 410 and 138; scale 16 479 and 230; scale 20 1281 and 627;
// scale 24 10267 and 6140; eight graphs of scales 14 to 20, 16 roots each, 1820
// and 890 (with every SM; leaving two out costs at most 0.9 %).  What bounds it: the bottom-up sweeps, half by instructions and half
// by the latency of their gathers (39 % of the issue slots, 39 % of the memory
// bandwidth at 64 registers, which two windows of loads and 64-bit roots need;
// 48 registers and a quarter more warps measured slower).
constexpr int kSB = 1024;
constexpr int kSW = kSB / 32;
constexpr uint32_t kItemEntries = 256;
constexpr uint64_t kClaimMax = 1u << 18;
constexpr uint64_t kClaimedItems = 1u << 19;
constexpr int kRing = 4;  // levels of sums held
// Roots whose frontier has less than 1/kFewShare of the graph's entries, and all
// together at most 1/kFewTotal, expand top-down in the graph's first bottom-up
// level.  A root that lags behind (its few frontier vertices are nobody's
// neighbours) keeps every row of that level from being left early: with all 64
// roots of a scale-22 batch the level examines 102.7 M of 128 M entries, without
// the four that lag most 42 M, without eight 33 M.  Top-down an entry costs more
// (atomics all over the parents), so only few.  us per batch, shares of 32, 64,
// 128, 256 and none: scale 24 6676, 6661, 6667, 6891, 7659; scale 20 672, 668,
// 671, 672, 715; the eight mixed graphs 1082, 1089, 1078, 1082, 1116 (with a
// total of 1/4 instead, scale 24 11300).  Graphs of fewer than kSplitEntries
// entries are not worth the counting (scale 8 70 and 76).
constexpr uint64_t kFewShare = 128, kFewTotal = 32;
constexpr int64_t kSplitEntries = 1 << 16;
constexpr uint32_t kRootEntries = 16;  // the unit of the per-root sums (so that a block's fit 32 bits)

// A work item: entries [start, start + cnt) of the row of global vertex u.
struct __align__(16) BItem {
    uint32_t u;
    uint32_t cnt;    // | graph << 16
    int64_t start;   // in the graph's col
};

struct GraphSum {
    unsigned long long nf, mf, amask, pad;
};

struct LevelMeet {
    unsigned long long arrive[5];  // meetings of a level
    unsigned long long alloc;      // claimed items of its frontier
    unsigned long long built;      // items built for it
    unsigned long long longs;      // pieces of long rows
};

struct PArgs {
    BArgs b;
    const GraphDesc *gd;    // the host's descriptors of this run
    uint64_t npred;         // parents in pred_out
    BItem *claimed[2];      // by level parity
    uint64_t claimed_cap;
    BItem *built;
    LongItem *longs;        // pieces of long rows (bottom-up)
    int vps_shift;          // log2 of the vertices per bottom-up warp step
    GraphSum *sums;         // kRing x ngraphs
    unsigned long long *rsums;  // kRing x ngraphs x 64: entries of each root's frontier, in kRootEntries
    LevelMeet *meets;       // kRing; kRing levels are cleared at the start of a run
    unsigned *abort;
    uint32_t unit;          // vertices per warp step of the passes over the words (32, 64, ... 256)
    uint8_t *live;          // per unit: its frontier is not empty
    BState *out;            // pinned host
};

struct TdScratch {
    uint32_t end[32];
    uint32_t u[32];
    int64_t base[32];
    uint64_t front[32];
    uint8_t g[32];
};

union BWarpScratch {
    BuScratch bu;
    TdScratch td;
};

struct PShared {
    GraphDesc gd[kMaxGraphs];
    unsigned long long nf[kMaxGraphs], mf[kMaxGraphs], am[kMaxGraphs];  // the block's share of the next frontier
    uint32_t rs[kMaxGraphs][64];                                        // and of each root's
    uint64_t td_mask[kMaxGraphs];  // roots that expand top-down
    BWarpScratch w[kSW];
    unsigned long long active, td_entries;
    uint32_t dirs;   // bit 0: a graph expands top-down, bit 1: bottom-up
    uint32_t build;  // some graph's items are to be built
    uint32_t steps;  // bottom-up steps given out
    uint32_t splits;  // some graph's roots may split
    uint8_t build_g[kMaxGraphs];
    uint8_t split[kMaxGraphs];  // the graph turns bottom-up with this level
    uint32_t stop;
};

__device__ __forceinline__ void pmeet(const PArgs &a, PShared &sh, unsigned long long *word)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(word, 1ull << kArrive);
        unsigned long long x;
        if (!await<1>(word, a.abort, &x)) sh.stop = 1;
        __threadfence();
    }
    __syncthreads();
}

// Appends the rows of the warp's vertices (lanes with nseg > 0) to the items;
// long rows are laid out by the whole warp.
__device__ __forceinline__ void put_rows(BItem *items, uint64_t cap, uint64_t base, uint32_t excl, uint32_t ug, int g,
                                         int64_t s, uint32_t d, uint32_t nseg)
{
    if (base + excl + nseg > cap) nseg = 0;  // no room: the caller sees it from the total
    BItem *p = items + base + excl;
    if (nseg <= 8)
        for (uint32_t k = 0; k < nseg; ++k) {
            BItem it;
            it.u = ug;
            it.cnt = min(d - k * kItemEntries, kItemEntries) | (uint32_t)g << 16;
            it.start = s + (int64_t)k * kItemEntries;
            p[k] = it;
        }
    unsigned big = __ballot_sync(0xFFFFFFFFu, nseg > 8);
    while (big) {
        const int l = __ffs(big) - 1;
        big &= big - 1;
        const uint32_t uu = __shfl_sync(0xFFFFFFFFu, ug, l), c = __shfl_sync(0xFFFFFFFFu, nseg, l);
        const uint32_t x = __shfl_sync(0xFFFFFFFFu, excl, l), dd = __shfl_sync(0xFFFFFFFFu, d, l);
        const int64_t ss = __shfl_sync(0xFFFFFFFFu, s, l);
        const int gg = __shfl_sync(0xFFFFFFFFu, g, l);
        for (uint32_t k = g5_lane(); k < c; k += 32) {
            BItem it;
            it.u = uu;
            it.cnt = min(dd - k * kItemEntries, kItemEntries) | (uint32_t)gg << 16;
            it.start = ss + (int64_t)k * kItemEntries;
            items[base + x + k] = it;
        }
    }
}

// Top-down over a list of items (vertices in no top-down root's frontier are
// passed over): 32 items per warp step, one, or a part of one, as many as it
// takes to give every warp some.
template <bool CLAIM>
__device__ __forceinline__ void bexp_items(const PArgs &a, PShared &sh, const BItem *items, uint64_t nitems, BItem *out,
                                           unsigned long long *alloc)
{
    const int lane = g5_lane();
    TdScratch &ws = sh.w[threadIdx.x >> 5].td;
    const uint64_t gw = (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x, nw = (uint64_t)gridDim.x * kSW;
    const uint32_t ipw = items_per_step(nitems, (uint32_t)nw);
    uint32_t split_shift = 0;
    while (split_shift < 3 && (nitems << (split_shift + 1)) <= nw) ++split_shift;
    const uint64_t units = ipw == 1 ? nitems << split_shift : item_steps(nitems, ipw);
    for (uint64_t t = gw; t < units; t += nw) {
        // a step's items lie apart, so that each has its share of the hubs',
        // which come first (taken in order, 32 a step: scale 22 1892 us a batch
        // and 1760 so, the eight mixed graphs 1059 and 890)
        const uint64_t i = ipw == 1 ? (t >> split_shift) + lane : t + lane * units;
        uint32_t cnt = 0, u = 0;
        int g = 0;
        int64_t s = 0;
        uint64_t f = 0;
        if ((uint32_t)lane < ipw && i < nitems) {
            const uint4 raw = __ldcg(reinterpret_cast<const uint4 *>(items + i));
            u = raw.x;
            g = (int)(raw.y >> 16);
            cnt = raw.y & 0xFFFFu;
            s = (int64_t)(raw.z | (uint64_t)raw.w << 32);
            const uint32_t part = kItemEntries >> split_shift;
            const uint32_t at = (uint32_t)(t & ((1u << split_shift) - 1)) * part;
            s += at;
            cnt = cnt > at ? min(cnt - at, part) : 0u;
            if (!sh.td_mask[g]) cnt = 0;
            if (cnt) f = a.b.front[u] & sh.td_mask[g];
            if (!f) cnt = 0;
        }
        uint32_t total;
        const uint32_t excl = warp_excl_u32(cnt, total);
        __syncwarp();
        ws.end[lane] = excl + cnt;
        // the parent's original id, which is what the parents hold
        ws.u[lane] = cnt ? __ldg(sh.gd[g].orig + (u - sh.gd[g].vbase)) : 0u;
        ws.base[lane] = s - (int64_t)excl;
        ws.front[lane] = f;
        ws.g[lane] = (uint8_t)g;
        __syncwarp();
        for (uint32_t e0 = 0; e0 < total; e0 += 32) {
            const uint32_t x = e0 + lane;
            bool claimed = false;
            uint32_t vl = 0, dv = 0;
            int64_t vs = 0;
            int gv = 0;
            if (x < total) {
                int lo = 0;
                if (ipw > 1) {
                    int hi = 31;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (ws.end[mid] <= x) lo = mid + 1;
                        else hi = mid;
                    }
                }
                gv = ws.g[lo];
                const GraphDesc &d = sh.gd[gv];
                vl = __ldg(d.col + (ws.base[lo] + (int64_t)x));
                const uint64_t vg = d.vbase + vl;
                const uint64_t seen = a.b.vis[vg];
                const uint32_t vo = __ldg(d.orig + vl);
                if (CLAIM) {
                    vs = __ldg(d.row_off + vl);
                    dv = __ldg(a.b.deg + vg);
                }
                const uint64_t nb = ws.front[lo] & ~seen;
                if (nb) {
                    const uint32_t ul = ws.u[lo];
                    uint32_t *pv = a.b.pred + d.pred_base + (uint64_t)vo * d.nroots;
                    if (CLAIM) {
                        for (uint64_t y = nb; y; y &= y - 1) atomicMin(pv + (__ffsll((long long)y) - 1), ul);
                    } else {
                        // the slots are read first: most hold a smaller parent
                        // already; four at a time (scale 20 630 -> 619 us a
                        // batch, 22 1744 -> 1725, against one after another)
                        for (uint64_t y = nb; y;) {
                            uint32_t r[4], x[4];
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                r[q] = y ? (uint32_t)(__ffsll((long long)y) - 1) : 64u;
                                y &= y - 1;
                            }
#pragma unroll
                            for (int q = 0; q < 4; ++q) x[q] = r[q] < 64 ? pv[r[q]] : 0u;
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                if (x[q] > ul) atomicMin(pv + r[q], ul);
                        }
                    }
                    if (CLAIM) claimed = atomicOr((unsigned long long *)&a.b.next[vg], (unsigned long long)nb) == 0;
                    else if (nb & ~a.b.next[vg]) atomicOr((unsigned long long *)&a.b.next[vg], (unsigned long long)nb);
                }
            }
            if (CLAIM && __any_sync(0xFFFFFFFFu, claimed)) {
                const uint32_t nseg = claimed ? (dv + kItemEntries - 1) / kItemEntries : 0u;
                uint32_t tot;
                const uint32_t at = warp_excl_u32(nseg, tot);
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(alloc, (unsigned long long)tot);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                put_rows(out, a.claimed_cap, base, at, (uint32_t)(sh.gd[gv].vbase + vl), gv, vs, dv, nseg);
            }
        }
    }
}

// visited |= next, next -> front, and the sums of the next frontier per graph.
// A unit idle this level and the last is passed over.
__device__ __forceinline__ void bcommit(const PArgs &a, PShared &sh, GraphSum *sums, unsigned long long *rsums)
{
    constexpr int kK = 8;
    const int lane = g5_lane();
    const uint32_t rounds = a.unit / 32;
    const uint64_t units = a.b.ntot / a.unit, nw = (uint64_t)gridDim.x * kSW;
    int cur = -1;
    uint32_t nf = 0;
    uint64_t mf = 0, am = 0, r0 = 0, r1 = 0;
    auto flush = [&]() {
        // (lane l has summed up roots l and l + 32)
        if (r0) atomicAdd(&sh.rs[cur][lane], (uint32_t)((r0 + kRootEntries - 1) / kRootEntries));
        if (r1) atomicAdd(&sh.rs[cur][lane + 32], (uint32_t)((r1 + kRootEntries - 1) / kRootEntries));
        r0 = r1 = 0;
        if (cur >= 0 && __any_sync(0xFFFFFFFFu, nf != 0)) {
            nf = __reduce_add_sync(0xFFFFFFFFu, nf);
            mf = warp_add_u51(mf);
            const uint32_t lo = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)am), hi = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(am >> 32));
            if (lane == 0) {
                atomicAdd(&sh.nf[cur], (unsigned long long)nf);
                atomicAdd(&sh.mf[cur], (unsigned long long)mf);
                atomicOr(&sh.am[cur], (unsigned long long)hi << 32 | lo);
            }
        }
        nf = 0;
        mf = am = 0;
    };
    for (uint64_t t = (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; t < units; t += nw) {
        const uint64_t v0 = t * a.unit;
        const int g = a.b.chunk_graph[v0 / kChunk];
        if (g != cur) {
            flush();
            cur = g;
        }
        const bool was = a.live[t] != 0;
        uint64_t nx[kK], all = 0;
#pragma unroll
        for (int k = 0; k < kK; ++k) {
            nx[k] = k < (int)rounds ? a.b.next[v0 + 32 * k + lane] : 0ull;
            all |= nx[k];
        }
        const bool now = __any_sync(0xFFFFFFFFu, all != 0);
        if (!now && !was) continue;
        if (lane == 0 && now != was) a.live[t] = now;
        uint64_t vs[kK];
        uint32_t dg[kK];
#pragma unroll
        for (int k = 0; k < kK; ++k) {
            vs[k] = nx[k] ? a.b.vis[v0 + 32 * k + lane] : 0ull;
            dg[k] = nx[k] ? __ldg(a.b.deg + v0 + 32 * k + lane) : 0u;
        }
        am |= all;
#pragma unroll
        for (int k = 0; k < kK; ++k) {
            if (k < (int)rounds) a.b.front[v0 + 32 * k + lane] = nx[k];
            if (nx[k]) {
                a.b.vis[v0 + 32 * k + lane] = vs[k] | nx[k];
                a.b.next[v0 + 32 * k + lane] = 0;
                ++nf;
                mf += dg[k];
            }
        }
        if (sh.gd[g].dir != TD || sh.gd[g].nnz < kSplitEntries) continue;
        // each root's entries, for the split of a first bottom-up level
#pragma unroll
        for (int k = 0; k < kK; ++k) {
            for (unsigned on = __ballot_sync(0xFFFFFFFFu, nx[k] != 0); on; on &= on - 1) {
                const int l = __ffs(on) - 1;
                const uint64_t x = __shfl_sync(0xFFFFFFFFu, nx[k], l);
                const uint32_t d = __shfl_sync(0xFFFFFFFFu, dg[k], l);
                if ((x >> lane) & 1u) r0 += d;
                if ((x >> (lane + 32)) & 1u) r1 += d;
            }
        }
    }
    flush();
    __syncthreads();
    for (int g = threadIdx.x; g < a.b.ngraphs; g += kSB) {
        if (sh.nf[g]) {
            atomicAdd(&sums[g].nf, sh.nf[g]);
            atomicAdd(&sums[g].mf, sh.mf[g]);
            atomicOr(&sums[g].amask, sh.am[g]);
        }
        sh.nf[g] = sh.mf[g] = sh.am[g] = 0;
    }
    for (int i = threadIdx.x; i < 64 * a.b.ngraphs; i += kSB) {
        const uint32_t x = (&sh.rs[0][0])[i];
        if (x) atomicAdd(&rsums[i], (unsigned long long)x);
        (&sh.rs[0][0])[i] = 0;
    }
    // (pmeet's barrier and fence follow)
}

// The items of the frontiers of the graphs marked in build_g.
__device__ __forceinline__ void bbuild(const PArgs &a, PShared &sh, unsigned long long *alloc)
{
    const int lane = g5_lane();
    const uint64_t units = a.b.ntot / a.unit, nw = (uint64_t)gridDim.x * kSW;
    for (uint64_t t = (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; t < units; t += nw) {
        if (!a.live[t]) continue;
        const uint64_t v0 = t * a.unit;
        const int g = a.b.chunk_graph[v0 / kChunk];
        if (!sh.build_g[g]) continue;
        for (uint32_t k = 0; k < a.unit; k += 32) {
            const uint64_t vg = v0 + k + lane;
            const bool on = (a.b.front[vg] & sh.td_mask[g]) != 0;
            if (!__any_sync(0xFFFFFFFFu, on)) continue;
            const uint32_t d = on ? __ldg(a.b.deg + vg) : 0u, nseg = (d + kItemEntries - 1) / kItemEntries;
            const int64_t s = on ? __ldg(sh.gd[g].row_off + (vg - sh.gd[g].vbase)) : 0;
            uint32_t tot;
            const uint32_t at = warp_excl_u32(nseg, tot);
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(alloc, (unsigned long long)tot);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            put_rows(a.built, ~0ull, base, at, (uint32_t)vg, g, s, d, nseg);
        }
    }
}

__global__ void __launch_bounds__(kSB, 1) k_bsearch(const __grid_constant__ PArgs a)
{
    extern __shared__ __align__(16) unsigned char s_batch[];
    PShared &sh = *reinterpret_cast<PShared *>(s_batch);
    const uint64_t tid = (uint64_t)blockIdx.x * kSB + threadIdx.x, nthr = (uint64_t)gridDim.x * kSB;
    const int ng = a.b.ngraphs, lane = g5_lane();
    // prologue: empty words, no parents, the graphs' descriptors
    for (uint64_t i = tid; i < 3 * a.b.ntot / 2; i += nthr)
        reinterpret_cast<ulonglong2 *>(a.b.vis)[i] = make_ulonglong2(0, 0);
    for (uint64_t i = tid; i < a.b.ntot / a.unit; i += nthr) a.live[i] = 0;
    const uint64_t head = min(a.npred, (uint64_t)((16 - ((uintptr_t)a.b.pred & 15)) & 15) / 4);
    const uint64_t vecs = (a.npred - head) / 4;
    for (uint64_t i = tid; i < vecs; i += nthr)
        reinterpret_cast<uint4 *>(a.b.pred + head)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    if (tid < head) a.b.pred[tid] = ~0u;
    if (tid < a.npred - head - 4 * vecs) a.b.pred[head + 4 * vecs + tid] = ~0u;
    for (uint32_t i = threadIdx.x; i < ng * sizeof(GraphDesc) / 8; i += kSB)
        reinterpret_cast<uint64_t *>(sh.gd)[i] = __ldcg(reinterpret_cast<const unsigned long long *>(a.gd) + i);
    for (int g = threadIdx.x; g < ng; g += kSB) sh.nf[g] = sh.mf[g] = sh.am[g] = 0;
    for (int i = threadIdx.x; i < 64 * ng; i += kSB) (&sh.rs[0][0])[i] = 0;
    for (uint64_t i = tid; i < (uint64_t)kRing * 64 * ng; i += nthr) a.rsums[i] = 0;
    if (threadIdx.x == 0) sh.stop = 0;
    pmeet(a, sh, &a.meets[0].arrive[0]);
    // the roots: into next, their own parents
    for (int g = blockIdx.x; g < ng; g += gridDim.x) {
        const GraphDesc &d = sh.gd[g];
        for (int r = threadIdx.x; r < d.nroots; r += kSB) {
            const int64_t root = a.b.roots[a.b.root_off[g] + r];
            atomicOr((unsigned long long *)&a.b.next[d.vbase + d.perm[root]], 1ull << r);
            a.b.pred[d.pred_base + (uint64_t)root * d.nroots + r] = (uint32_t)root;
        }
    }
    for (int g = threadIdx.x; g < ng; g += kSB) {
        sh.gd[g].dir = TD;
        sh.gd[g].mu = (uint64_t)sh.gd[g].nnz;
    }
    pmeet(a, sh, &a.meets[0].arrive[1]);
    uint32_t err = 0;
    bool claim = false;  // the level before claimed: its items are those of the top-down graphs
    int32_t L = -1;
    for (;; ++L) {
        // level L: expand its frontier (none before level 0), then commit
        LevelMeet *cur = a.meets + (L + kRing) % kRing, *nxt = a.meets + (L + 1) % kRing;
        GraphSum *sums = a.sums + (uint64_t)((L + 1) % kRing) * ng;
        unsigned long long *rsums = a.rsums + (uint64_t)((L + 1) % kRing) * ng * 64;
        if (L >= 0) {
            // (the records of the level after next)
            if (tid < sizeof(LevelMeet) / 8)
                reinterpret_cast<unsigned long long *>(a.meets + (L + 2) % kRing)[tid] = 0;
            for (uint64_t i = tid; i < (uint64_t)ng * sizeof(GraphSum) / 8; i += nthr)
                reinterpret_cast<unsigned long long *>(a.sums + (uint64_t)((L + 2) % kRing) * ng)[i] = 0;
            for (uint64_t i = tid; i < (uint64_t)ng * 64; i += nthr)
                a.rsums[(uint64_t)((L + 2) % kRing) * ng * 64 + i] = 0;
            const uint64_t nclaimed = claim ? __ldcg(&cur->alloc) : 0;
            if (sh.build) {
                bbuild(a, sh, &cur->built);
                pmeet(a, sh, &cur->arrive[2]);
                if (sh.stop) break;
            }
            const uint64_t nbuilt = sh.build ? __ldcg(&cur->built) : 0;
            const bool now = sh.td_entries <= kClaimMax;
            if (sh.dirs & 1u) {
                BItem *out = a.claimed[(L + 1) & 1];
                if (now) {
                    bexp_items<true>(a, sh, a.claimed[L & 1], nclaimed, out, &nxt->alloc);
                    bexp_items<true>(a, sh, a.built, nbuilt, out, &nxt->alloc);
                } else {
                    bexp_items<false>(a, sh, a.claimed[L & 1], nclaimed, nullptr, nullptr);
                    bexp_items<false>(a, sh, a.built, nbuilt, nullptr, nullptr);
                }
            }
            if (sh.dirs & 2u) {
                uint64_t ex = 0;
                const uint64_t gw = (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x, nw = (uint64_t)gridDim.x * kSW;
                __syncwarp();
                bexp_bu<true>(a.b, sh.gd, sh.w[threadIdx.x >> 5].bu, gw, nw, a.vps_shift, LongRows{a.longs, &cur->longs, &sh.steps}, ex);
                pmeet(a, sh, &cur->arrive[4]);
                if (sh.stop) break;
                bexp_long(a.b, sh.gd, a.longs, __ldcg(&cur->longs), gw, nw);
            }
            claim = now;
            pmeet(a, sh, &nxt->arrive[0]);
            if (sh.stop) break;
        }
        bcommit(a, sh, sums, rsums);
        pmeet(a, sh, L < 0 ? &a.meets[0].arrive[3] : &nxt->arrive[1]);
        if (sh.stop) break;
        // decide, alike in every block: Beamer's switch on the union frontier of
        // the graph's roots
        if (threadIdx.x == 0) {
            sh.active = sh.td_entries = 0;
            sh.dirs = sh.build = sh.splits = 0;
            sh.steps = kSW;
        }
        __syncthreads();
        const bool fits = claim && L >= 0 && __ldcg(&nxt->alloc) <= a.claimed_cap;
        for (int g = threadIdx.x; g < ng; g += kSB) {
            GraphDesc &d = sh.gd[g];
            const uint64_t tn = __ldcg(&sums[g].nf), tm = __ldcg(&sums[g].mf);
            const uint64_t mu = d.mu >= tm ? d.mu - tm : 0;
            const int was = d.dir;
            int nd = was;
            if (L >= 0) {
                if (was == TD) {
                    // a frontier large enough, too, to pay for a sweep over all
                    // of the graph's vertices
                    if (above_quotient(tm, mu, a.b.alpha) && tm > (uint64_t)d.n / kBuMinFrac) nd = BU;
                } else if (tn < d.nf && below_quotient(tn, (uint64_t)d.n, a.b.beta)) {
                    nd = TD;
                }
            }
            d.mu = mu;
            d.dir = nd;
            d.nf = tn;
            d.mf = tm;
            d.amask = __ldcg(&sums[g].amask) & d.mask;
            sh.td_mask[g] = nd == TD ? ~0ull : 0ull;
            sh.split[g] = nd == BU && was == TD && d.nnz >= kSplitEntries;
            if (sh.split[g]) sh.splits = 1;
            const bool build = nd == TD && tn && !(fits && was == TD);
            sh.build_g[g] = build;
            if (tn) {
                atomicAdd(&sh.active, (unsigned long long)tn);
                atomicOr(&sh.dirs, nd == TD ? 1u : 2u);
                if (nd == TD) atomicAdd(&sh.td_entries, (unsigned long long)tm);
                if (build) atomicOr(&sh.build, 1u);
            }
        }
        __syncthreads();
        for (int g = threadIdx.x >> 5; sh.splits && g < ng; g += kSW) {
            if (!sh.split[g]) continue;
            const uint64_t r0 = __ldcg(rsums + 64 * g + lane), r1 = __ldcg(rsums + 64 * g + 32 + lane);
            const uint64_t all = (uint64_t)sh.gd[g].nnz / kRootEntries;
            uint64_t most = all / kFewShare, few;
            for (;; most /= 2) {
                few = warp_sum_u64((r0 < most ? r0 : 0) + (r1 < most ? r1 : 0));
                if (few <= all / kFewTotal) break;
            }
            const uint64_t mask = __ballot_sync(0xFFFFFFFFu, r0 && r0 < most) |
                                  (uint64_t)__ballot_sync(0xFFFFFFFFu, r1 && r1 < most) << 32;
            if (lane == 0 && mask) {
                sh.td_mask[g] = mask;
                sh.gd[g].amask &= ~mask;
                atomicAdd(&sh.td_entries, (unsigned long long)few * kRootEntries);
                atomicOr(&sh.dirs, 1u);
                if (!fits) {
                    sh.build_g[g] = 1;
                    atomicOr(&sh.build, 1u);
                }
            }
        }
        if (sh.splits) __syncthreads();
        claim = fits;
        if (sh.active == 0) break;
        if (L + 2 >= kMaxLevels) {
            err = 8u;
            break;
        }
    }
    if (tid == 0) {
        a.out->level = L + 1;
        a.out->err = err | (sh.stop ? 16u : 0u);
        a.out->active = sh.active;
    }
}

// Continuous batching: roots admitted into free slots (bit r of their
// graph) join the next level as its frontier; retired roots' visited bits are
// cleared so the slot can be reused.
struct Admit {
    int32_t graph;
    int32_t slot;
    int64_t root;
};

__global__ void k_sadmit(BArgs a, const Admit *adm, int nadm)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nadm; i += gridDim.x * blockDim.x) {
        const Admit x = adm[i];
        const GraphDesc &d = a.gd[x.graph];
        atomicOr((unsigned long long *)&a.next[d.vbase + d.perm[x.root]], 1ull << x.slot);
        a.pred[d.pred_base + (uint64_t)x.root * d.nroots + x.slot] = (uint32_t)x.root;
    }
}

__global__ void k_sclear(BArgs a, const uint64_t *clear_mask)
{
    // a retired slot's visited vertices get their parent entry back to
    // 0xFFFFFFFF: every entry of a free slot is unvisited again
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < a.ntot;
         v += (uint64_t)gridDim.x * blockDim.x) {
        const int g = graph_of(a, v);
        const uint64_t m = clear_mask[g];
        if (m) {
            const uint64_t x = a.vis[v];
            if (x & m) {
                a.vis[v] = x & ~m;
                const GraphDesc &d = a.gd[g];
                uint32_t *p = a.pred + d.pred_base + (uint64_t)d.orig[v - d.vbase] * d.nroots;
                uint64_t y = x & m;
                while (y) {
                    const int r = __ffsll((long long)y) - 1;
                    y &= y - 1;
                    p[r] = 0xFFFFFFFFu;
                }
            }
        }
    }
}

// One root's parents out of the vertex-major array: dst[v] = pred[v * R + r].
__global__ void k_gather_root(const uint32_t *pred, uint32_t R, uint32_t r, int64_t n, uint32_t *dst)
{
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        dst[v] = pred[(uint64_t)v * R + r];
}

__global__ void k_bdeg(const GraphDesc *gd, const uint8_t *chunk_graph, uint64_t ntot, uint32_t *deg,
                       uint32_t *iso)
{
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < ntot;
         v += (uint64_t)gridDim.x * blockDim.x) {
        const GraphDesc &d = gd[chunk_graph[v / kChunk]];
        const int64_t vl = (int64_t)(v - d.vbase);
        const uint32_t dv = vl < d.n ? (uint32_t)(d.row_off[vl + 1] - d.row_off[vl]) : 0u;
        deg[v] = dv;
        const unsigned z = __ballot_sync(0xFFFFFFFFu, dv == 0u);
        if ((threadIdx.x & 31) == 0) iso[v >> 5] = z;
    }
}

// ---- degree-ordered copy of a graph ----------------------------------------------------

__global__ void k_rl_deg(const int64_t *row_off, int64_t n, uint32_t *deg, uint32_t *ids)
{
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        deg[v] = (uint32_t)(row_off[v + 1] - row_off[v]);
        ids[v] = (uint32_t)v;
    }
}

// perm[orig[p]] = p; row2[p] = degree of new vertex p (scanned into offsets)
__global__ void k_rl_perm(const uint32_t *orig, const uint32_t *deg_sorted, int64_t n, uint32_t *perm, int64_t *row2)
{
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p <= n; p += (int64_t)gridDim.x * blockDim.x) {
        if (p < n) {
            perm[orig[p]] = (uint32_t)p;
            row2[p] = deg_sorted[p];
        } else {
            row2[n] = 0;
        }
    }
}

// The bottom-up sweep's record of a vertex with edges: original id, new id, where
// its row starts in the copy (low 32 bits; 8 more in the last word) and its
// degree (24 bits; all ones: take it from the row offsets).
// One 16-byte load instead of the chain list, permutation and row start and
// degree by original id: us per batch, before and after, scale 24 6515 and 6352,
// scale 22 1914 and 1871, the eight mixed graphs 1063 and 1049 (scale 18, 16
// roots 231 and 235).
__global__ void k_rl_list(const uint32_t *ids, int64_t count, const uint32_t *perm, const int64_t *row2, uint4 *list)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t o = ids[i], p = perm[o];
        const uint64_t s = (uint64_t)row2[p], d = (uint64_t)row2[p + 1] - s;
        list[i] = make_uint4(o, p, (uint32_t)s,
                             (uint32_t)(s >> 32) << kListDegBits | (uint32_t)(d < kListDeg ? d : kListDeg));
    }
}

// one warp per new row: the original row, neighbours renamed, order kept
__global__ void k_rl_cols(const int64_t *row_off, const uint32_t *col, const uint32_t *orig, const uint32_t *perm,
                          const int64_t *row2, int64_t n, uint32_t *col2)
{
    const int lane = g5_lane();
    for (int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < n;
         p += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const uint32_t o = orig[p];
        const int64_t s = row_off[o], len = row_off[o + 1] - s, d0 = row2[p];
        for (int64_t k = lane; k < len; k += 32) col2[d0 + k] = perm[col[s + k]];
    }
}

}  // namespace

struct g5_batch {
    std::vector<g5_graph *> graphs;
    std::vector<GraphDesc> hgd;
    BArgs args;
    cudaStream_t stream = nullptr;
    GraphDesc *gd = nullptr;
    uint8_t *chunk_graph = nullptr;
    uint8_t *step_graph = nullptr;  // graph of each bottom-up warp step
    uint32_t *deg = nullptr;
    uint32_t *iso = nullptr;
    uint64_t *words = nullptr;  // vis | front | next
    uint32_t *queue = nullptr;
    uint64_t *qoff = nullptr;
    int64_t *qbase = nullptr;
    uint32_t *tile_start = nullptr;
    uint64_t *chunks = nullptr;
    BState *st = nullptr;
    int64_t *roots = nullptr;
    int32_t *root_off = nullptr;
    uint64_t *level_log = nullptr;
    int64_t *h_roots = nullptr;
    int32_t *h_root_off = nullptr;
    BState *h_st = nullptr;
    uint32_t *bound_pred = nullptr;  // pred pointer the graph was built for
    void *adm_dev = nullptr;          // serving: admissions + retire masks
    void *adm_host = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaGraph_t graph = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    std::vector<void *> owned;        // degree-ordered graph copies
    // the one-launch form (g5_batch_run; made on its first call)
    void *scratch = nullptr;          // queue arrays of the level graph, or built items
    size_t scratch_bytes = 0;
    BItem *built = nullptr;           // built items that the scratch has no room for
    int pgrid = 0;                    // its blocks (0: not made, -1: the device cannot hold it)
    PArgs pargs;
    BItem *claimed = nullptr;
    uint8_t *live = nullptr;
    unsigned long long *rsums = nullptr;
    LongItem *longs = nullptr;
    char *stage = nullptr, *h_stage = nullptr;  // descriptors, roots and cleared records of a run
    size_t stage_bytes = 0, roots_at = 0, off_at = 0, zero_at = 0;
};

namespace {

void enqueue_batch(g5_batch *b, const BArgs &a, cudaStream_t s, bool body, std::vector<cudaEvent_t> *ev = nullptr)
{
    auto mark = [&]() {
        if (ev) {
            cudaEvent_t e;
            cudaEventCreate(&e);
            cudaEventRecord(e, s);
            ev->push_back(e);
        }
    };
    if (!body) {
        cudaMemsetAsync(b->words, 0, sizeof(uint64_t) * 3 * a.ntot, s);
        cudaMemsetAsync(a.chunk_live, 0, a.nchunks, s);
        k_binit<<<std::max(1, a.ngraphs), kB, 0, s>>>(a);
        return;
    }
    mark();
    k_bcount<<<g5::grid_for(8), kB, 0, s>>>(a);
    mark();
    k_bscan<<<1, 1024, 0, s>>>(a);
    mark();
    k_bwrite<<<g5::grid_for(4), kB, 0, s>>>(a);
    mark();
    k_btd<<<g5::grid_for(8), kB, 0, s>>>(a);
    k_bbu<<<g5::grid_for(4), kB, 0, s>>>(a);
    mark();
    mark();
}

g5_status build_batch_graph(g5_batch *b)
{
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
    cudaStream_t s = b->stream;
    cudaGraph_t pro = nullptr;
    G5_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    enqueue_batch(b, b->args, s, false);
    G5_CUDA(cudaStreamEndCapture(s, &pro));
    cudaGraph_t g = nullptr;
    G5_CUDA(cudaGraphCreate(&g, 0));
    cudaGraphNode_t pn;
    G5_CUDA(cudaGraphAddChildGraphNode(&pn, g, nullptr, 0, pro));
    cudaGraphDestroy(pro);
    cudaGraphConditionalHandle h;
    G5_CUDA(cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t cn;
    G5_CUDA(cudaGraphAddNode(&cn, g, &pn, nullptr, 1, &cp));
    BArgs a = b->args;
    a.cond = h;
    a.use_cond = 1;
    G5_CUDA(cudaStreamBeginCaptureToGraph(s, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                          cudaStreamCaptureModeThreadLocal));
    enqueue_batch(b, a, s, true);
    cudaGraph_t body = nullptr;
    G5_CUDA(cudaStreamEndCapture(s, &body));
    G5_CUDA(cudaGraphInstantiate(&b->exec, g, 0));
    b->graph = g;
    return G5_OK;
}

// Bytes of the level graph's queue arrays.
size_t queue_bytes(const BArgs &a)
{
    return sizeof(uint64_t) * (2 * a.ntot + 2) + sizeof(uint32_t) * (a.ntot + a.max_tiles);
}

// Calls f(pointer, bytes) for every device buffer of a workspace but its graph
// copies and the one-launch form's: one list of what is allocated, freed and
// charged (from ngraphs, ntot, nchunks, nsteps and max_tiles of its arguments).
template <typename F>
void each_buffer(g5_batch *b, F f)
{
    const BArgs &a = b->args;
    const size_t ng = (size_t)a.ngraphs;
    f(b->gd, sizeof(GraphDesc) * ng);
    f(b->step_graph, a.nsteps + 1);
    f(b->chunk_graph, (size_t)a.nchunks);
    f(b->deg, sizeof(uint32_t) * a.ntot);
    f(b->iso, sizeof(uint32_t) * (a.ntot / 32));
    f(b->words, sizeof(uint64_t) * 3 * a.ntot);
    f(b->scratch, queue_bytes(a));
    f(b->chunks, sizeof(uint64_t) * 2 * a.nchunks + a.nchunks);
    f(b->st, sizeof(BState));
    f(b->roots, sizeof(int64_t) * 64 * ng);
    f(b->root_off, sizeof(int32_t) * (ng + 1));
    f(b->level_log, sizeof(uint64_t) * kMaxLevels);
}

// Gives back what the one-launch form holds.
void drop_one_launch(g5_batch *b)
{
    cudaFree(b->claimed);
    cudaFree(b->built);
    cudaFree(b->live);
    cudaFree(b->rsums);
    cudaFree(b->longs);
    cudaFree(b->stage);
    cudaFreeHost(b->h_stage);
    b->claimed = b->built = nullptr;
    b->live = nullptr;
    b->rsums = nullptr;
    b->longs = nullptr;
    b->stage = b->h_stage = nullptr;
    b->pgrid = 0;
}

void free_batch(g5_batch *b)
{
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    each_buffer(b, [](auto *&p, size_t) { cudaFree(p); });
    drop_one_launch(b);
    cudaFree(b->adm_dev);
    cudaFreeHost(b->adm_host);
    cudaFreeHost(b->h_roots);
    cudaFreeHost(b->h_root_off);
    cudaFreeHost(b->h_st);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    for (void *p : b->owned) cudaFree(p);
    b->owned.clear();
    if (b->stream) cudaStreamDestroy(b->stream);
}

struct HasEdges {
    const uint32_t *deg;
    __device__ bool operator()(const uint32_t &v) const { return deg[v] > 0; }
};

// Degree-ordered copy of g on b's stream: new ids by descending degree (ties
// by original id), rows in new-id order, each row's neighbours renamed but in
// their original order.
g5_status build_relabel(g5_batch *b, const g5_graph *g, GraphDesc &d)
{
    const int64_t n = g->n, nnz = g->nnz;
    cudaStream_t s = b->stream;
    auto alloc = [&](void **p, size_t bytes) -> bool {
        if (cudaMalloc(p, bytes ? bytes : 16) != cudaSuccess) return false;
        b->owned.push_back(*p);
        return true;
    };
    uint32_t *orig = nullptr, *perm = nullptr, *col2 = nullptr;
    int64_t *row2 = nullptr;
    if (!alloc((void **)&orig, sizeof(uint32_t) * n) || !alloc((void **)&perm, sizeof(uint32_t) * n) ||
        !alloc((void **)&row2, sizeof(int64_t) * (n + 1)) || !alloc((void **)&col2, sizeof(uint32_t) * nnz))
        return G5_ERR_OOM;
    if (nnz >> (32 + 32 - kListDegBits)) return G5_ERR_INVALID_ARG;  // (row starts take 40 bits)
    d.orig = orig;
    d.perm = perm;
    d.row_off = row2;
    d.col = col2;
    if (n == 0) {
        G5_CUDA(cudaMemsetAsync(row2, 0, sizeof(int64_t), s));
        return G5_OK;
    }
    g5::DevBuf<uint32_t> deg, ids, deg_sorted;
    if (deg.alloc(n) != G5_OK || ids.alloc(n) != G5_OK || deg_sorted.alloc(n) != G5_OK) return G5_ERR_OOM;
    const int blocks = g5::grid_for(8);
    k_rl_deg<<<blocks, 256, 0, s>>>(g->row_off, n, deg.p, ids.p);
    size_t t1 = 0, t2 = 0;
    G5_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, t1, deg.p, deg_sorted.p, ids.p, orig, n, 0, 32, s));
    G5_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, t2, row2, row2, n + 1, s));
    g5::DevBuf<uint8_t> tmp;
    if (tmp.alloc(std::max(t1, t2)) != G5_OK) return G5_ERR_OOM;
    G5_CUDA(cub::DeviceRadixSort::SortPairsDescending(tmp.p, t1, deg.p, deg_sorted.p, ids.p, orig, n, 0, 32, s));
    k_rl_perm<<<blocks, 256, 0, s>>>(orig, deg_sorted.p, n, perm, row2);
    G5_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, t2, row2, row2, n + 1, s));
    k_rl_cols<<<blocks, 256, 0, s>>>(g->row_off, g->col, orig, perm, row2, n, col2);
    // the bottom-up sweep's vertex list: original ids with edges, ascending
    // (ids still holds 0..n-1: the sort wrote its values elsewhere)
    g5::DevBuf<uint32_t> &with = deg_sorted;  // (no longer needed)
    g5::DevBuf<int64_t> nsel;
    if (nsel.alloc(1) != G5_OK) return G5_ERR_OOM;
    size_t t3 = 0;
    const HasEdges pred{deg.p};
    G5_CUDA(cub::DeviceSelect::If(nullptr, t3, ids.p, with.p, nsel.p, (int64_t)n, pred, s));
    g5::DevBuf<uint8_t> tmp3;
    if (tmp3.alloc(t3) != G5_OK) return G5_ERR_OOM;
    G5_CUDA(cub::DeviceSelect::If(tmp3.p, t3, ids.p, with.p, nsel.p, (int64_t)n, pred, s));
    int64_t nl = 0;
    G5_CUDA(cudaMemcpyAsync(&nl, nsel.p, sizeof nl, cudaMemcpyDeviceToHost, s));
    G5_CUDA(cudaStreamSynchronize(s));
    uint4 *blist = nullptr;
    if (!alloc((void **)&blist, sizeof(uint4) * (size_t)nl)) return G5_ERR_OOM;
    k_rl_list<<<blocks, 256, 0, s>>>(with.p, nl, perm, row2, blist);
    G5_CUDA(cudaStreamSynchronize(s));  // (the temporary arrays go)
    d.blist = blist;
    d.nblist = (uint64_t)nl;
    return G5_OK;
}

}  // namespace

namespace {

// Sets up the one-launch form: its buffers, grid and arguments; pgrid = -1 if
// the device cannot hold a block per SM of it.
g5_status plan_one_launch(g5_batch *b)
{
    const int ng = (int)b->graphs.size();
    const uint64_t vb = b->args.ntot;
    uint64_t nnz = 0;
    for (const g5_graph *g : b->graphs) nnz += (uint64_t)g->nnz;
    int per_sm = 0;
    cudaError_t e = cudaFuncSetAttribute(k_bsearch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PShared));
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bsearch, kSB, sizeof(PShared));
    if (e != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        if (e == cudaErrorMemoryAllocation) return G5_ERR_OOM;
        b->pgrid = -1;
        return G5_OK;
    }
    PArgs &a = b->pargs;
    memset(&a, 0, sizeof a);
    a.claimed_cap = std::min<uint64_t>(std::min<uint64_t>(vb, kClaimMax) + nnz / kItemEntries + 1, kClaimedItems);
    auto align16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    b->roots_at = align16(sizeof(GraphDesc) * ng);
    b->off_at = align16(b->roots_at + sizeof(int64_t) * 64 * ng);
    b->zero_at = align16(b->off_at + sizeof(int32_t) * (ng + 1));
    const size_t sums_at = b->zero_at + sizeof(LevelMeet) * kRing, abort_at = sums_at + sizeof(GraphSum) * kRing * ng;
    b->stage_bytes = abort_at + 16;
    // (a failed call leaves what it has made to drop_one_launch)
    G5_CUDA(cudaMalloc(&b->claimed, sizeof(BItem) * 2 * a.claimed_cap));
    // (more than some 85 entries a vertex: the built items outgrow the queue arrays)
    const size_t built_bytes = sizeof(BItem) * (vb + nnz / kItemEntries + 1);
    if (built_bytes > b->scratch_bytes) G5_CUDA(cudaMalloc(&b->built, built_bytes));
    G5_CUDA(cudaMalloc(&b->live, vb / 32));
    G5_CUDA(cudaMalloc(&b->rsums, sizeof(uint64_t) * kRing * 64 * ng));
    // (a row has a piece per kLongRow entries and one for the rest, and more
    // than kLongRow entries to have any)
    G5_CUDA(cudaMalloc(&b->longs, sizeof(LongItem) * (2 * (nnz / kLongRow) + 1)));
    G5_CUDA(cudaMalloc(&b->stage, b->stage_bytes));
    G5_CUDA(cudaMallocHost(&b->h_stage, b->stage_bytes));
    memset(b->h_stage, 0, b->stage_bytes);
    a.gd = reinterpret_cast<const GraphDesc *>(b->stage);
    a.claimed[0] = b->claimed;
    a.claimed[1] = b->claimed + a.claimed_cap;
    a.built = b->built ? b->built : static_cast<BItem *>(b->scratch);
    a.meets = reinterpret_cast<LevelMeet *>(b->stage + b->zero_at);
    a.sums = reinterpret_cast<GraphSum *>(b->stage + sums_at);
    a.abort = reinterpret_cast<unsigned *>(b->stage + abort_at);
    a.live = b->live;
    a.rsums = b->rsums;
    a.longs = b->longs;
    a.out = b->h_st;
    // a block per SM (but those left out), fewer where their warps would have no words or entries
    const uint64_t warps = std::max<uint64_t>(vb / 32, nnz / 64);
    b->pgrid = (int)std::min<uint64_t>((uint64_t)std::min(g5::meeting_sms(), kMaxBlocks), (warps + kSW - 1) / kSW);
    a.unit = 256;
    while (a.unit > 32 && vb / a.unit < (uint64_t)b->pgrid * kSW) a.unit /= 2;
    a.vps_shift = 5;
    while (a.vps_shift > 2 && (b->args.nsteps << (5 - a.vps_shift)) < (uint64_t)b->pgrid * kSW) --a.vps_shift;
    return G5_OK;
}


// A batch workspace over `graphs`; with `share` (a workspace over the same
// graphs), its degree-ordered graph copies are borrowed instead of built, so
// several workspaces on one graph hold one copy (the owner must outlive the
// borrowers).
g5_status batch_create_impl(g5_graph *const *graphs, int ngraphs, const g5_batch *share, g5_batch **out)
{
    if (!graphs || !out || ngraphs < 1 || ngraphs > kMaxGraphs) return G5_ERR_INVALID_ARG;
    *out = nullptr;
    g5_batch *b = new g5_batch();
    auto fail = [&](g5_status s) {
        free_batch(b);
        delete b;
        return s;
    };
    uint64_t vb = 0, nnz_max = 0;
    std::vector<uint8_t> cg;
    for (int i = 0; i < ngraphs; ++i) {
        if (!graphs[i]) return fail(G5_ERR_INVALID_ARG);
        b->graphs.push_back(graphs[i]);
        GraphDesc d;
        memset(&d, 0, sizeof d);
        d.n = graphs[i]->n;
        d.nnz = graphs[i]->nnz;
        d.vbase = vb;
        const uint64_t chunks = ((uint64_t)d.n + kChunk - 1) / kChunk;
        for (uint64_t c = 0; c < chunks; ++c) cg.push_back((uint8_t)i);
        vb += chunks * kChunk;
        nnz_max += (uint64_t)d.nnz;
        b->hgd.push_back(d);
    }
    if (vb >= (1ull << 32)) return fail(G5_ERR_CAPACITY);
    BArgs &a = b->args;
    memset(&a, 0, sizeof a);
    a.ngraphs = ngraphs;
    a.nchunks = (uint32_t)cg.size();
    a.ntot = vb;
    a.max_tiles = nnz_max / kTile + 2 + (uint64_t)ngraphs;
    a.alpha = 14.0;
    a.beta = 24.0;
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(G5_ERR_CUDA);
    cudaEventCreate(&b->ev0);
    cudaEventCreate(&b->ev1);
    for (int i = 0; i < ngraphs; ++i) {
        if (share) {
            if ((int)share->graphs.size() != ngraphs || share->graphs[i] != graphs[i]) return fail(G5_ERR_INVALID_ARG);
            GraphDesc &d = b->hgd[i];
            const GraphDesc &o = share->hgd[i];
            d.row_off = o.row_off;
            d.col = o.col;
            d.orig = o.orig;
            d.perm = o.perm;
            d.blist = o.blist;
            d.nblist = o.nblist;
            continue;
        }
        const g5_status rs = build_relabel(b, graphs[i], b->hgd[i]);
        if (rs != G5_OK) return fail(rs);
    }
    // bottom-up warp steps: each graph's list in 32-entry steps, graphs one
    // after another
    std::vector<uint8_t> sg;
    for (int i = 0; i < ngraphs; ++i) {
        GraphDesc &d = b->hgd[i];
        d.step0 = sg.size();
        const uint64_t steps = (d.nblist + 31) / 32;
        sg.insert(sg.end(), steps, (uint8_t)i);
    }
    a.nsteps = sg.size();
    bool room = true;
    each_buffer(b, [&](auto *&p, size_t bytes) { room = room && cudaMalloc(&p, bytes) == cudaSuccess; });
    if (!room) return fail(G5_ERR_OOM);
    b->scratch_bytes = queue_bytes(a);
    b->qoff = static_cast<uint64_t *>(b->scratch);
    b->qbase = reinterpret_cast<int64_t *>(b->qoff + vb + 2);
    b->queue = reinterpret_cast<uint32_t *>(b->qbase + vb);
    b->tile_start = b->queue + vb;
    if (cudaMallocHost(&b->h_roots, sizeof(int64_t) * 64 * ngraphs) != cudaSuccess ||
        cudaMallocHost(&b->h_root_off, sizeof(int32_t) * (ngraphs + 1)) != cudaSuccess ||
        cudaMallocHost(&b->h_st, sizeof(BState)) != cudaSuccess)
        return fail(G5_ERR_OOM);
    if ((!sg.empty() && cudaMemcpy(b->step_graph, sg.data(), sg.size(), cudaMemcpyHostToDevice) != cudaSuccess) ||
        cudaMemcpy(b->chunk_graph, cg.data(), cg.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(b->gd, b->hgd.data(), sizeof(GraphDesc) * ngraphs, cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(G5_ERR_CUDA);
    a.gd = b->gd;
    a.chunk_graph = b->chunk_graph;
    a.deg = b->deg;
    a.iso = b->iso;
    a.vis = b->words;
    a.front = b->words + vb;
    a.next = b->words + 2 * vb;
    a.queue = b->queue;
    a.qoff = b->qoff;
    a.qbase = b->qbase;
    a.tile_start = b->tile_start;
    a.chunk_n = b->chunks;
    a.chunk_m = b->chunks + a.nchunks;
    a.chunk_live = reinterpret_cast<uint8_t *>(b->chunks + 2 * (uint64_t)a.nchunks);
    a.step_graph = b->step_graph;
    a.st = b->st;
    a.roots = b->roots;
    a.root_off = b->root_off;
    a.level_log = b->level_log;
    k_bdeg<<<g5::grid_for(8), kB, 0, b->stream>>>(b->gd, b->chunk_graph, vb, b->deg, b->iso);
    if (cudaStreamSynchronize(b->stream) != cudaSuccess) return fail(G5_ERR_CUDA);
    *out = b;
    return G5_OK;
}

}  // namespace

namespace g5 {

g5_status batch_create_sharing(g5_batch *owner, g5_batch **out)
{
    if (!owner || !out) return G5_ERR_INVALID_ARG;
    return batch_create_impl(owner->graphs.data(), (int)owner->graphs.size(), owner, out);
}

size_t batch_workspace_bytes(const g5_graph *g)
{
    g5_batch b;
    BArgs &a = b.args;
    memset(&a, 0, sizeof a);
    a.ngraphs = 1;
    a.nchunks = (uint32_t)(((uint64_t)g->n + kChunk - 1) / kChunk);
    a.ntot = (uint64_t)a.nchunks * kChunk;
    a.nsteps = ((uint64_t)g->n + 31) / 32;
    a.max_tiles = (uint64_t)g->nnz / kTile + 3;
    size_t total = 0;
    each_buffer(&b, [&](auto *&, size_t bytes) { total += device_bytes(bytes); });
    return total;
}

size_t batch_copy_bytes(const g5_graph *g)
{
    // degree-ordered copy: two id maps, offsets, columns and a list of the
    // vertices with edges, which are not counted here
    const size_t n = (size_t)g->n, nnz = (size_t)g->nnz;
    return 2 * device_bytes(sizeof(uint32_t) * n) + device_bytes(sizeof(int64_t) * (n + 1)) +
           device_bytes(sizeof(uint32_t) * nnz) + device_bytes(sizeof(uint4) * std::min(n, nnz));
}

}  // namespace g5

extern "C" {

g5_status g5_batch_create(g5_graph *const *graphs, int ngraphs, g5_batch **out)
{
    return batch_create_impl(graphs, ngraphs, nullptr, out);
}

g5_status g5_batch_set_direction(g5_batch *b, double alpha, double beta)
{
    if (!b || !(alpha > 0) || !(beta > 0)) return G5_ERR_INVALID_ARG;
    b->args.alpha = alpha;
    b->args.beta = beta;
    b->bound_pred = nullptr;  // rebuild the graph with the new kernel arguments
    return G5_OK;
}

g5_status g5_batch_profile(g5_batch *b, const int64_t *roots_host, const int *nroots, uint32_t *pred_out_dev,
                           double *kernel_ms, int64_t *level_active, double *level_expand_ms, int64_t *level_examined, int32_t *level_dirs,
                           int max_levels,
                           int *levels)
{
    // host-driven level loop with CUDA events around every launch: kernel_ms
    // gets count, scan, write, expand, fixup totals (ms); level_active the
    // active vertices of each level
    if (!b || !roots_host || !nroots || !pred_out_dev || !kernel_ms || !levels) return G5_ERR_INVALID_ARG;
    const int ng = (int)b->graphs.size();
    uint64_t pb = 0;
    int off = 0;
    for (int i = 0; i < ng; ++i) {
        if (nroots[i] < 0 || nroots[i] > 64) return G5_ERR_INVALID_ARG;
        GraphDesc &d = b->hgd[i];
        d.nroots = nroots[i];
        d.mask = nroots[i] == 64 ? ~0ull : ((1ull << nroots[i]) - 1);
        d.pred_base = pb;
        pb += (uint64_t)nroots[i] * (uint64_t)d.n;
        b->h_root_off[i] = off;
        for (int r = 0; r < nroots[i]; ++r) b->h_roots[off + r] = roots_host[off + r];
        off += nroots[i];
    }
    b->h_root_off[ng] = off;
    cudaStream_t s = b->stream;
    BArgs a = b->args;
    a.pred = pred_out_dev;
    a.use_cond = 0;
    G5_CUDA(cudaMemcpyAsync(b->gd, b->hgd.data(), sizeof(GraphDesc) * ng, cudaMemcpyHostToDevice, s));
    G5_CUDA(cudaMemcpyAsync(b->roots, b->h_roots, sizeof(int64_t) * (off ? off : 1), cudaMemcpyHostToDevice, s));
    G5_CUDA(cudaMemcpyAsync(b->root_off, b->h_root_off, sizeof(int32_t) * (ng + 1), cudaMemcpyHostToDevice, s));
    if (pb) G5_CUDA(cudaMemsetAsync(pred_out_dev, 0xFF, sizeof(uint32_t) * pb, s));
    enqueue_batch(b, a, s, false);
    for (int k = 0; k < 5; ++k) kernel_ms[k] = 0;
    int L = 0;
    for (; L < kMaxLevels; ++L) {
        std::vector<cudaEvent_t> ev;
        enqueue_batch(b, a, s, true, &ev);
        G5_CUDA(cudaMemcpyAsync(b->h_st, b->st, sizeof(BState), cudaMemcpyDeviceToHost, s));
        G5_CUDA(cudaStreamSynchronize(s));
        for (size_t k = 0; k + 1 < ev.size(); ++k) {
            float t = 0;
            cudaEventElapsedTime(&t, ev[k], ev[k + 1]);
            kernel_ms[k] += t;
            if (k == 3 && level_expand_ms && L < max_levels) level_expand_ms[L] = t;
        }
        if (level_examined && L < max_levels) level_examined[L] = (int64_t)b->h_st->examined;
        if (level_dirs && L < max_levels) level_dirs[L] = (int32_t)b->h_st->dirs;
        for (cudaEvent_t e : ev) cudaEventDestroy(e);
        if (level_active && L < max_levels) level_active[L] = (int64_t)b->h_st->active;
        if (b->h_st->active == 0 || b->h_st->err) break;
    }
    *levels = L + 1;
    return b->h_st->err ? G5_ERR_CAPACITY : G5_OK;
}

g5_status g5_batch_serve_begin(g5_batch *b, uint32_t *pred_dev, const int *slots)
{
    // every graph gets `slots[g]` root slots whose parents live in pred_dev,
    // root-major per graph (graph 0 slot 0, slot 1, ..., graph 1 ...)
    if (!b || !pred_dev || !slots) return G5_ERR_INVALID_ARG;
    const int ng = (int)b->graphs.size();
    uint64_t pb = 0;
    for (int i = 0; i < ng; ++i) {
        if (slots[i] < 0 || slots[i] > 64) return G5_ERR_INVALID_ARG;
        GraphDesc &d = b->hgd[i];
        d.nroots = slots[i];
        d.mask = slots[i] == 64 ? ~0ull : ((1ull << slots[i]) - 1);
        d.pred_base = pb;
        d.dir = TD;
        d.mu = (uint64_t)d.nnz;
        d.nf = d.mf = d.examined = d.amask = d.amask_next = 0;
        pb += (uint64_t)slots[i] * (uint64_t)d.n;
    }
    cudaStream_t s = b->stream;
    b->args.pred = pred_dev;
    b->args.serving = 1;
    b->args.use_cond = 0;
    if (!b->adm_dev) G5_CUDA(cudaMalloc(&b->adm_dev, sizeof(Admit) * 64 * ng + sizeof(uint64_t) * ng));
    if (!b->adm_host) G5_CUDA(cudaMallocHost(&b->adm_host, sizeof(Admit) * 64 * ng + sizeof(uint64_t) * ng));
    G5_CUDA(cudaMemcpyAsync(b->gd, b->hgd.data(), sizeof(GraphDesc) * ng, cudaMemcpyHostToDevice, s));
    G5_CUDA(cudaMemsetAsync(b->words, 0, sizeof(uint64_t) * 3 * b->args.ntot, s));
    G5_CUDA(cudaMemsetAsync(b->args.chunk_live, 0, b->args.nchunks, s));
    // every entry starts unvisited; a retired slot's entries are reset by
    // k_sclear, so an admitted root always starts from a clean column
    if (pb) G5_CUDA(cudaMemsetAsync(pred_dev, 0xFF, sizeof(uint32_t) * pb, s));
    BState z;
    memset(&z, 0, sizeof z);
    z.level = 0;
    *b->h_st = z;
    G5_CUDA(cudaMemcpyAsync(b->st, b->h_st, sizeof(BState), cudaMemcpyHostToDevice, s));
    G5_CUDA(cudaStreamSynchronize(s));
    return G5_OK;
}

g5_status g5_batch_serve_step(g5_batch *b, const int32_t *adm_graph, const int32_t *adm_slot,
                              const int64_t *adm_root, int nadm, const uint64_t *retire_mask,
                              uint64_t *active_mask, double *device_ms)
{
    // one level of continuous batching: clear the visited bits of retired
    // slots, start the admitted roots, run one level; active_mask[g] gets the
    // slots whose frontier is still non-empty
    if (!b || (nadm && (!adm_graph || !adm_slot || !adm_root)) || !active_mask || !b->args.serving)
        return G5_ERR_INVALID_ARG;
    const int ng = (int)b->graphs.size();
    if (nadm > 64 * ng) return G5_ERR_CAPACITY;
    cudaStream_t s = b->stream;
    Admit *ah = reinterpret_cast<Admit *>(b->adm_host);
    uint64_t *rh = reinterpret_cast<uint64_t *>(ah + 64 * ng);
    bool any_retire = false;
    for (int g = 0; g < ng; ++g) {
        rh[g] = retire_mask ? retire_mask[g] : 0;
        any_retire |= rh[g] != 0;
    }
    for (int i = 0; i < nadm; ++i) {
        const int g = adm_graph[i];
        if (g < 0 || g >= ng || adm_slot[i] < 0 || adm_slot[i] >= b->hgd[g].nroots || adm_root[i] < 0 ||
            adm_root[i] >= b->hgd[g].n)
            return G5_ERR_INVALID_ARG;
        ah[i].graph = g;
        ah[i].slot = adm_slot[i];
        ah[i].root = adm_root[i];
    }
    Admit *ad = reinterpret_cast<Admit *>(b->adm_dev);
    uint64_t *rd = reinterpret_cast<uint64_t *>(ad + 64 * ng);
    G5_CUDA(cudaEventRecord(b->ev0, s));
    if (any_retire || nadm) {
        G5_CUDA(cudaMemcpyAsync(b->adm_dev, b->adm_host, sizeof(Admit) * 64 * ng + sizeof(uint64_t) * ng,
                                cudaMemcpyHostToDevice, s));
    }
    if (any_retire) k_sclear<<<g5::grid_for(8), kB, 0, s>>>(b->args, rd);
    if (nadm) k_sadmit<<<1, 128, 0, s>>>(b->args, ad, nadm);
    enqueue_batch(b, b->args, s, true);
    G5_CUDA(cudaEventRecord(b->ev1, s));
    G5_CUDA(cudaMemcpyAsync(b->hgd.data(), b->gd, sizeof(GraphDesc) * ng, cudaMemcpyDeviceToHost, s));
    G5_CUDA(cudaMemcpyAsync(b->h_st, b->st, sizeof(BState), cudaMemcpyDeviceToHost, s));
    G5_CUDA(cudaStreamSynchronize(s));
    // active slots: in the frontier the step just wrote (collected by the
    // count kernel) plus anything the expansion put into the next frontier
    for (int g = 0; g < ng; ++g) active_mask[g] = b->hgd[g].amask;
    if (device_ms) {
        float ms = 0;
        cudaEventElapsedTime(&ms, b->ev0, b->ev1);
        *device_ms = ms;
    }
    return b->h_st->err ? G5_ERR_CAPACITY : G5_OK;
}

g5_status g5_batch_root_parents(const uint32_t *pred_dev, int64_t n, int nroots, int r, uint32_t *dst_dev,
                                void *stream)
{
    if (!pred_dev || !dst_dev || n < 0 || nroots < 1 || nroots > 64 || r < 0 || r >= nroots)
        return G5_ERR_INVALID_ARG;
    if (n == 0) return G5_OK;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int blocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)g5::grid_for(8));
    k_gather_root<<<blocks, 256, 0, s>>>(pred_dev, (uint32_t)nroots, (uint32_t)r, n, dst_dev);
    return cudaGetLastError() == cudaSuccess ? G5_OK : G5_ERR_CUDA;
}

g5_status g5_batch_destroy(g5_batch *b)
{
    if (!b) return G5_ERR_INVALID_ARG;
    cudaStreamSynchronize(b->stream);
    free_batch(b);
    delete b;
    return G5_OK;
}

// Checks the roots of a run and lays them out: the graphs' descriptors, h_roots
// and h_root_off; *npred = parents in the output, *count = roots.
static g5_status bind_roots(g5_batch *b, const int64_t *roots_host, const int *nroots, uint64_t *npred, int *count)
{
    const int ng = (int)b->graphs.size();
    uint64_t pb = 0;
    int off = 0;
    for (int i = 0; i < ng; ++i) {
        if (nroots[i] < 0 || nroots[i] > 64) return G5_ERR_INVALID_ARG;
        GraphDesc &d = b->hgd[i];
        d.nroots = nroots[i];
        d.mask = nroots[i] == 64 ? ~0ull : ((1ull << nroots[i]) - 1);
        d.pred_base = pb;
        pb += (uint64_t)nroots[i] * (uint64_t)d.n;
        b->h_root_off[i] = off;
        for (int r = 0; r < nroots[i]; ++r) {
            const int64_t v = roots_host[off + r];
            if (v < 0 || v >= d.n) return G5_ERR_INVALID_ARG;
            b->h_roots[off + r] = v;
        }
        off += nroots[i];
    }
    b->h_root_off[ng] = off;
    *npred = pb;
    *count = off;
    return G5_OK;
}

g5_status g5_batch_launch(g5_batch *b, const int64_t *roots_host, const int *nroots, uint32_t *pred_out_dev)
{
    if (!b || !roots_host || !nroots || !pred_out_dev) return G5_ERR_INVALID_ARG;
    const int ng = (int)b->graphs.size();
    uint64_t pb = 0;
    int off = 0;
    G5_TRY(bind_roots(b, roots_host, nroots, &pb, &off));
    cudaStream_t s = b->stream;
    b->args.pred = pred_out_dev;
    b->args.serving = 0;
    if (!b->exec || b->bound_pred != pred_out_dev) {
        G5_TRY(build_batch_graph(b));
        b->bound_pred = pred_out_dev;
    }
    G5_CUDA(cudaMemcpyAsync(b->gd, b->hgd.data(), sizeof(GraphDesc) * ng, cudaMemcpyHostToDevice, s));
    G5_CUDA(cudaMemcpyAsync(b->roots, b->h_roots, sizeof(int64_t) * (off ? off : 1), cudaMemcpyHostToDevice, s));
    G5_CUDA(cudaMemcpyAsync(b->root_off, b->h_root_off, sizeof(int32_t) * (ng + 1), cudaMemcpyHostToDevice, s));
    G5_CUDA(cudaEventRecord(b->ev0, s));
    if (pb) G5_CUDA(cudaMemsetAsync(pred_out_dev, 0xFF, sizeof(uint32_t) * pb, s));
    G5_CUDA(cudaGraphLaunch(b->exec, s));
    G5_CUDA(cudaEventRecord(b->ev1, s));
    G5_CUDA(cudaMemcpyAsync(b->h_st, b->st, sizeof(BState), cudaMemcpyDeviceToHost, s));
    return G5_OK;
}

g5_status g5_batch_poll(g5_batch *b, int wait, int *done, double *device_ms)
{
    if (!b || !done) return G5_ERR_INVALID_ARG;
    if (wait) {
        G5_CUDA(cudaStreamSynchronize(b->stream));
    } else {
        const cudaError_t e = cudaStreamQuery(b->stream);
        if (e == cudaErrorNotReady) {
            *done = 0;
            return G5_OK;
        }
        G5_CUDA(e);
    }
    *done = 1;
    if (device_ms) {
        float ms = 0;
        cudaEventElapsedTime(&ms, b->ev0, b->ev1);
        *device_ms = ms;
    }
    if (b->h_st->err & 24u) return G5_ERR_TIMEOUT;  // the level cap, or a wait
    if (b->h_st->err) return G5_ERR_CAPACITY;
    return G5_OK;
}

g5_status g5_batch_run(g5_batch *b, const int64_t *roots_host, const int *nroots, uint32_t *pred_out_dev,
                       double *device_ms)
{
    if (!b || !roots_host || !nroots || !pred_out_dev) return G5_ERR_INVALID_ARG;
    if (!b->pgrid) {
        const g5_status st = plan_one_launch(b);
        if (st != G5_OK) {
            // (no memory for it now: the level graph needs none, and the next
            // call tries again)
            drop_one_launch(b);
            cudaGetLastError();
            if (st != G5_ERR_OOM) return st;
        }
    }
    if (b->pgrid <= 0) {
        G5_TRY(g5_batch_launch(b, roots_host, nroots, pred_out_dev));
        int done = 0;
        return g5_batch_poll(b, 1, &done, device_ms);
    }
    const int ng = (int)b->graphs.size();
    uint64_t pb = 0;
    int off = 0;
    G5_TRY(bind_roots(b, roots_host, nroots, &pb, &off));
    cudaStream_t s = b->stream;
    b->args.serving = 0;
    memcpy(b->h_stage, b->hgd.data(), sizeof(GraphDesc) * ng);
    memcpy(b->h_stage + b->roots_at, b->h_roots, sizeof(int64_t) * off);
    memcpy(b->h_stage + b->off_at, b->h_root_off, sizeof(int32_t) * (ng + 1));
    G5_CUDA(cudaMemcpyAsync(b->stage, b->h_stage, b->stage_bytes, cudaMemcpyHostToDevice, s));
    PArgs a = b->pargs;
    a.b = b->args;
    a.b.pred = pred_out_dev;
    a.b.roots = reinterpret_cast<const int64_t *>(b->stage + b->roots_at);
    a.b.root_off = reinterpret_cast<const int32_t *>(b->stage + b->off_at);
    a.npred = pb;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(b->pgrid);
    cfg.blockDim = dim3(kSB);
    cfg.dynamicSmemBytes = sizeof(PShared);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    G5_CUDA(cudaEventRecord(b->ev0, s));
    G5_CUDA(cudaLaunchKernelEx(&cfg, k_bsearch, a));
    G5_CUDA(cudaEventRecord(b->ev1, s));
    int done = 0;
    return g5_batch_poll(b, 1, &done, device_ms);
}

}  // extern "C"
