// g5_search.cuh -- one root's whole search as one launch.
//
// The plain search (no codec, parents by atomicMin) runs as a single kernel
// whose blocks are all resident and meet at the end of each level, instead of
// four launches a level under the while node of a CUDA graph: those cost 18 us
// a level whatever it held (128 us for the 7 levels of a scale-10 search whose
// 2000 entries take none of that).  What a level costs now is its chain of
// dependent loads and one meeting: 1-3 us in a block, 2-5 in a cluster, 3-8
// over the grid.  Device time per search, before and after (thresholds at
// their defaults): scale 10 108 -> 22 us, 16 164 -> 44, 20 193 -> 71, 22 280 ->
// 149, 24 619 -> 392, 26 (tuned) 1451 -> 1219.
// Four forms (enum below), by the graph's size: see search_form().
//
// The level's result is accounted while it is produced, so no counting or
// compaction pass follows a level:
//   top-down   the lane that sets a vertex's next bit first (a returning
//              atomicOr) adds its degree to the level's sums and appends its
//              row as work items of at most `tile` entries, which are the
//              next top-down level's queue (unordered: parents come from
//              atomicMin whatever the order);
//   bottom-up  a warp owns whole bitmap words, so it writes the next words
//              with plain stores and adds up the found vertices' degrees.
// Extra passes run only where the accounting would cost more: a top-down
// level with more than kClaimMax entries keeps its next-bit atomics
// fire-and-forget and counts the bitmap afterwards, and the first top-down
// level after such a level or after a bottom-up one builds its items from the
// frontier bitmap.
//
// Bitmaps at the start of level L: V holds the vertices up to level L - 1,
// N[L % 3] the frontier, N[(L + 1) % 3] is clear and collects the next
// frontier, and N[(L + 2) % 3] is cleared during the level.  The frontier
// joins V during the level, which changes nothing for a reader that tests
// both.
#pragma once

#include <cstdint>

#include "g5_common.cuh"

namespace {

enum : int32_t { DIR_TD = 0, DIR_BU = 1 };

struct LevelRec {
    int32_t dir;        // direction used to expand this level's frontier
    int32_t pad;
    uint64_t nf;        // frontier vertices
    uint64_t mf;        // their adjacency entries
    uint64_t examined;  // adjacency entries read while expanding
};

// A frontier probe: through the read-only path where the bitmap does not
// change while the kernel runs, else an ordinary load.
template <bool RO>
__device__ __forceinline__ bool front_bit(const uint32_t *front, uint32_t u)
{
    return ((RO ? __ldg(front + (u >> 5)) : front[u >> 5]) >> (u & 31)) & 1u;
}

// Warp-collective search of each active lane's adjacency [s, e) for its
// first vertex in the frontier: every lane scans its first `serial` entries
// alone (four independent loads at a time), then the warp finishes the longer
// lists one at a time, 32 entries per step (the first set ballot bit is the
// smallest index).  Returns found / par per lane and the entries read.
template <typename Off, bool RO>
__device__ __forceinline__ void first_hit(const uint32_t *front, const uint32_t *__restrict__ col, int serial,
                                          bool mine, Off s, Off e, uint32_t u0, bool &found, uint32_t &par,
                                          uint64_t &ex)
{
    const int lane = g5_lane();
    found = false;
    par = 0;
    Off j = s;
    // the first neighbour comes from the dense copy (loaded with the offsets,
    // coalesced), so a vertex whose first neighbour is in the frontier never
    // touches its row
    if (mine && s < e) {
        if (front_bit<RO>(front, u0)) {
            found = true;
            par = u0;
        }
        j = s + 1;
    }
    // (callers pass s = e = 0 on lanes without a candidate, so those lanes
    // scan nothing here)
    const Off lim = min(e, (Off)(s + serial));
    while (j < lim && !found) {
        uint32_t u[4];
        bool h[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) u[k] = (j + k < lim) ? __ldg(col + j + k) : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) h[k] = (j + k < lim) && front_bit<RO>(front, u[k]);
        int k = 0;
        while (k < 4 && j + k < lim && !h[k]) ++k;
        if (k < 4 && j + k < lim) {
            found = true;
            par = u[k];
            j += k + 1;
        } else {
            j = min((Off)(j + 4), lim);
        }
    }
    ex = mine ? (uint64_t)(j - s) : 0;
    unsigned pend = __ballot_sync(0xFFFFFFFFu, mine && !found && j < e);
    while (pend) {
        const int l = __ffs(pend) - 1;
        pend &= pend - 1;
        Off jj = __shfl_sync(0xFFFFFFFFu, j, l);
        const Off ee = __shfl_sync(0xFFFFFFFFu, e, l);
        const Off st = jj;
        bool got = false;
        uint32_t gpar = 0;
        while (jj < ee) {
            const Off idx = jj + (Off)lane;
            uint32_t u = 0;
            bool hit = false;
            if (idx < ee) {
                u = __ldg(col + idx);
                hit = front_bit<RO>(front, u);
            }
            const unsigned m = __ballot_sync(0xFFFFFFFFu, hit);
            if (m) {
                const int f = __ffs(m) - 1;
                gpar = __shfl_sync(0xFFFFFFFFu, u, f);
                got = true;
                jj += f + 1;
                break;
            }
            jj += 32;
        }
        jj = min(jj, ee);
        if (lane == l) {
            found = got;
            par = gpar;
            ex += (uint64_t)(jj - st);
        }
    }
}

// ---- the search ------------------------------------------------------------------------

constexpr int kSB = 1024;                // threads per block
constexpr int kSW = kSB / 32;
constexpr int kList = 128;               // bottom-up candidates a warp lists at a time
constexpr uint64_t kClaimMax = 1u << 18;  // frontier entries up to which top-down claims vertices
constexpr uint64_t kThin = 8;            // candidates per bitmap word below which a bottom-up level is thin
constexpr uint64_t kClaimedItems = 1u << 19;  // items a claimed frontier may have (else it is built from its bitmap)
// An item holds 256 entries at least (the tile size if that is larger): items of
// 128, 64 and 32 cost memory and gain nothing, as short levels are cut further
// anyway (us per search for 256 / 128 / 64 / 32: scale 16 44.0 / 44.7 / 45.7 /
// 46.3, 20 69.5 / 71.0 / 71.8 / 73.8, 24 391 / 393 / 396 / 401, 26 1487 / 1490 /
// 1497 / 1520; 512 and 1024 within 1 % of 256).
constexpr int kMinItemShift = 8;
constexpr uint64_t kBuildWarp = 8192;    // frontier vertices up to which a thin bitmap's items are allocated by warps
constexpr int kClusterBlocks = 16;       // blocks of the cluster form

// Where the blocks of a search meet: one block whose bitmaps and sums live in
// shared memory, one cluster, or a cooperative grid of one block per SM (64
// registers) or two (32 registers, twice the loads in flight), two SMs left out.
enum { SEARCH_BLOCK, SEARCH_CLUSTER, SEARCH_GRID1, SEARCH_GRID2 };

// The form for a graph, and where each pays (us per search, mean of 8 roots):
//             block  cluster  grid1  grid2
//   scale 10   22.3    27.5    32.4   42.2    few vertices: no latency beyond
//   scale 11   25.8    28.9    33.9   44.2    the block's own shared memory
//   scale 12   33.6    28.9    36.7   50.4    16 SMs, the hardware barrier
//   scale 15           38.1    38.7   52.4
//   scale 16           47.5    43.6   58.2    the whole GPU's loads in flight
//   scale 21                   88.4  100.6
//   scale 22                  156.3  146.8    the sweeps outweigh the meetings
//   scale 24                  482.6  391.5
constexpr int64_t kBlockVertices = 1 << 12, kBlockEntries = 1 << 16;
constexpr int64_t kClusterVertices = 1 << 15, kClusterEntries = 1 << 20;
constexpr int64_t kGrid2Vertices = 1 << 22;

inline int search_form(int64_t n, int64_t nnz)
{
    if (n <= kBlockVertices && nnz <= kBlockEntries) return SEARCH_BLOCK;
    if (n <= kClusterVertices && nnz <= kClusterEntries) return SEARCH_CLUSTER;
    return n < kGrid2Vertices ? SEARCH_GRID1 : SEARCH_GRID2;
}

// Whether the device can hold a cluster of `blocks` blocks of the cluster form.
// Sixteen is more than every device or share of one must have in one place, and
// neither the attribute that allows it nor the blocks per SM tell.
inline bool cluster_fits(const void *kern, int blocks, size_t smem)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kSB);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess) return n > 0;
    cudaGetLastError();
    return false;
}

// Bitmap words per warp step of a bottom-up level: the fewest steps of at most
// 32 words, all warps alike.  A step is a chain (words, list, offsets, probes)
// that pipelines over its own rounds only, and a last round of steps that half
// of the warps take costs the other half the same.  us per search, against
// powers of two of which each warp took about eight steps: scale 19 66 -> 60,
// 20 79 -> 71, 21 96 -> 89, 22 159 -> 149, 24 399 -> 393, 26 1435 -> 1424; two
// or three times as many steps: scale 20 75 and 78, 22 154 and 156, 26 1405 and
// 1409.
inline uint32_t bu_step_words(uint64_t nwords, uint64_t warps)
{
    const uint64_t per = (nwords + warps - 1) / warps, steps = (per + 31) / 32;
    return (uint32_t)((per + steps - 1) / steps);
}

// One level's sums, in a ring (a level adds to the next one's nf, mf and
// nitems and to its own examined, and clears the two after that, so the ring
// goes on from search to search without being cleared by the host).  In the
// grid form nf, mf, nitems and meet hold the blocks that have added their
// share in the top 12 bits, so a reader knows each by itself to be complete.
struct __align__(32) LevelSum {
    unsigned long long nf, mf, nitems;  // vertices, adjacency entries, work items of the level's frontier
    unsigned long long alloc;           // work items of claimed vertices allocated so far
    unsigned long long examined;        // adjacency entries read while expanding it
    unsigned long long meet[2];         // arrivals before its items are built, before its vertices are counted
    unsigned long long built;           // work items built from its bitmap so far
};
constexpr int kRing = 8;

// A work item: entries [start, start + cnt) of vertex u's row.
struct __align__(16) Item {
    uint32_t u;
    uint32_t cnt;   // kFirst set on the first item of a row
    int64_t start;
};
constexpr uint32_t kFirst = 1u << 31;

struct SearchArgs {
    const int64_t *row_off;
    const uint32_t *ro32;      // row offsets as uint32 when nnz < 2^32, else null
    const uint32_t *col;
    const uint32_t *deg;
    const uint32_t *first;     // first neighbour of each vertex
    const uint32_t *isolated;  // one bit per vertex without edges
    int64_t n, nnz;
    int64_t with_edges;        // vertices with edges
    uint64_t nwords, stride;   // bitmap words, rounded up to a multiple of 4
    uint32_t *bitmaps;         // V, then the three N
    int64_t *pred;
    int32_t *level;            // may be null
    Item *claimed[2];          // work items of claimed frontiers, by level parity
    uint64_t claimed_cap;
    Item *built;               // work items of a frontier built from its bitmap (room for any)
    uint64_t built_cap;
    LevelSum *sums;            // the ring
    unsigned *ring;            // [0] its place of the next search's level 0, [1] set by a block that gave up waiting
    struct SearchState *out;   // pinned host: the search's result
    LevelRec *log;             // pinned host: its level records
    int64_t root;
    uint64_t per_warp;         // bitmap words per warp of the grid
    uint32_t wps;              // bitmap words per step of a bottom-up level
    int tile_shift;
    int bu_serial;
    int max_levels;
    double alpha, beta;
};

// What the host reads after a search.
struct SearchState {
    int32_t level;       // index of the last (empty) level's frontier
    uint32_t err;
    uint64_t nvisited;
    uint64_t ns;         // the kernel's own time
};

// Per-warp scratch: the items of a top-down step or the words and candidates
// of a bottom-up one.
union WarpScratch {
    struct {
        uint32_t end[32];   // inclusive entry counts of the step's items
        uint32_t u[32];
        int64_t base[32];   // column index of entry e of item i: base[i] + e
    } td;
    struct {
        uint32_t out[32];      // found vertices of the step's words
        uint16_t list[kList];  // candidates: word of the step * 32 + bit
    } bu;
};

struct SearchShared {
    WarpScratch w[kSW];
    LevelSum sums[kRing];                 // SEARCH_BLOCK: the ring
    unsigned long long nf, mf, nitems, ex;  // the block's share of the level's sums
    unsigned long long got[2][kClusterBlocks][3];  // SEARCH_CLUSTER: every block's share, by level parity
    unsigned long long lvl[3];            // nf, mf, items of the next level
    int32_t dir;                          // its direction
    uint32_t stop;
    uint32_t warp_items[kSW];
    unsigned long long item_base;
    uint64_t t0;                          // start of the search (block 0)
};

__device__ __forceinline__ uint64_t now_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void offsets_of(const SearchArgs &a, uint64_t v, uint32_t &s, uint32_t &e)
{
    s = __ldg(a.ro32 + v);
    e = __ldg(a.ro32 + v + 1);
}
__device__ __forceinline__ void offsets_of(const SearchArgs &a, uint64_t v, int64_t &s, int64_t &e)
{
    s = __ldg(a.row_off + v);
    e = __ldg(a.row_off + v + 1);
}

// The warp's new vertices and their entries, into the block's share.
__device__ __forceinline__ void add_sums(SearchShared &sh, uint32_t nf, uint64_t mf)
{
    if (!__any_sync(0xFFFFFFFFu, nf != 0)) return;
    nf = __reduce_add_sync(0xFFFFFFFFu, nf);
    mf = warp_add_u51(mf);
    if (g5_lane() == 0) {
        atomicAdd(&sh.nf, (unsigned long long)nf);
        atomicAdd(&sh.mf, (unsigned long long)mf);
    }
}

// All blocks meet inside a level; what any of them wrote before is visible to
// all after.  `word` counts the arrivals (grid form).
template <int MODE>
__device__ __forceinline__ void meet(const SearchArgs &a, SearchShared &sh, unsigned long long *word)
{
    if (MODE == SEARCH_CLUSTER) {
        asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
        return;
    }
    __syncthreads();
    if (MODE == SEARCH_BLOCK) return;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(word, 1ull << kArrive);
        unsigned long long x;
        if (!await<1>(word, a.ring + 1, &x)) sh.stop = 1;
        __threadfence();
    }
    __syncthreads();
}

// The end of a level: the blocks' shares of the next level's sums come
// together in sh.lvl, its direction in sh.dir, and everything written during
// the level is visible.  mu and cnf: the entries of the vertices not visited
// before the level, and its frontier's vertices.
template <int MODE>
__device__ __forceinline__ void finish_level(const SearchArgs &a, SearchShared &sh, LevelSum *cur, LevelSum *next,
                                             int32_t L, int32_t dir, uint64_t cnf, uint64_t mu)
{
    __syncthreads();
    if (MODE == SEARCH_CLUSTER) {
        // every block hands its share to every block's shared memory
        if (threadIdx.x < gridDim.x) {
            const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&sh.got[L & 1][blockIdx.x][0]);
            uint32_t there;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(there) : "r"(mine), "r"(threadIdx.x));
            asm volatile("st.shared::cluster.u64 [%0], %1;\n" ::"r"(there), "l"(sh.nf) : "memory");
            asm volatile("st.shared::cluster.u64 [%0], %1;\n" ::"r"(there + 8), "l"(sh.mf) : "memory");
            asm volatile("st.shared::cluster.u64 [%0], %1;\n" ::"r"(there + 16), "l"(sh.nitems) : "memory");
            if (threadIdx.x == 0 && sh.ex) atomicAdd(&cur->examined, sh.ex);
        }
        meet<MODE>(a, sh, nullptr);
        if (threadIdx.x < 32) {
            unsigned long long t = 0;
            if (threadIdx.x < 3)
                for (uint32_t b = 0; b < gridDim.x; ++b) t += sh.got[L & 1][b][threadIdx.x];
            if (threadIdx.x < 3) sh.lvl[threadIdx.x] = t;
            __syncwarp();
        }
    } else if (threadIdx.x == 0) {
        if (MODE == SEARCH_BLOCK) {
            sh.lvl[0] = sh.nf;
            sh.lvl[1] = sh.mf;
            sh.lvl[2] = sh.nitems;
            cur->examined = sh.ex;
        } else {
            if (sh.ex) atomicAdd(&cur->examined, sh.ex);
            __threadfence();
            atomicAdd(&next->nf, sh.nf + (1ull << kArrive));
            atomicAdd(&next->mf, sh.mf + (1ull << kArrive));
            atomicAdd(&next->nitems, sh.nitems + (1ull << kArrive));
            if (!await<3>(&next->nf, a.ring + 1, sh.lvl)) sh.stop = 1;
            __threadfence();
        }
    }
    if (threadIdx.x == 0) {
        // the direction switch (Beamer), decided alike by every block
        const uint64_t tn = sh.lvl[0], tm = sh.lvl[1], mu_after = mu >= tm ? mu - tm : 0;
        int32_t nd = dir;
        if (dir == DIR_TD) {
            if (above_quotient(tm, mu_after, a.alpha)) nd = DIR_BU;
        } else if (tn < cnf && below_quotient(tn, (uint64_t)a.n, a.beta)) {
            nd = DIR_TD;
        }
        sh.dir = nd;
        sh.nf = sh.mf = sh.nitems = sh.ex = 0;
    }
    __syncthreads();
}

// Writes the items of a row [s, e) of vertex v, `nseg` of them, at p.
template <typename Off>
__device__ __forceinline__ void put_item(Item *p, uint32_t v, Off s, Off e, uint32_t k, int tile_shift)
{
    const Off at = s + ((Off)k << tile_shift);
    Item it;
    it.u = v;
    it.cnt = (uint32_t)min(e - at, (Off)1 << tile_shift) | (k == 0 ? kFirst : 0u);
    it.start = (int64_t)at;
    *p = it;
}

// Appends the rows of the warp's vertices (lanes with nseg > 0) to the work
// items, lane by lane from items[base + excl] on.  Long rows (hubs) are laid
// out by the whole warp, the rest by their lane.
template <typename Off>
__device__ __forceinline__ void append_items(Item *items, uint64_t cap, uint64_t base, uint32_t excl, uint32_t v,
                                             Off s, Off e, uint32_t nseg, int tile_shift)
{
    if (base + excl + nseg > cap) nseg = 0;  // no room: the caller sees it from the total
    Item *p = items + base + excl;
    if (nseg <= 8)
        for (uint32_t k = 0; k < nseg; ++k) put_item<Off>(p + k, v, s, e, k, tile_shift);
    unsigned big = __ballot_sync(0xFFFFFFFFu, nseg > 8);
    while (big) {
        const int l = __ffs(big) - 1;
        big &= big - 1;
        const uint32_t vv = __shfl_sync(0xFFFFFFFFu, v, l), c = __shfl_sync(0xFFFFFFFFu, nseg, l);
        const uint32_t x = __shfl_sync(0xFFFFFFFFu, excl, l);
        const Off ss = __shfl_sync(0xFFFFFFFFu, s, l), ee = __shfl_sync(0xFFFFFFFFu, e, l);
        for (uint32_t k = g5_lane(); k < c; k += 32) put_item<Off>(items + base + x + k, vv, ss, ee, k, tile_shift);
    }
}

// Top-down.  Many items: 32 per warp step, their entries spread over the
// lanes; few: one per warp; fewer still: an item's entries split over several
// warps, down to 32 each, so that a short level keeps every chain short.
// Every entry (u, v) with v not visited takes its parent by atomicMin and sets
// v's next bit.
template <typename Off, bool CLAIM>
__device__ __forceinline__ void search_td(const SearchArgs &a, SearchShared &sh, uint32_t *V, const uint32_t *front, uint32_t *next,
                          const Item *items, uint64_t nitems, Item *out, unsigned long long *alloc, int32_t L)
{
    const int lane = g5_lane();
    WarpScratch &ws = sh.w[threadIdx.x >> 5];
    // neighbouring warps of the work order sit in different blocks
    const uint64_t gw = (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const uint64_t nw = (uint64_t)gridDim.x * kSW;
    const uint32_t ipw = items_per_step(nitems, (uint32_t)nw);
    uint32_t split_shift = 0;
    while ((5 + (int)split_shift) < a.tile_shift && (nitems << (split_shift + 1)) <= nw) ++split_shift;
    uint32_t nf = 0;
    uint64_t mf = 0;
    const uint64_t units = ipw == 1 ? nitems << split_shift : item_steps(nitems, ipw);
    for (uint64_t t = gw; t < units; t += nw) {
        // (a step's items lie apart, so that each has its share of the hubs')
        const uint64_t i = ipw == 1 ? (t >> split_shift) + lane : t + lane * units;
        uint32_t cnt = 0, u = 0;
        int64_t s = 0;
        if ((uint32_t)lane < ipw && i < nitems) {
            const uint4 raw = __ldcg(reinterpret_cast<const uint4 *>(items + i));
            u = raw.x;
            cnt = raw.y & ~kFirst;
            s = (int64_t)(raw.z | (uint64_t)raw.w << 32);
            const uint32_t part = (1u << a.tile_shift) >> split_shift;
            const uint32_t at = (uint32_t)(t & ((1u << split_shift) - 1)) * part;
            // the frontier joins the visited set
            if ((raw.y & kFirst) && at == 0) atomicOr(V + (u >> 5), 1u << (u & 31));
            s += at;
            cnt = cnt > at ? min(cnt - at, part) : 0u;
        }
        uint32_t total;
        const uint32_t excl = warp_excl_u32(cnt, total);
        __syncwarp();
        ws.td.end[lane] = excl + cnt;
        ws.td.u[lane] = u;
        ws.td.base[lane] = s - (int64_t)excl;
        __syncwarp();
        for (uint32_t e0 = 0; e0 < total; e0 += 32) {
            const uint32_t x = e0 + lane;
            bool claimed = false;
            uint32_t v = 0;
            Off vs = 0, ve = 0;
            if (x < total) {
                int lo = 0;
                if (ipw > 1) {
                    int hi = 31;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (ws.td.end[mid] <= x) lo = mid + 1;
                        else hi = mid;
                    }
                }
                v = __ldg(a.col + (ws.td.base[lo] + (int64_t)x));
                const uint32_t w = v >> 5, bit = 1u << (v & 31);
                // every load the entry may need goes out together
                const uint32_t seen = V[w] | front[w];
                if (CLAIM) offsets_of(a, v, vs, ve);
                if (!(seen & bit)) {
                    const unsigned long long p = ws.td.u[lo];
                    if (CLAIM) {
                        atomicMin((unsigned long long *)(a.pred + v), p);
                        claimed = !(atomicOr(next + w, bit) & bit);
                    } else {
                        // parents only decrease during a level, so a read
                        // value <= u (even a stale one) makes the atomic moot
                        if ((unsigned long long)a.pred[v] > p) atomicMin((unsigned long long *)(a.pred + v), p);
                        if (!(next[w] & bit)) atomicOr(next + w, bit);
                    }
                }
            }
            if (CLAIM && __any_sync(0xFFFFFFFFu, claimed)) {
                uint32_t nseg = 0;
                if (claimed) {
                    const uint64_t d = (uint64_t)(ve - vs);
                    nseg = (uint32_t)((d + (1u << a.tile_shift) - 1) >> a.tile_shift);
                    ++nf;
                    mf += d;
                    if (a.level) a.level[v] = L + 1;
                }
                uint32_t tot;
                const uint32_t at = warp_excl_u32(nseg, tot);
                unsigned long long base = 0;
                if (lane == 0) {
                    base = atomicAdd(alloc, (unsigned long long)tot);
                    atomicAdd(&sh.nitems, (unsigned long long)tot);
                }
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                append_items<Off>(out, a.claimed_cap, base, at, v, vs, ve, nseg, a.tile_shift);
            }
        }
    }
    if (CLAIM) add_sums(sh, nf, mf);
}

// Searches the `total` listed candidates of a step, 32 together, the row offsets
// and first neighbours loaded one round ahead.  (The sums go to shared memory
// round by round: registers are what this loop is short of.)
template <typename Off, bool WIDE>
__device__ __forceinline__ void search_bu_rounds(const SearchArgs &a, SearchShared &sh, WarpScratch &ws,
                                                 const uint32_t *front, uint32_t *next, uint32_t w0, uint32_t total,
                                                 int32_t L)
{
    const int lane = g5_lane();
    Off s1 = 0, e1 = 0;
    uint32_t f1 = 0;
    if ((uint32_t)lane < total) {
        const uint64_t v = (uint64_t)w0 * 32 + ws.bu.list[lane];
        offsets_of(a, v, s1, e1);
        f1 = __ldg(a.first + v);
    }
    for (uint32_t k = lane; k < total + lane; k += 32) {
        const bool mine = k < total;
        const uint32_t u0 = f1;
        const Off s = s1, e = e1;
        s1 = e1 = 0;
        if (k + 32 < total) {
            const uint64_t v = (uint64_t)w0 * 32 + ws.bu.list[k + 32];
            offsets_of(a, v, s1, e1);
            f1 = __ldg(a.first + v);
        }
        bool found;
        uint32_t par;
        uint64_t ex;
        first_hit<Off, false>(front, a.col, a.bu_serial, mine, s, e, u0, found, par, ex);
        if (found) {
            const uint32_t id = ws.bu.list[k];
            const uint64_t v = (uint64_t)w0 * 32 + id;
            a.pred[v] = (int64_t)par;
            if (a.level) a.level[v] = L + 1;
            if (WIDE) atomicOr(next + w0 + (id >> 5), 1u << (id & 31));
            else atomicOr(&ws.bu.out[id >> 5], 1u << (id & 31));
        }
        const unsigned fm = __ballot_sync(0xFFFFFFFFu, found);
        // (with 32-bit offsets the degrees of distinct vertices add up to less than 2^32)
        const uint64_t x = sizeof(Off) == 4 ? (uint64_t)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)ex) : warp_add_u51(ex);
        const uint64_t d = sizeof(Off) == 4 ? (uint64_t)__reduce_add_sync(0xFFFFFFFFu, found ? (uint32_t)(e - s) : 0u)
                                            : warp_add_u51(found ? (uint64_t)(e - s) : 0u);
        if (lane == 0) {
            atomicAdd(&sh.ex, (unsigned long long)x);
            if (fm) {
                atomicAdd(&sh.nf, (unsigned long long)__popc(fm));
                atomicAdd(&sh.mf, (unsigned long long)d);
            }
        }
    }
    __syncwarp();
}

// Bottom-up.  A warp takes a step of bitmap words and lists their unvisited
// vertices, so that every lane of a round has one.  It owns the step's words,
// so the visited ones take plain stores.
//   narrow  up to 32 words, one per lane; as many at a time as fit the list;
//           the found bits are gathered in shared memory
//   WIDE    (few candidates per word) 128 words, four per lane in one vector
//           load, and every lane lists its own, so that a step with hardly any
//           candidates costs little more than the loads; found bits by atomicOr
template <typename Off, bool WIDE>
__device__ __forceinline__ void search_bu(const SearchArgs &a, SearchShared &sh, uint32_t *V, const uint32_t *front, uint32_t *next,
                          uint32_t *spare, uint32_t wps, int32_t L)
{
    const int lane = g5_lane();
    WarpScratch &ws = sh.w[threadIdx.x >> 5];
    if (WIDE) wps = 128;
    const uint32_t nwords = (uint32_t)a.nwords;  // at most 2^27
    const uint32_t stride = gridDim.x * kSW * wps;
    for (uint32_t w0 = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * wps; w0 < nwords; w0 += stride) {
        uint32_t total = 0;
        unsigned todo = 0;           // words of the lanes still to be listed
        int q = WIDE ? -1 : 3;       // WIDE, more candidates than the list holds: the words' place in their vectors
        __syncwarp();
        if (WIDE) {
            const uint32_t w = w0 + 4 * lane;
            uint4 c = make_uint4(0, 0, 0, 0);
            if (w < nwords) {  // (the bitmaps are padded to whole vectors)
                const uint4 f = *reinterpret_cast<const uint4 *>(front + w);
                uint4 v = *reinterpret_cast<const uint4 *>(V + w);
                v = make_uint4(v.x | f.x, v.y | f.y, v.z | f.z, v.w | f.w);
                if (f.x | f.y | f.z | f.w) *reinterpret_cast<uint4 *>(V + w) = v;
                *reinterpret_cast<uint4 *>(spare + w) = c;
                c = make_uint4(~v.x, ~v.y, ~v.z, ~v.w);
            }
            uint32_t at = warp_excl_u32(__popc(c.x) + __popc(c.y) + __popc(c.z) + __popc(c.w), total);
            if (total == 0) continue;
            if (total <= kList) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    for (uint32_t t = k == 0 ? c.x : k == 1 ? c.y : k == 2 ? c.z : c.w; t; t &= t - 1)
                        ws.bu.list[at++] = (uint16_t)((4 * lane + k) * 32 + __ffs(t) - 1);
                __syncwarp();
                search_bu_rounds<Off, WIDE>(a, sh, ws, front, next, w0, total, L);
                continue;
            }
        } else {
            uint32_t c = 0;
            if (lane < wps && w0 + lane < nwords) {
                const uint32_t f = front[w0 + lane], v = V[w0 + lane] | f;
                if (f) V[w0 + lane] = v;
                spare[w0 + lane] = 0;
                c = ~v;
            }
            ws.bu.out[lane] = 0;
            todo = __ballot_sync(0xFFFFFFFFu, c != 0);
        }
        for (;;) {
            while (WIDE && !todo && q < 3) {
                ++q;
                todo = __ballot_sync(0xFFFFFFFFu, w0 + 4 * lane + q < nwords && ~V[w0 + 4 * lane + q] != 0);
            }
            if (!todo) break;
            // words in order, as long as the list has room for a whole one
            // (read again here: nothing of them is held during the rounds)
            const uint32_t w = WIDE ? w0 + 4 * lane + q : w0 + lane;
            const uint32_t c = (todo >> lane) & 1u ? ~V[w] : 0u;
            total = 0;
            while (todo && total + 32 <= kList) {
                const int j = __ffs(todo) - 1;
                todo &= todo - 1;
                const uint32_t cj = __shfl_sync(0xFFFFFFFFu, c, j);
                if ((cj >> lane) & 1u)
                    ws.bu.list[total + __popc(cj & g5_lanemask_lt())] = (uint16_t)((WIDE ? 4 * j + q : j) * 32 + lane);
                total += __popc(cj);
            }
            __syncwarp();
            search_bu_rounds<Off, WIDE>(a, sh, ws, front, next, w0, total, L);
        }
        if (!WIDE) {
            const uint32_t o = ws.bu.out[lane];
            if (o) next[w0 + lane] = o;
        }
    }
}

// After a top-down level that did not claim: the new vertices and their degree
// sum, and their levels.  A lane walks its own word, two bits at a time.
__device__ __forceinline__ void search_count(const SearchArgs &a, SearchShared &sh, const uint32_t *next, int32_t L)
{
    uint32_t nf = 0;
    uint64_t mf = 0;
    const uint64_t nthr = (uint64_t)gridDim.x * kSB;
    for (uint64_t w = (uint64_t)blockIdx.x * kSB + threadIdx.x; w < a.nwords; w += nthr) {
        uint32_t x = next[w];
        nf += __popc(x);
        while (x) {
            const uint64_t v = w * 32 + (__ffs(x) - 1);
            x &= x - 1;
            const uint64_t v2 = x ? w * 32 + (__ffs(x) - 1) : v;
            const uint32_t d = __ldg(a.deg + v), d2 = __ldg(a.deg + v2);
            mf += d;
            if (a.level) a.level[v] = L + 1;
            if (x) {
                mf += d2;
                if (a.level) a.level[v2] = L + 1;
                x &= x - 1;
            }
        }
    }
    add_sums(sh, nf, mf);
}

// The work items of a frontier of nf vertices held as a bitmap.  Few vertices
// per word, or no more than two per warp: a warp looks through 32 words and
// allocates for each that holds any.  Many: a lane takes four words, and one
// allocation serves a block step; so also from kBuildWarp vertices on, where the
// warps' allocations queue up at their one counter (43,541 vertices in 2 M words:
// 40 us of 52 for the level, now 18; mean search at scale 24 417 -> 400 us, 26
// 1456 -> 1393).  (Two per warp: 1038 vertices in 2048 words took one block 9.5
// us; mean search at scale 16 49 -> 44 us, 14 36 -> 32, 18 52 -> 49.)
template <typename Off>
__device__ __forceinline__ void search_build(const SearchArgs &a, SearchShared &sh, const uint32_t *front, uint64_t nf, Item *items,
                             unsigned long long *alloc)
{
    const int lane = g5_lane(), wid = threadIdx.x >> 5;
    const uint32_t round = (1u << a.tile_shift) - 1;
    if (nf <= kBuildWarp && (4 * nf <= a.nwords || nf <= 2 * gridDim.x * kSW)) {
        const uint64_t gw = (uint64_t)wid * gridDim.x + blockIdx.x;
        // (small graphs: fewer words per warp, so that every warp has some)
        uint32_t wpw = 32;
        while (wpw > 1 && (uint64_t)wpw > a.per_warp) wpw >>= 1;
        for (uint64_t w0 = gw * wpw; w0 < a.nwords; w0 += (uint64_t)gridDim.x * kSW * wpw) {
            const uint32_t x = (uint32_t)lane < wpw && w0 + lane < a.nwords ? front[w0 + lane] : 0u;
            for (unsigned t = __ballot_sync(0xFFFFFFFFu, x != 0u); t; t &= t - 1) {
                const int j = __ffs(t) - 1;
                const uint32_t xj = __shfl_sync(0xFFFFFFFFu, x, j);
                const uint32_t v = (uint32_t)((w0 + j) * 32 + lane);
                Off s = 0, e = 0;
                if ((xj >> lane) & 1u) offsets_of(a, v, s, e);
                const uint32_t nseg = (uint32_t)(((uint64_t)(e - s) + round) >> a.tile_shift);
                uint32_t tot;
                const uint32_t at = warp_excl_u32(nseg, tot);
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(alloc, (unsigned long long)tot);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                append_items<Off>(items, ~0ull, base, at, v, s, e, nseg, a.tile_shift);
            }
        }
        return;
    }
    const uint64_t step = (uint64_t)gridDim.x * kSB * 4;
    for (uint64_t b0 = (uint64_t)blockIdx.x * kSB * 4; b0 < a.nwords; b0 += step) {
        const uint64_t w0 = b0 + 4 * threadIdx.x;
        uint4 x = make_uint4(0, 0, 0, 0);
        if (w0 < a.nwords) x = *reinterpret_cast<const uint4 *>(front + w0);
        uint32_t mine = 0;
#pragma unroll 1
        for (int q = 0; q < 4; ++q)
            for (uint32_t t = q == 0 ? x.x : q == 1 ? x.y : q == 2 ? x.z : x.w; t; t &= t - 1)
                mine += (uint32_t)(((uint64_t)__ldg(a.deg + (w0 + q) * 32 + (__ffs(t) - 1)) + round) >> a.tile_shift);
        uint32_t tot;
        uint32_t at = warp_excl_u32(mine, tot);
        if (lane == 0) sh.warp_items[wid] = tot;
        __syncthreads();
        if (wid == 0) {
            const uint32_t ex = warp_excl_u32(sh.warp_items[lane], tot);
            sh.warp_items[lane] = ex;
            if (lane == 0 && tot) sh.item_base = atomicAdd(alloc, (unsigned long long)tot);
        }
        __syncthreads();
        const uint64_t base = sh.item_base + sh.warp_items[wid];
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
            uint32_t t = q == 0 ? x.x : q == 1 ? x.y : q == 2 ? x.z : x.w;
            while (__any_sync(0xFFFFFFFFu, t != 0)) {
                uint32_t v = 0, nseg = 0;
                Off s = 0, e = 0;
                if (t) {
                    v = (uint32_t)((w0 + q) * 32 + (__ffs(t) - 1));
                    t &= t - 1;
                    offsets_of(a, v, s, e);
                    nseg = (uint32_t)(((uint64_t)(e - s) + round) >> a.tile_shift);
                }
                append_items<Off>(items, ~0ull, base, at, v, s, e, nseg, a.tile_shift);
                at += nseg;
            }
        }
        __syncthreads();  // warp_items and item_base are free again
    }
}

template <typename Off, int MODE>
__global__ void __launch_bounds__(kSB, MODE == SEARCH_GRID2 ? 2 : 1) k_search(const __grid_constant__ SearchArgs a)
{
    extern __shared__ __align__(16) unsigned char s_search[];
    SearchShared &sh = *reinterpret_cast<SearchShared *>(s_search);
    const uint64_t tid = (uint64_t)blockIdx.x * kSB + threadIdx.x, nthr = (uint64_t)gridDim.x * kSB;
    uint32_t *V = MODE == SEARCH_BLOCK ? reinterpret_cast<uint32_t *>(s_search + sizeof(SearchShared)) : a.bitmaps;
    uint32_t *N = V + a.stride;
    LevelSum *sums = MODE == SEARCH_BLOCK ? sh.sums : a.sums;
    if (blockIdx.x == 0 && threadIdx.x == kSB - 1) sh.t0 = now_ns();
    // prologue: vertices without edges count as visited (they are never
    // reached), as do the ones past n
    const uint64_t root = (uint64_t)a.root;
    for (uint64_t w = tid; w < a.stride; w += nthr) {
        uint32_t iso = w < a.nwords ? a.isolated[w] : ~0u;
        if (w == a.nwords - 1 && (a.n & 31)) iso |= ~((1u << (a.n & 31)) - 1u);
        V[w] = iso;
        N[w] = w == (root >> 5) ? 1u << (root & 31) : 0u;
        N[a.stride + w] = 0;
        N[2 * a.stride + w] = 0;
    }
    for (uint64_t i = tid; i < (uint64_t)a.n / 2; i += nthr) {
        longlong2 p = make_longlong2(-1, -1);
        if (i == (root >> 1)) {
            if (root & 1) p.y = (long long)root;
            else p.x = (long long)root;
        }
        reinterpret_cast<longlong2 *>(a.pred)[i] = p;
    }
    if ((a.n & 1) && tid == 0) a.pred[a.n - 1] = root == (uint64_t)a.n - 1 ? (int64_t)root : -1;
    if (a.level)
        for (uint64_t v = tid; v < (uint64_t)a.n; v += nthr) a.level[v] = v == root ? 0 : -1;
    Off rs, re;
    offsets_of(a, root, rs, re);
    const uint64_t rdeg = (uint64_t)(re - rs);
    const uint64_t ritems = (rdeg + ((uint64_t)1 << a.tile_shift) - 1) >> a.tile_shift;
    for (uint64_t k = tid; k < ritems && ritems <= a.claimed_cap; k += nthr)
        put_item<Off>(a.claimed[0] + k, (uint32_t)root, rs, re, (uint32_t)k, a.tile_shift);
    if (threadIdx.x == 0) {
        sh.nf = sh.mf = sh.nitems = sh.ex = 0;
        // (a search queued behind one that gave up waiting, whose ring the host
        // has not cleared yet, gives up as well)
        sh.stop = MODE >= SEARCH_GRID1 ? __ldcg(a.ring + 1) : 0;
    }
    if (MODE == SEARCH_BLOCK)
        for (uint32_t i = threadIdx.x; i < kRing * sizeof(LevelSum) / 8; i += kSB)
            reinterpret_cast<unsigned long long *>(sums)[i] = 0;
    const uint32_t place = MODE == SEARCH_BLOCK ? 0u : __ldcg(a.ring);
    uint64_t cnf = 1, cmf = rdeg, citems = ritems, mu = (uint64_t)a.nnz - rdeg, visited = 1;
    bool have_items = ritems <= a.claimed_cap;
    int32_t dir = DIR_TD, L = 0;
    uint32_t err = 0;
    meet<MODE>(a, sh, &sums[place % kRing].meet[0]);
    while (!sh.stop) {
        uint32_t *front = N + (uint64_t)(L % 3) * a.stride;
        uint32_t *next = N + (uint64_t)((L + 1) % 3) * a.stride;
        uint32_t *spare = N + (uint64_t)((L + 2) % 3) * a.stride;
        LevelSum *cur = sums + (place + L) % kRing, *nxt = sums + (place + L + 1) % kRing;
        if (tid < 2 * sizeof(LevelSum) / 8) {
            const uint32_t k = (uint32_t)tid / (sizeof(LevelSum) / 8), f = (uint32_t)tid % (sizeof(LevelSum) / 8);
            reinterpret_cast<unsigned long long *>(sums + (place + L + 2 + k) % kRing)[f] = 0;
        }
        const bool claim = cmf <= kClaimMax;
        if (dir == DIR_TD) {
            const Item *items = have_items ? a.claimed[L & 1] : a.built;
            if (!have_items) {
                // (a claimed frontier without room has used alloc: count anew)
                search_build<Off>(a, sh, front, cnf, a.built, &cur->built);
                meet<MODE>(a, sh, &cur->meet[1]);
                if (sh.stop) break;
                citems = MODE == SEARCH_BLOCK ? cur->built : __ldcg(&cur->built);
            }
            for (uint64_t w = tid; w < a.nwords; w += nthr) spare[w] = 0;
            if (claim) {
                search_td<Off, true>(a, sh, V, front, next, items, citems, a.claimed[(L + 1) & 1], &nxt->alloc, L);
            } else {
                search_td<Off, false>(a, sh, V, front, next, items, citems, nullptr, nullptr, L);
                meet<MODE>(a, sh, &nxt->meet[0]);
                if (sh.stop) break;
                search_count(a, sh, next, L);
            }
        } else {
            const uint64_t unv = (uint64_t)a.with_edges - visited;
            const bool thin = unv < a.nwords * kThin;
            if (thin && a.per_warp > 32) {
                search_bu<Off, true>(a, sh, V, front, next, spare, 0, L);
            } else {
                search_bu<Off, false>(a, sh, V, front, next, spare, a.wps, L);
            }
        }
        finish_level<MODE>(a, sh, cur, nxt, L, dir, cnf, mu);
        if (sh.stop) break;
        if (blockIdx.x == 0 && threadIdx.x == kSB - 1) {
            // (the block's last warp, the last to be given work)
            LevelRec r;
            r.dir = dir;
            r.pad = 0;
            r.nf = cnf;
            r.mf = cmf;
            r.examined = dir == DIR_TD ? cmf : MODE == SEARCH_BLOCK ? cur->examined : __ldcg(&cur->examined);
            a.log[L] = r;
        }
        const uint64_t tn = sh.lvl[0], tm = sh.lvl[1];
        mu = mu >= tm ? mu - tm : 0;
        have_items = dir == DIR_TD && claim && sh.lvl[2] <= a.claimed_cap;
        citems = sh.lvl[2];
        cnf = tn;
        cmf = tm;
        visited += tn;
        dir = sh.dir;
        ++L;
        if (tn == 0) break;
        if (L + 1 >= a.max_levels) {
            err = G5_DEVERR_LEVELS;
            break;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == kSB - 1) {
        if (L < a.max_levels) {
            LevelRec r;
            r.dir = dir;
            r.pad = 0;
            r.nf = cnf;
            r.mf = cmf;
            r.examined = 0;
            a.log[L] = r;
        }
        a.out->level = L;
        a.out->err = err | (sh.stop ? (uint32_t)G5_DEVERR_WAIT : 0u);
        a.out->nvisited = visited;
        a.out->ns = now_ns() - sh.t0;
        // levels L and L + 1 of this search are the last records used, and
        // level L - 1 cleared the two after its next one
        if (MODE != SEARCH_BLOCK) a.ring[0] = (place + L + 1) % kRing;
    }
}

}  // namespace
