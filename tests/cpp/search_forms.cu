// Every form of the one-launch search (g5_search.cuh) on one graph, with 32-bit
// and with 64-bit row offsets, whatever form the library would choose for it.
//   search_forms parents GRAPH OUT ROOT...   parents (int64) and levels (int32) of
//       every form, offset width and root, in that order, to OUT
//   search_forms waits GRAPH OUT ROOT        a search whose blocks wait for arrivals
//       that never come, one queued behind it, and one after the ring is cleared:
//       the error bits and parents of each, per grid form, to OUT
//   search_forms clusters GRAPH OUT N...     1 or 0 (int64) to OUT for each N: whether
//       the device can hold a cluster of N blocks of the cluster form
// GRAPH: int64 n, int64 nnz, int64 row offsets, uint32 columns.  Built with a
// short G5_MEET_NS.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "g5_search.cuh"

#define CHECK(x)                                                                      \
    do {                                                                              \
        cudaError_t e_ = (x);                                                         \
        if (e_ != cudaSuccess) {                                                      \
            std::fprintf(stderr, "%s: %s\n", #x, cudaGetErrorString(e_));             \
            std::exit(2);                                                             \
        }                                                                             \
    } while (0)

template <typename T>
static T *device(const std::vector<T> &h, size_t room = 0)
{
    T *p;
    CHECK(cudaMalloc(&p, sizeof(T) * std::max<size_t>(1, std::max(h.size(), room))));
    CHECK(cudaMemcpy(p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
    return p;
}

struct Searcher {
    SearchArgs a = {};
    SearchState *out;
    cudaStream_t s;

    Searcher(const std::vector<int64_t> &ro, const std::vector<uint32_t> &col)
    {
        const size_t n = ro.size() - 1;
        std::vector<uint32_t> ro32(ro.begin(), ro.end()), deg(n), first(n), iso((n + 31) / 32);
        for (size_t v = 0; v < n; ++v) {
            deg[v] = (uint32_t)(ro[v + 1] - ro[v]);
            first[v] = deg[v] ? col[ro[v]] : 0u;
            if (!deg[v]) iso[v / 32] |= 1u << (v % 32);
            a.with_edges += deg[v] != 0;
        }
        a.n = (int64_t)n;
        a.nnz = (int64_t)col.size();
        a.nwords = iso.size();
        a.stride = (a.nwords + 3) & ~(uint64_t)3;
        a.row_off = device(ro);
        a.ro32 = device(ro32);
        a.col = device(col);
        a.deg = device(deg);
        a.first = device(first);
        a.isolated = device(iso);
        a.tile_shift = kMinItemShift;
        a.bu_serial = 8;
        a.max_levels = 4096;
        a.alpha = 14;
        a.beta = 24;
        const uint64_t tiles = (uint64_t)a.nnz >> a.tile_shift;
        a.claimed_cap = std::min<uint64_t>(n + tiles + 1, kClaimedItems);
        a.built_cap = n + tiles + 1;
        CHECK(cudaMalloc(&a.bitmaps, 16 * a.stride));
        CHECK(cudaMalloc(&a.pred, 8 * n));
        CHECK(cudaMalloc(&a.level, 4 * n));
        for (Item *&c : a.claimed) CHECK(cudaMalloc(&c, sizeof(Item) * a.claimed_cap));
        CHECK(cudaMalloc(&a.built, sizeof(Item) * a.built_cap));
        CHECK(cudaMalloc(&a.sums, sizeof(LevelSum) * (kRing + 1)));
        a.ring = reinterpret_cast<unsigned *>(a.sums + kRing);
        CHECK(cudaMallocHost(&a.log, sizeof(LevelRec) * (size_t)a.max_levels));
        CHECK(cudaMallocHost(&out, sizeof(SearchState)));
        CHECK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        clear();
    }

    void clear()
    {
        CHECK(cudaMemsetAsync(a.sums, 0, sizeof(LevelSum) * (kRing + 1), s));
        CHECK(cudaStreamSynchronize(s));
    }

    template <typename Off>
    void launch(int form, int64_t root)
    {
        void (*kern)(const SearchArgs) = form == SEARCH_BLOCK     ? k_search<Off, SEARCH_BLOCK>
                                         : form == SEARCH_CLUSTER ? k_search<Off, SEARCH_CLUSTER>
                                         : form == SEARCH_GRID1   ? k_search<Off, SEARCH_GRID1>
                                                                  : k_search<Off, SEARCH_GRID2>;
        const size_t smem = sizeof(SearchShared) + (form == SEARCH_BLOCK ? (size_t)kBlockVertices / 8 * 4 : 0);
        CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (form == SEARCH_CLUSTER) CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        int per_sm = 0, sms = 0;
        CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSB, smem));
        CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0));
        const int grid = form == SEARCH_BLOCK ? 1 : form == SEARCH_CLUSTER ? kClusterBlocks : sms * per_sm;
        SearchArgs x = a;
        x.root = root;
        x.out = out;
        x.per_warp = x.nwords / ((uint64_t)grid * kSW);
        x.wps = bu_step_words(x.nwords, (uint64_t)grid * kSW);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(kSB);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        cfg.attrs = at;
        cfg.numAttrs = form == SEARCH_BLOCK ? 0 : 1;
        if (form == SEARCH_CLUSTER) {
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = grid;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        } else {
            at[0].id = cudaLaunchAttributeCooperative;
            at[0].val.cooperative = 1;
        }
        CHECK(cudaLaunchKernelEx(&cfg, kern, x));
    }

    std::vector<int64_t> parents()
    {
        std::vector<int64_t> p((size_t)a.n);
        CHECK(cudaMemcpyAsync(p.data(), a.pred, 8 * p.size(), cudaMemcpyDeviceToHost, s));
        CHECK(cudaStreamSynchronize(s));
        return p;
    }
};

int main(int argc, char **argv)
{
    if (argc < 5) return 1;
    FILE *f = std::fopen(argv[2], "rb");
    int64_t size[2];
    if (!f || std::fread(size, 8, 2, f) != 2) return 1;
    std::vector<int64_t> ro((size_t)size[0] + 1);
    std::vector<uint32_t> col((size_t)size[1]);
    if (std::fread(ro.data(), 8, ro.size(), f) != ro.size() || std::fread(col.data(), 4, col.size(), f) != col.size()) return 1;
    std::fclose(f);
    f = std::fopen(argv[3], "wb");
    if (!f) return 1;
    Searcher x(ro, col);
    auto put = [&](const void *p, size_t bytes) { std::fwrite(p, 1, bytes, f); };
    if (!std::strcmp(argv[1], "parents")) {
        for (int wide = 0; wide < 2; ++wide)
            for (int form = SEARCH_BLOCK; form <= SEARCH_GRID2; ++form) {
                if (form == SEARCH_BLOCK && x.a.n > kBlockVertices) continue;
                for (int i = 4; i < argc; ++i) {
                    if (wide) x.launch<int64_t>(form, std::atoll(argv[i]));
                    else x.launch<uint32_t>(form, std::atoll(argv[i]));
                    const std::vector<int64_t> p = x.parents();
                    std::vector<int32_t> lev((size_t)x.a.n);
                    CHECK(cudaMemcpy(lev.data(), x.a.level, 4 * lev.size(), cudaMemcpyDeviceToHost));
                    if (x.out->err) return 3;
                    put(p.data(), 8 * p.size());
                    put(lev.data(), 4 * lev.size());
                }
            }
    } else if (!std::strcmp(argv[1], "clusters")) {
        auto kern = k_search<uint32_t, SEARCH_CLUSTER>;
        CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SearchShared)));
        CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        for (int i = 4; i < argc; ++i) {
            const int64_t fits = cluster_fits((const void *)kern, std::atoi(argv[i]), sizeof(SearchShared));
            CHECK(cudaGetLastError());  // (none left behind)
            put(&fits, 8);
        }
    } else {
        for (int form = SEARCH_GRID1; form <= SEARCH_GRID2; ++form) {
            // arrivals of blocks that are not there: the meeting after the prologue
            // never comes to the grid's number
            const unsigned long long extra = 5ull << kArrive;
            CHECK(cudaMemcpyAsync(&x.a.sums[0].meet[0], &extra, 8, cudaMemcpyHostToDevice, x.s));
            for (int i = 0; i < 3; ++i) {
                if (i == 2) x.clear();
                x.launch<uint32_t>(form, std::atoll(argv[4]));
                const std::vector<int64_t> p = x.parents();
                const int64_t err = x.out->err;
                put(&err, 8);
                put(p.data(), 8 * p.size());
            }
            x.clear();
        }
    }
    std::fclose(f);
    return 0;
}
