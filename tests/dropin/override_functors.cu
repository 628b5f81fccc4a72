// Functors derived from the bundled ones that override a method: the engine must
// run the override, not an extension the base declares for its own method.
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "sg_apps.cuh"
#include "sg_runtime.cuh"

using namespace sepgraph;

// Two levels per hop.
template <typename TValue, typename TBuffer, typename TWeight, typename... UnusedData>
struct TwoStepBFS : apps::BFS<TValue, TBuffer, TWeight> {
    using Base = apps::BFS<TValue, TBuffer, TWeight>;
    explicit TwoStepBFS(index_t root) : Base(root, false) {}

    __forceinline__ __device__ utils::pair<TBuffer, bool> CombineValueBuffer(index_t node, TValue *p_value,
                                                                            TBuffer *p_buffer) override {
        const TBuffer level = *p_buffer;
        const bool improved = *p_value > level;
        auto r = Base::CombineValueBuffer(node, p_value, p_buffer);
        if (improved) r.first = level + 2;
        return r;
    }
};

using U = uint32_t;
using N = graphs::NoWeight;
template <typename Base>
struct Plain : Base {
    using Base::Base;
};
template <typename Base>
struct OwnCombine : Base {
    using Base::Base;
    __device__ utils::pair<U, bool> CombineValueBuffer(index_t node, U *v, U *b) override {
        return Base::CombineValueBuffer(node, v, b);
    }
};
template <typename Base>
struct OwnBoth : OwnCombine<Base> {
    using OwnCombine<Base>::OwnCombine;
    __device__ utils::pair<U, bool> CombinePull(index_t node, U &v, U &b) const { return Base::CombinePull(node, v, b); }
};
template <typename Base, typename TB>
struct OwnAccumulate : Base {
    using Base::Base;
    using Base::AccumulateBuffer;
    __device__ int AccumulateBuffer(index_t s, index_t d, TB *p, TB b) override { return Base::AccumulateBuffer(s, d, p, b); }
};
using Bfs = apps::BFS<U, U, N>;
using Bc = apps::BCForward<U, U, N>;
using Pr = apps::PageRank<float, float, N>;
using Sssp = apps::SSSP<U, U, U>;
using namespace sepgraph::engine;
static_assert(has_combine_pull<Bfs, U, U>::value && has_combine_pull<Plain<Bfs>, U, U>::value, "inherited");
static_assert(has_combine_pull<Sssp, U, U>::value && has_combine_pull<Pr, float, float>::value, "declared");
static_assert(!has_combine_pull<OwnCombine<Bfs>, U, U>::value, "the override counts");
static_assert(has_combine_pull<OwnBoth<Bfs>, U, U>::value, "declared beside the override");
static_assert(has_take_frontier<Bc>::value && has_take_frontier<Plain<Bc>>::value, "inherited");
static_assert(!has_take_frontier<OwnCombine<Bc>>::value && has_pull_term<OwnCombine<Bc>>::value, "by method");
static_assert(has_pull_term<Bc>::value && !has_pull_term<OwnAccumulate<Bc, U>>::value, "the override counts");
static_assert(has_active_is_pending<Pr>::value && !has_active_is_pending<OwnAccumulate<Pr, float>>::value, "likewise");

int main(int argc, char **argv) {
    if (argc < 4) return 2;
    sg_ctx *ctx = nullptr;
    sg_hgraph *h = nullptr;
    sg_graph *g = nullptr;
    if (sg_init(0, &ctx) != SG_OK ||
        sg_hgraph_gen_rmat((uint32_t)std::atoi(argv[1]), 16, 0.57, 0.19, 0.19, 1, SG_GEN_SYMMETRIC, &h) != SG_OK ||
        sg_graph_create_from_host(ctx, h, SG_GRAPH_SYMMETRIC, &g) != SG_OK)
        return 1;
    for (int pull = 0; pull < 2; ++pull) {  // hybrid policy, then pull rounds alone
        engine::Engine<U, U, N, TwoStepBFS, index_t> e(policy::AlgoType::TRAVERSAL_SCHEME);
        common::EngineOptions opt;
        if (pull) opt.ForceVariant(common::AlgoVariant::ASYNC_PULL_DD);
        e.SetOptions(opt);
        e.LoadGraph(g);
        index_t r = (uint32_t)std::atoi(argv[2]);
        e.InitGraph(r);
        if (e.Start() != SG_OK) return 1;
        const std::vector<U> v = e.GatherValue();
        FILE *f = std::fopen((std::string(argv[3]) + (pull ? "_pull.u32" : "_hybrid.u32")).c_str(), "wb");
        if (!f || std::fwrite(v.data(), sizeof(U), v.size(), f) != v.size()) return 1;
        std::fclose(f);
    }
    sg_graph_destroy(g);
    sg_hgraph_destroy(h);
    sg_destroy(ctx);
    return 0;
}
