// A test-only level-synchronous operator on the frontier engine: hop counts
// from a source, -1 where unreached (the built-in BFS starts its labels at
// mgops::UNSET).
#include "mg_plugin.cuh"

struct Hops {
    static constexpr const char *kTag = "hops";
    static constexpr bool kLevelSync = true, kFirstParent = true, kWeighted = false, kPathCounts = false,
                          kMinPlusBound = false;
    __device__ static __forceinline__ int32_t initialize() { return -1; }
    __device__ static __forceinline__ int32_t source_value() { return 0; }
    __device__ static __forceinline__ int32_t get_partial_result(int32_t src_hops, int32_t) { return src_hops + 1; }
    __device__ static __forceinline__ void accumulate_nonAtomics(int32_t &acc, int32_t data, int32_t) { acc = data; }
    __device__ static __forceinline__ bool update_condition(int32_t old, int32_t, int32_t) { return old < 0; }
    __device__ static __forceinline__ bool fused_update_condition(int32_t *loc, int32_t data, int32_t)
    {
        return atomicCAS(loc, -1, data) == -1;
    }
};

MG_FRONTIER_OPERATOR(mg_hops, Hops)
