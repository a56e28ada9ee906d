// chunk_graph.h -- a chunk of solver iterations as a CUDA graph.
//
// Every launch of an iterative solve is the same (the iteration state is on
// the device), so one capture serves every chunk of this and of later solves
// with the same kernel arguments, which are the key.  At most kMost are kept;
// the oldest goes first.
#pragma once
#include <cuda_runtime.h>

#include <cstring>
#include <vector>

namespace chdwf {

#ifdef __CUDACC__
// At the start of a kernel launched with programmatic serialisation: all that
// the kernels before it wrote is visible, and the next one may be scheduled.
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

struct ChunkGraphs {
    static constexpr size_t kMost = 16;
    struct G {
        std::vector<unsigned char> key;
        cudaGraphExec_t exec = nullptr;
    };
    std::vector<G> g;
    void release() {
        for (G& x : g)
            if (x.exec) cudaGraphExecDestroy(x.exec);
        g.clear();
    }
    ~ChunkGraphs() { release(); }
    // args: plain data with its padding cleared; launch() queues the chunk on
    // st.  Null: not captured, the caller launches directly.
    template <class A, class F>
    cudaGraphExec_t get(const A& args, int variant, cudaStream_t st, F&& launch) {
        std::vector<unsigned char> key(sizeof(args) + sizeof(int));
        memcpy(key.data(), &args, sizeof(args));
        memcpy(key.data() + sizeof(args), &variant, sizeof(int));
        for (const G& x : g)
            if (x.key == key) return x.exec;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            launch();
            if (cudaStreamEndCapture(st, &graph) == cudaSuccess && graph) {
                if (cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) exec = nullptr;
                cudaGraphDestroy(graph);
            }
        }
        cudaGetLastError();
        if (!exec) return nullptr;
        if (g.size() >= kMost) {
            if (g[0].exec) cudaGraphExecDestroy(g[0].exec);
            g.erase(g.begin());
        }
        g.push_back(G{key, exec});
        return exec;
    }
};

}  // namespace chdwf
