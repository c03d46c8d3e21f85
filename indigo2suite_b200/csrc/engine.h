// Internal interface between the engine's translation units.
#pragma once
#include <cuda_runtime.h>
#include "../../include/i2b200.h"
#include "common.cuh"

namespace i2 {

typedef void (*KernelFn)(Ctx);

int cuda_status(cudaError_t e);
int grid_for(KernelFn fn, int max_per_sm);
// Relax kernels of one algorithm, each set instantiated in a translation unit
// of its own (relax_*.cu, resident_*.cu: they compile in parallel).
// relax_fn: one launch per iteration in style v, whose last block picks the next
// style (`select`) or stays with v; dispatch_fn: one launch per iteration in the
// style the selectors picked; resident_fn: every iteration in one launch, in
// style v or (v < 0) the selectors' per-iteration pick. `wide`: the form compiled
// for more resident blocks per SM (I2_FIXED_MIN_BLOCKS), which the selectors'
// kernels and the edge-balanced style have (engine.cu: wide_form).
template <int ALG>
KernelFn relax_fn(int v, bool select, bool wide);
template <int ALG>
KernelFn dispatch_fn(bool wide);
template <int ALG>
KernelFn resident_fn(int v, bool wide);
KernelFn near_far_kernel(bool resident);  // SSSP with the near/far ordering (relax_sssp.cu, resident_sssp.cu)
KernelFn mis_kernel(bool resident);       // maximal independent set (relax_mis.cu)
const float* mlp_device_params();
int mlp_install(const float* params, int count);

// One traversal of a device graph from one source (srcs_host == nullptr) or
// from nsrc sources at once (batched graphs). The result stays in the graph's
// workspace; one of a small graph may be copied to host_out (nodes ints) with
// the report (i2_graph::staged).
int run_traversal(i2_graph* g, int algo, int src, const int* srcs_host, int nsrc, const i2_opts* opts,
                  i2_report* rep, int* host_out = nullptr);

// True when [p, p + bytes) lies inside one allocation of the current device
// (or managed memory); host pointers and other GPUs' memory are refused.
bool device_range_ok(const void* p, size_t bytes);

// Take ownership of CSR arrays already on the device and build a graph handle.
// `symmetric`: 1 when the lists are known to be sorted and to hold every
// (u, v, w) with its (v, u, w), -1 to have that checked on first need.
int graph_adopt(int nodes, int edges, int* d_nindex, int* d_nlist, int* d_eweight, int symmetric, i2_graph** out);

// Whether g is known to be symmetric (by construction, or checked before).
bool graph_known_symmetric(const i2_graph* g);

// The device CSR arrays of a graph (weights null when it has none).
int graph_device_csr(const i2_graph* g, int* nodes, int* edges, const int** nindex, const int** nlist,
                     const int** eweight);

// A copy of g with its vertices renumbered by descending degree, ties by
// ascending ID (gen_device.cu): *twin is a new graph, *inv (g.nodes ints,
// from dev_alloc) maps each original ID to the copy's.
int degree_ordered_copy(const i2_graph* g, i2_graph** twin, int** inv);

// Copy the last traversal's values to a host array of g.nodes ints.
int graph_copy_result(i2_graph* g, int* host_out, const i2_opts* opts);

// Device memory of graphs (CSR arrays, workspaces, scratch) comes from one
// stream-ordered pool per device that keeps freed blocks reserved: a graph
// uploaded after another was freed reuses that memory instead of paying a
// cudaMalloc and a cudaFree (a change of the device's mappings, milliseconds
// per GB) for every array. dev_alloc returns memory every stream may use;
// dev_free keeps cudaFree's contract (the device finishes its work before the
// block goes back to the pool). Every pointer dev_free gets must come from
// dev_alloc.
cudaError_t dev_alloc_bytes(void** p, size_t bytes);
void dev_free(void* p);
int dev_trim();  // the pool's unused blocks back to the driver; a status
template <class T>
inline cudaError_t dev_alloc(T** p, size_t bytes) {
  return dev_alloc_bytes(reinterpret_cast<void**>(p), bytes);
}

}  // namespace i2
