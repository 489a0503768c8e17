// Test driver of the BVH walks' step budget (tests/test_gpu_walk_limit.py): one
// warp whose first lane walks a chain of TLAS nodes whose boxes the ray enters,
// under a budget that may differ from its scene's own.
#include "../hydra_lotus_b200/csrc/scene.cuh"

using namespace lotus;

namespace {

// `round`: through walk_round, as the persistent kernels walk; otherwise
// through traverse, whose budget is the scene's.
__global__ void k_walk(SceneView S, uint32_t limit, int round, uint32_t* steps) {
  uint32_t rng = 1;
  if (!round) {
    Hit hit;
    bool found = false;
    if (threadIdx.x == 0) traverse<false, false, false>(S, V(0.0f), V(0.0f, 0.0f, 1.0f), 0.0f, 1e30f, rng, hit, found);
    return;
  }
  Walk W;
  LocalStore store;
  WalkStack stack;
  bool active = threadIdx.x == 0;
  walk_begin(S, W, store, V(0.0f), V(0.0f, 0.0f, 1.0f), 0.0f, 1e30f);
  for (int k = 0; k < 64 && __any_sync(0xFFFFFFFFu, active); ++k)
    if (walk_round<false, false, false>(S, W, store, stack, rng, limit, active, nullptr)) {
      active = false;
      *steps = W.steps;
    }
}

}  // namespace

// A TLAS of `nodes` nodes, each the only child of the one before and the last
// without children; failure[0..1] are the walk-failure words, failure[2] the
// steps of the round's walk.
extern "C" int walk_chain(int nodes, unsigned scene_limit, unsigned limit, int round, unsigned* failure) {
  if (nodes < 1 || nodes > 32) return -1;
  Bvh4Node host[32];
  for (int i = 0; i < nodes; ++i) {
    const float inf = 3.4e38f, far[4] = {-inf, -inf, -inf, -inf}, near[4] = {inf, inf, inf, inf};
    float4* rows = reinterpret_cast<float4*>(&host[i]);
    for (int a = 0; a < 3; ++a) {
      float4 lo = make_float4(near[0], near[1], near[2], near[3]), hi = make_float4(far[0], far[1], far[2], far[3]);
      if (i + 1 < nodes) {
        lo.x = -1.0f;
        hi.x = 1.0f;
      }
      rows[node_row(i, 2 * a)] = lo;
      rows[node_row(i, 2 * a + 1)] = hi;
    }
    const int4 child = make_int4(i + 1 < nodes ? i + 1 : kEmptyChild, kEmptyChild, kEmptyChild, kEmptyChild);
    reinterpret_cast<int4*>(rows)[node_row(i, 6)] = child;
    reinterpret_cast<int4*>(rows)[node_row(i, 7)] = make_int4(0, 0, 0, 0);
  }
  Bvh4Node* device = nullptr;
  uint32_t* words = nullptr;
  if (cudaMalloc(&device, sizeof(host)) != cudaSuccess || cudaMalloc(&words, 12) != cudaSuccess) return -2;
  cudaMemcpy(device, host, sizeof(Bvh4Node) * nodes, cudaMemcpyHostToDevice);
  cudaMemset(words, 0, 12);
  SceneView S{};
  S.tlas = S.blas = device;
  S.instance_count = 1;
  S.step_limit = scene_limit;
  S.walk_failure = words;
  k_walk<<<1, 32>>>(S, limit, round, words + 2);
  const cudaError_t e = cudaDeviceSynchronize();
  cudaMemcpy(failure, words, 12, cudaMemcpyDeviceToHost);
  cudaFree(words);
  cudaFree(device);
  return e == cudaSuccess ? 0 : (int)e;
}
