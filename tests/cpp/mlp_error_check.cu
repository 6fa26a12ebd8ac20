// Check of what a training call does once a wait for the tensor cores has run
// out: the error word is set by hand, as the kernels set it, and the call has to
// report it and leave the weights and Adam's moments alone; with the word
// cleared, training goes on as on a network that never saw the error.  Includes
// the unit under test for its handle.  Prints "bad 0" and exits 0 when it holds.
#include <cstdio>
#include <cstring>
#include <vector>

#include "fvs_mlp_train.cu"

namespace fvs {
void SetLastError(const std::string&) {}
}  // namespace fvs

namespace {

constexpr int kRows = 4096, kBatch = 1024;

std::vector<float> State(const fvs_mlp* m) {  // master weights and both moments
  std::vector<float> h(3 * fvs::mlp::kParams);
  cudaMemcpy(h.data(), m->buf, h.size() * sizeof(float), cudaMemcpyDeviceToHost);
  return h;
}

bool Same(const std::vector<float>& a, const std::vector<float>& b) {
  return std::memcmp(a.data(), b.data(), a.size() * sizeof(float)) == 0;
}

}  // namespace

int main() {
  std::vector<float> feat(kRows * fvs::mlp::kIn), lab(kRows);
  for (size_t i = 0; i < feat.size(); ++i) feat[i] = float((i * 2654435761u >> 8) % 1000) / 500 - 1;
  for (size_t i = 0; i < lab.size(); ++i) lab[i] = 0.3f * feat[i * fvs::mlp::kIn];
  float *f = nullptr, *l = nullptr;
  if (cudaMalloc(&f, feat.size() * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&l, lab.size() * sizeof(float)) != cudaSuccess)
    return 2;
  cudaMemcpy(f, feat.data(), feat.size() * sizeof(float), cudaMemcpyHostToDevice);
  cudaMemcpy(l, lab.data(), lab.size() * sizeof(float), cudaMemcpyHostToDevice);
  fvs_mlp *a = nullptr, *b = nullptr;
  if (fvs_mlp_create(5, &a) || fvs_mlp_create(5, &b)) return 2;
  int bad = 0;
  float loss = 0.0f;
  auto train = [&](fvs_mlp* m, int steps) {
    return fvs_mlp_train(m, f, l, kRows, steps, kBatch, 1e-3f, 7, &loss);
  };
  auto set_error = [](fvs_mlp* m, int v) {
    cudaMemcpy(m->error, &v, sizeof v, cudaMemcpyHostToDevice);
    cudaDeviceSynchronize();
  };
  bad += train(a, 3) != FVS_OK;
  bad += train(b, 3) != FVS_OK;
  const std::vector<float> before = State(a);
  bad += !Same(before, State(b));
  set_error(a, 1);
  bad += train(a, 4) != FVS_ERR_CUDA;
  bad += !Same(before, State(a));
  set_error(a, 0);
  bad += train(a, 3) != FVS_OK;
  bad += train(b, 3) != FVS_OK;
  bad += Same(before, State(a));
  bad += !Same(State(a), State(b));
  std::printf("bad %d\n", bad);
  fvs_mlp_destroy(a);
  fvs_mlp_destroy(b);
  return bad ? 1 : 0;
}
