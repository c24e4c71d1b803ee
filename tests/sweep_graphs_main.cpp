// Runs of sweeps only on an engine: prints, per number of sweeps, the ticks'
// CUDA graphs captured and replayed, and whether the labels and sums are those
// of the same sweeps issued without graphs.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "engine.h"

using namespace sbp;

int main(int argc, char** argv) {
  const int32_t N = 3000, K = 6, B = 20;
  std::vector<int32_t> ptr(N + 1), out((size_t)N * K), in((size_t)N * K), part(N);
  std::vector<uint32_t> w((size_t)N * K, 1u), deg(N, K);
  const int32_t step[K] = {1, 7, 20, 40, 300, 1111};  // most neighbours in v's own block
  for (int32_t v = 0; v < N; ++v) {
    ptr[v + 1] = (v + 1) * K;
    part[v] = (v * 7 + v / 64) % B;
    for (int k = 0; k < K; ++k) {
      out[(size_t)v * K + k] = (v + step[k]) % N;
      in[(size_t)v * K + k] = (v + N - step[k]) % N;
    }
  }
  const sbp_graph_csr g{N, N * K, ptr.data(), out.data(), w.data(), ptr.data(),
                        in.data(), w.data(), deg.data(), deg.data()};
  const int32_t nb = 4;
  Engine eng;
  if (eng.init(0) != SBP_OK) return 2;
  for (int a = 1; a < argc; ++a) {
    const int32_t sweeps = std::atoi(argv[a]);
    std::vector<double> sums[2];
    std::vector<int32_t> labels[2];
    long long captures = 0, replays = 0;
    for (int graphs = 0; graphs < 2; ++graphs) {
      Job J;
      if (job_create(J, 0, N, N * K, 1, nb * sweeps, 4096) != SBP_OK) return 2;
      if (job_upload(J, &g) != SBP_OK) return 2;
      cudaMemcpy(J.part, part.data(), 4 * (size_t)N, cudaMemcpyHostToDevice);
      if (cudaStreamSynchronize(J.st) != cudaSuccess) return 2;
      Run r;
      r.J = &J;
      sbp_default_options(&r.o);
      r.o.num_batches = nb;
      r.o.use_graphs = graphs;
      sums[graphs].resize((size_t)nb * sweeps);
      labels[graphs].resize(N);
      r.sums_out = sums[graphs].data();
      r.labels_out = labels[graphs].data();
      r.start_sweeps(B, 5, sweeps);
      captures = -eng.graph_captures;
      replays = -eng.graph_replays;
      eng.runs.push_back(&r);
      while (r.stage != Run::kDone)
        if (eng.tick() != SBP_OK) return 2;
      eng.reset();
      captures += eng.graph_captures;
      replays += eng.graph_replays;
    }
    std::printf("%d %lld %lld %d %d\n", sweeps, captures, replays,
                (int)(sums[0] == sums[1] && labels[0] == labels[1]), (int)(labels[0] != part));
  }
  return 0;
}
