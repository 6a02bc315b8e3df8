// The device error flags of a matrix: set here as a kernel whose wait ran out sets them,
// they have to outlive asynchronous calls until a blocking one reports them, once.
#include <cstdio>
#include <vector>

#include "eh_matrix.cuh"

static int failed = 0;
static void expect(eh_status got, eh_status want, const char* what) {
  if (got == want) return;
  printf("%s: %d (%s) instead of %d\n", what, (int)got, eh_last_error(), (int)want);
  failed = 1;
}
static void set_flag(eh_matrix_t m) {
  const uint32_t one = 1;
  cudaDeviceSynchronize();
  cudaMemcpy(reinterpret_cast<eh::Matrix*>(m)->counters + eh::kFlagWord, &one, sizeof(one), cudaMemcpyHostToDevice);
}

int main() {
  const uint32_t n = 6;  // a complete graph
  std::vector<uint64_t> off{0};
  std::vector<uint32_t> nbr;
  for (uint32_t i = 0; i < n; i++) {
    for (uint32_t j = 0; j < n; j++)
      if (i != j) nbr.push_back(j);
    off.push_back(nbr.size());
  }
  eh_matrix_t m = nullptr;
  expect(eh_matrix_build(n, off.data(), nbr.data(), nullptr, EH_SELECT_LOWER, EH_LAYOUT_UINTEGER, nullptr, &m), EH_OK,
         "build");
  uint64_t* out = nullptr;
  cudaMalloc((void**)&out, 4 * sizeof(uint64_t));
  uint64_t count = 0;
  expect(eh_count_triangles(m, &count, nullptr), EH_OK, "triangles");
  for (uint32_t k : {4u, 5u}) {
    set_flag(m);
    expect(eh_count_cliques_async(m, k, out, nullptr), EH_OK, "cliques");
    expect(eh_count_triangles(m, &count, nullptr), EH_ERR_DEVICE_CHECK, "triangles after cliques");
    expect(eh_count_triangles(m, &count, nullptr), EH_OK, "triangles once reported");
    set_flag(m);
    expect(eh_count_cliques(m, k, &count, nullptr), EH_ERR_DEVICE_CHECK, "blocking cliques");
    expect(eh_count_cliques(m, k, &count, nullptr), EH_OK, "cliques once reported");
  }
  eh_matrix_free(m);

  const uint64_t rows[] = {0, n};
  eh_batch_t b = nullptr;
  expect(eh_batch_build(1, rows, n, off.data(), nbr.data(), EH_LAYOUT_UINTEGER, nullptr, &b), EH_OK, "batch");
  expect(eh_batch_matrix(b, &m), EH_OK, "batch matrix");
  cudaStream_t st;
  cudaStreamCreate(&st);
  for (int graph : {0, 1}) {
    expect(eh_batch_run(b, out, out + 1, graph, st), EH_OK, "batch run");
    set_flag(m);
    expect(eh_batch_run(b, out, out + 1, graph, st), EH_OK, "batch run");
    expect(eh_count_triangles(m, &count, st), EH_ERR_DEVICE_CHECK, "triangles of a batch's matrix");
    expect(eh_count_triangles(m, &count, st), EH_OK, "triangles once reported");
  }
  eh_batch_free(b);
  if (!failed) printf("ok\n");
  return failed;
}
