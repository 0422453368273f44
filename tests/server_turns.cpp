// Drives the serving loop (csrc/host/server.cpp) on the CPU: the CUDA runtime
// and the engine calls are stand-ins that count the CTAs of the cooperative
// launches in progress. Usage: server_turns WORKERS OVERLAP; prints the largest
// sum of CTAs and the largest number of launches at one time.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "mosp_b200.h"

namespace {
constexpr int kSms = 148;
std::atomic<int> ctasNow{0}, ctasMost{0}, launchesNow{0}, launchesMost{0};

void raise(std::atomic<int> &most, int x) {
  int old = most.load();
  while (old < x && !most.compare_exchange_weak(old, x)) {
  }
}
}  // namespace

struct mosp_workspace {
  int grid = 0;
};

namespace {
int launch(mosp_workspace *ws) {
  const int ctas = ws->grid > 0 && ws->grid < kSms ? ws->grid : kSms;
  raise(ctasMost, ctasNow.fetch_add(ctas) + ctas);
  raise(launchesMost, launchesNow.fetch_add(1) + 1);
  std::this_thread::sleep_for(std::chrono::milliseconds(2));
  launchesNow.fetch_sub(1);
  ctasNow.fetch_sub(ctas);
  return MOSP_OK;
}
}  // namespace

namespace mospb200 {
int recordFailure(int status, const char *) { return status; }
}  // namespace mospb200

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = kSms, cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t bytes) { return *p = std::calloc(bytes, 1), cudaSuccess; }
cudaError_t cudaFree(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { return *p = std::calloc(bytes, 1), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void *to, const void *from, size_t bytes, cudaMemcpyKind) {
  return std::memcpy(to, from, bytes), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t bytes, cudaMemcpyKind, cudaStream_t) {
  return std::memcpy(to, from, bytes), cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *a, size_t *b) { return *a = *b = size_t(1) << 40, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }

const char *mosp_last_error(void) { return ""; }
long long mosp_default_delta(long long, int, long long) { return 1; }
long long mosp_preference_scale(const int *, int) { return 1; }
int mosp_workspace_create(mosp_workspace **out) { return *out = new mosp_workspace(), MOSP_OK; }
void mosp_workspace_destroy(mosp_workspace *ws) { delete ws; }
int mosp_workspace_reserve_graph(mosp_workspace *, int, long long, int) { return MOSP_OK; }
int mosp_workspace_set_canonical_trees(mosp_workspace *, int) { return MOSP_OK; }
int mosp_workspace_set_grid(mosp_workspace *ws, int ctas, int) { return ws->grid = ctas, MOSP_OK; }
int mosp_apply_batch_device(mosp_workspace *ws, int, int K, int m, const int *, const int *, const int *, int n_ins,
                            const int *, const int *, const int *, int, const int *, const int *, int *, int *,
                            int *, long long, int *new_m, unsigned *, long long *most, long long *sum, void *) {
  *new_m = m + n_ins;
  for (int k = 0; k < K; ++k) most[k] = sum[k] = 1;
  return launch(ws);
}
int mosp_build_device_graph(mosp_workspace *ws, int, int, int, const int *, const int *, const int *, int *, int *,
                            int *, int *, void *) {
  return launch(ws);
}
int mosp_update_device(mosp_workspace *ws, int, int, int, const int *, const int *, const int *, const int *,
                       const int *, const int *, const int *, const int *, const int *, const int *, int, int,
                       const long long *, const long long *, const int *, long long *, int *, long long *, int *,
                       mosp_sosp_stats *, mosp_combine_stats *, void *) {
  return launch(ws);
}
int mosp_sosp_from_scratch(mosp_workspace *ws, int, int, const int *, const int *, const int *, int, long long,
                           long long, long long *, int *, mosp_sosp_stats *, void *) {
  return launch(ws);
}
int mosp_combined_sosp(mosp_workspace *ws, int, int, const int *, const int *, int, long long, long long *, int *,
                       mosp_combine_stats *, void *) {
  return launch(ws);
}
}  // extern "C"

int main(int argc, char **argv) {
  if (argc != 3) return 2;
  const int workers = std::atoi(argv[1]), graphs = workers + 1;
  mosp_server *srv = nullptr;
  if (mosp_server_create(workers, 0, 1, &srv) != MOSP_OK) return 1;
  mosp_server_set_overlap(srv, std::atoi(argv[2]));
  const int row[3] = {0, 1, 1}, col[1] = {1}, w[1] = {5};
  auto add = [&] {
    int id = 0;
    if (mosp_server_add_graph(srv, 2, 1, 1, row, col, w, 1, 0, nullptr, &id) != MOSP_OK) std::exit(1);
    return id;
  };
  std::vector<int> ids;
  for (int i = 0; i < graphs; ++i) ids.push_back(add());
  std::vector<long long> tickets;
  const int from = 0, to = 1;
  for (int round = 0; round < 12; ++round) {
    for (int id : ids) {
      long long t = 0;
      if (mosp_server_submit(srv, id, 1, &from, &to, w, 1, &from, &to, &t) != MOSP_OK) return 1;
      tickets.push_back(t);
    }
    if (round == 4) add();  // a graph comes in while passes run
  }
  for (long long t : tickets) {
    mosp_server_result info{};
    if (mosp_server_wait(srv, t, nullptr, nullptr, &info) != MOSP_OK || info.status != MOSP_OK) return 1;
  }
  mosp_server_destroy(srv);
  std::printf("%d %d\n", ctasMost.load(), launchesMost.load());
  return 0;
}
