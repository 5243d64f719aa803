// A stand-in for the CUDA runtime, preloaded into a CPU process by
// test_nv_queue_host.py: memory is the host's, kernels do nothing, and a
// kernel that hands values to the host hands over one constant.  It records
// the launches of the N_Vector queue and can refuse one of them, or one of all.
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "nv_queue.h"

namespace {
double g_value = 1e-3;
long g_refuse = -1, g_flushes = 0, g_refuse_any = -1, g_launches = 0;
int g_last = 0;
std::vector<const unsigned int *> g_words;
std::map<const void *, std::string> &names() {
  static std::map<const void *, std::string> n;
  return n;
}

int launch(const void *func, void **args) {
  const std::string &name = names()[func];
  if (g_launches++ == g_refuse_any) return g_last = 999;
  double *host = nullptr;
  uint64_t *word = nullptr, seq = 0;
  if (name.find("k_seq") != std::string::npos) {
    const pihm_nv::Seq &q = *(const pihm_nv::Seq *)args[0];
    if (!q.host_seq) {
      if (g_flushes++ == g_refuse) return g_last = 999;
      return 0;
    }
    g_words.push_back(q.word);
    host = q.host;
    word = q.host_seq;
    seq = q.seq;
    for (int k = 0; k < q.fetch; k++) host[2 + k] = g_value;
  } else if (name.find("k_red") != std::string::npos) {
    host = *(double **)args[9];
    word = *(uint64_t **)args[10];
    seq = *(uint64_t *)args[11];
  } else if (name.find("k_status") != std::string::npos) {
    (*(uint64_t **)args[1])[0] = **(unsigned int **)args[0];
    (*(uint64_t **)args[1])[1] = *(uint64_t *)args[2];
  }
  if (!word) return 0;
  host[0] = host[1] = g_value;
  __atomic_store_n(word, seq, __ATOMIC_RELEASE);
  return 0;
}
struct Dim {
  unsigned x, y, z;
};
}  // namespace

extern "C" {
void fake_refuse(long flush) { g_refuse = flush; }
long fake_flushes() { return g_flushes; }
void fake_refuse_any(long launch) { g_refuse_any = launch; }
long fake_launches() { return g_launches; }
void fake_reset() {
  g_flushes = g_launches = 0;
  g_words.clear();
}
long fake_words(uint64_t *out, long n) {
  for (long k = 0; k < n && k < (long)g_words.size(); k++) out[k] = (uint64_t)g_words[k];
  return (long)g_words.size();
}

// what a library's kernels are called (the rest of their registration is the
// CUDA runtime's)
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *,
                            int *) {
  names()[host] = name;
}
int cudaLaunchKernelExC(const void *, const void *func, void **args) { return launch(func, args); }
int cudaLaunchKernel(const void *func, Dim, Dim, void **args, size_t, void *) { return launch(func, args); }
int __cudaGetKernel(const void **kernel, const void *func) {
  *kernel = func;
  return 0;
}
int __cudaLaunchKernel(const void *kernel, Dim, Dim, void **args, size_t, void *) { return launch(kernel, args); }
int cudaGetLastError() {
  const int e = g_last;
  g_last = 0;
  return e;
}
int cudaMalloc(void **p, size_t n) { return (*p = std::calloc(n ? n : 1, 1)) ? 0 : 2; }
int cudaFree(void *p) {
  std::free(p);
  return 0;
}
int cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
int cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
int cudaFreeHost(void *p) { return cudaFree(p); }
int cudaMemset(void *p, int v, size_t n) {
  std::memset(p, v, n);
  return 0;
}
int cudaMemsetAsync(void *p, int v, size_t n, void *) { return cudaMemset(p, v, n); }
int cudaMemcpy(void *d, const void *s, size_t n, int) {
  std::memcpy(d, s, n);
  return 0;
}
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *) { return cudaMemcpy(d, s, n, k); }
int cudaStreamSynchronize(void *) { return 0; }
int cudaDeviceSynchronize() { return 0; }
int cudaGetDevice(int *d) { return *d = 0; }
int cudaDeviceGetAttribute(int *v, int attr, int) {
  *v = attr == 16 ? 152 : (attr == 95 ? 1 : 0);  // SMs; cooperative launch
  return 0;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
  *n = 1;
  return 0;
}
}
