// Host-only check of integrator_create's failure paths (csrc/integrator.cu):
// the CUDA runtime is a fake that counts allocations and fails the k-th
// fallible call.  Built with g++; everything the checked path does not reach
// stays unresolved.
#include <set>
#include <stdio.h>
#include <string>

#include "integrator.cu"

static std::set<void*> live;
static int calls, fail_at, wrong_frees;
static bool bad() { return ++calls == fail_at; }
std::string last_error;
void llg_set_error(const std::string& m) { last_error = m; }
void devint_destroy(DevInteg*) {}
extern "C" {
cudaError_t cudaMalloc(void** p, size_t) {
  if (bad()) return cudaErrorMemoryAllocation;
  *p = new char[1];
  live.insert(*p);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (p && !live.erase(p)) wrong_frees++;
  delete[] static_cast<char*>(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) {
  return bad() ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int, size_t, cudaStream_t) {
  return bad() || !live.count(p) ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return bad() ? cudaErrorUnknown : cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

static bool whole(const Integrator* b) {   // every vector allocated, none twice
  std::set<const void*> s;
  size_t n = 0;
  for (int j = 0; j <= b->qmax; j++, n++) s.insert(b->zn[j]);
  for (int j = 0; j <= b->maxl; j++, n++) s.insert(b->V[j]);
  const double* vs[] = {b->ewt, b->acor, b->y, b->tempv, b->delta};
  for (const double* v : vs) { s.insert(v); n++; }
  for (const void* v : s)
    if (!live.count(const_cast<void*>(v))) return false;
  return s.size() == n;
}

#define CHECK(cond)                                                       \
  do {                                                                    \
    if (!(cond)) {                                                        \
      printf("line %d, failing call %d: %s\n", __LINE__, k, #cond);       \
      return 1;                                                           \
    }                                                                     \
  } while (0)

int main() {
  alignas(double) static char y0[8];
  const double* y = reinterpret_cast<const double*>(y0);
  // replaced integrators smaller and larger than the new one, on its stream or not
  const int maxls[3] = {5, 3, 7};
  for (int variant = 0; variant < 3; variant++)
    for (int other_stream = 0; other_stream < 2; other_stream++)
      for (int k = 1;; k++) {
        llg_ctx c{};
        c.neq = 24;
        llg_solver_opts o{};
        o.maxl = maxls[variant];
        calls = 0;
        fail_at = 0;
        CHECK(integrator_create(&c, 0.0, y, &o) == 0 && whole(c.integ));
        Integrator* const old = c.integ;
        old->tn = 1.5;
        if (other_stream) old->stream = reinterpret_cast<cudaStream_t>(y0);
        o.maxl = 5;
        calls = 0;
        fail_at = k;
        const int rc = integrator_create(&c, 0.0, y, &o);
        const bool reached = calls >= k;
        CHECK((rc != 0) == reached);
        // a failed call leaves the old integrator whole, or none at all
        CHECK(!c.integ || whole(c.integ));
        CHECK(rc == 0 || !c.integ || (c.integ == old && old->tn == 1.5));
        size_t held = 0;
        if (c.integ) held = (size_t)c.integ->qmax + 1 + c.integ->maxl + 1 + 5;
        CHECK(live.size() == held);   // nothing leaked
        integrator_destroy(c.integ);
        CHECK(live.empty() && wrong_frees == 0);
        if (!reached) break;
      }
  return 0;
}
