// launch.h — kernel launches with programmatic dependent launch (PDL).
//
// Kernels of the integrator's hot loop are launched with the
// programmatic-stream-serialisation attribute and begin with pdl_entry():
// griddepcontrol.wait holds this kernel until the previous one has finished
// and its memory is visible, then griddepcontrol.launch_dependents lets the
// next kernel of the stream be scheduled.  The next launch's set-up therefore
// overlaps the body of the current kernel instead of following it.  Both
// instructions are no-ops for a kernel launched without the attribute.
//
// The order matters.  Triggering before waiting lets kernel C (after B after
// A) be dispatched while A still runs; C's SMs may then keep lines that A
// loaded, and when B rewrites them in place (the Gram-Schmidt update of a
// Krylov vector between its dot products and its normalisation) C reads the
// old values through the non-coherent load path that const __restrict__
// pointers compile to.  Waiting first means a kernel is dispatched only after
// every kernel two places before it in the stream has finished.
//
// That leaves the kernel just before.  C's SMs may keep a line that B loaded
// after C was dispatched and that another block of B then rewrote: B works in
// place, and its blocks' shares meet inside a 32-byte sector (components of an
// odd number of cells, spectrum columns of an odd height, scalar slots next to
// one another).  griddepcontrol.wait covers ordinary loads, not the non-coherent
// path, so such vectors are read past L1 (__ldcg) on one side at least: by the
// in-place kernels whose shares can meet so (k_normalize, k_predict_fused), by
// the readers of the spectrum (k_rows_inv, k_rows_inv64); scalar slots are read
// with ordinary loads.  The other in-place kernels' blocks own whole 256-element
// slices of vectors that start on 256 bytes.
//
// A PDL launch relaxes the dependency on the preceding kernel only, so it is
// used only where every operation of the stream between two such kernels is
// itself a kernel: inside the host integrator's step loop on the legacy
// default stream (PdlScope).  Elsewhere — graph capture, streams that replay
// the demag chain as a graph, set-up copies — g_no_pdl keeps launches plain.


#pragma once
#include <cuda_runtime.h>

extern thread_local int g_no_pdl;
extern thread_local int g_pdl_break;   // the next launch follows a non-kernel operation: plain

// The first launch of a scope follows whatever the caller left on the stream,
// so it is plain too.
struct PdlScope {
  int saved;
  explicit PdlScope(bool on) : saved(g_no_pdl) {
    if (on) g_no_pdl = 0;
    g_pdl_break = 1;
  }
  ~PdlScope() { g_no_pdl = saved; }
};
inline void pdl_break() { g_pdl_break = 1; }

// Shared memory's share of an SM's L1, in percent, for the launches of a scope
// (-1: the driver's choice per kernel).  Kernels that follow one another with
// different shares wait for the SM to drain and be split anew.
extern thread_local int g_carveout;
struct CarveoutScope {
  int saved;
  explicit CarveoutScope(int percent) : saved(g_carveout) { g_carveout = percent; }
  ~CarveoutScope() { g_carveout = saved; }
};

template <typename... KArgs, typename... Args>
inline void klaunch(void (*kernel)(KArgs...), dim3 g, dim3 b, size_t smem, cudaStream_t s, Args... args) {
#ifdef LLG_PLAIN_LAUNCH
  const bool plain = true;
#else
  const bool plain = g_no_pdl || g_pdl_break;
#endif
  if (plain) g_pdl_break = 0;
  if (plain && g_carveout < 0) {
    kernel<<<g, b, smem, s>>>(args...);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = g;
  cfg.blockDim = b;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (!plain) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (g_carveout >= 0) {
    at[n].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at[n++].val.sharedMemCarveout = (unsigned)g_carveout;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

#ifdef __CUDACC__
__device__ __forceinline__ void pdl_entry() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
#endif
