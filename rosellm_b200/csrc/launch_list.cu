// Launches noted once and issued again.  What a step launches depends on its sizes alone, and most of a short prompt step's
// time was the host's: 87 calls through the Python binding (conversion of some thirty arguments each, the checks and choices behind
// them) took 0.54 ms for a first token of GPT-2 124M whose kernels run in less.  Here the kernels themselves are
// noted, with their arguments as bytes, and a step of sizes seen before is one call that launches them in a loop.
#include <new>

#include "common.cuh"

// How many kernels the entry points have launched on this host thread (rl_notes_replay's are not among them).
RL_EXPORT int rl_launches_made() { return rl::launches_made; }

// From here on this thread's launches are noted, until rl_notes_end.  0, or -2 when they are being noted already.
RL_EXPORT int rl_notes_begin() {
  if (rl::launch_notes != nullptr) return -2;
  rl::LaunchNotes* notes = new (std::nothrow) rl::LaunchNotes();
  if (notes == nullptr) return -3;
  try {  // room for a step of twelve layers
    notes->launches.reserve(96);
    notes->at.reserve(2048);
    notes->bytes.reserve(64 * 1024);
  } catch (...) {
    delete notes;
    return -3;
  }
  rl::launch_notes = notes;
  return 0;
}

// The notes are complete: a handle for rl_notes_replay and rl_notes_free, or nullptr where a launch could not be noted.
RL_EXPORT void* rl_notes_end() {
  rl::LaunchNotes* notes = rl::launch_notes;
  rl::launch_notes = nullptr;
  if (notes != nullptr && !notes->whole) {
    delete notes;
    return nullptr;
  }
  return notes;
}

RL_EXPORT void rl_notes_free(void* handle) { delete (rl::LaunchNotes*)handle; }

// The noted launches again, on `stream`, in order.  0 or the first error.
RL_EXPORT int rl_notes_replay(void* handle, cudaStream_t stream) {
  constexpr size_t MOST = 64;
  const rl::LaunchNotes& notes = *(const rl::LaunchNotes*)handle;
  for (const rl::NotedLaunch& n : notes.launches) {
    void* params[MOST];
    if (n.n_args > MOST) return -2;
    for (size_t i = 0; i < n.n_args; ++i) params[i] = (void*)(notes.bytes.data() + notes.at[n.first_arg + i]);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = n.grid;
    cfg.blockDim = n.block;
    cfg.dynamicSmemBytes = n.smem;
    cfg.stream = stream;
    cfg.attrs = const_cast<cudaLaunchAttribute*>(n.attrs);
    cfg.numAttrs = n.n_attrs;
    cudaError_t e = cudaLaunchKernelExC(&cfg, n.kernel, params);
    if (e == cudaErrorInvalidValue && n.smem > 48 * 1024) {
      // some kernels have their limit of shared memory set to what each launch needs: a launch since the notes were taken may
      // have lowered it
      cudaGetLastError();
      cudaFuncSetAttribute(n.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n.smem);
      e = cudaLaunchKernelExC(&cfg, n.kernel, params);
    }
    rl::note_launch(e);
  }
  return rl::take_launch_error();
}
