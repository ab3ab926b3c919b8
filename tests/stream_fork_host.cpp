// StreamFork (csrc/stream_fork.hpp) over fakes of the CUDA calls that it makes:
// each call is written to a log, and the one named by `failing` returns an error.
#include <cstdint>
#include <string>

#include "stream_fork.hpp"

namespace {
std::string calls, failing;
cudaError_t note(const std::string &c) {
  calls += c + ";";
  return c == failing ? cudaErrorLaunchFailure : cudaSuccess;
}
std::string name(const void *p) { return std::string(1, (char)(uintptr_t)p); }
template <class T> T handle(char c) { return (T)(uintptr_t)c; }
}  // namespace

extern "C" {
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return note("record " + name(e) + " on " + name(s)); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { return note(name(s) + " waits " + name(e)); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return note("synchronize " + name(s)); }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }

// streams m (main) and s (side), events f and j; work: 0 ends well, 1 throws.
// The log, with "work;" for the work and "error;" for an exception that leaves.
const char *stream_fork_log(const char *fail, int work) {
  calls.clear();
  failing = fail;
  try {
    pda::StreamFork fork(handle<cudaStream_t>('m'), handle<cudaStream_t>('s'), handle<cudaEvent_t>('f'),
                         handle<cudaEvent_t>('j'));
    calls += "work;";
    if (work == 1) throw pda::Error(PDA_ERR_CUDA, "launch");
    fork.join();
  } catch (const pda::Error &) {
    calls += "error;";
  }
  return calls.c_str();
}
}
