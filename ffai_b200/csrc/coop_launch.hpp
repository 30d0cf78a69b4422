// What becomes of a call whose fast form is one cooperative launch and whose other form is a chain of plain ones.
// Host code without CUDA calls of its own: the caller passes them in.
#pragma once
#include <cuda_runtime_api.h>

namespace ffai {

enum class CoopLaunch { ran, chain, failed };

// `opt_in` (shared memory of the kernel) and `launch` return a status; `clear` takes a refusal back, so that it is not found
// after a later launch.  All CTAs of a cooperative launch must be resident at once: a process or stream that may use a part of
// the SMs only (an MPS share, a green context) is refused, and the chain runs there.  So it is where the device lacks the
// shared memory.  Any other status is an error of the call.
template <typename OptIn, typename Launch, typename Clear>
CoopLaunch try_cooperative(bool fits, OptIn&& opt_in, Launch&& launch, Clear&& clear, cudaError_t* status) {
    *status = cudaSuccess;
    if (!fits) return CoopLaunch::chain;
    if (!opt_in()) {
        clear();
        return CoopLaunch::chain;
    }
    *status = launch();
    if (*status == cudaSuccess) return CoopLaunch::ran;
    clear();
    const bool refused = *status == cudaErrorCooperativeLaunchTooLarge || *status == cudaErrorLaunchOutOfResources || *status == cudaErrorNotSupported;
    return refused ? CoopLaunch::chain : CoopLaunch::failed;
}

}  // namespace ffai
