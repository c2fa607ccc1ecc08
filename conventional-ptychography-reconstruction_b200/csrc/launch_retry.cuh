// launch_retry.cuh -- a kernel launch whose per-device set-up (attributes) may be gone.
//
// Host code without CUDA types, so that it can be compiled and tested alone.
#pragma once

namespace pty {

// set_up(again): sets the kernel's attributes where they are not known to be set, all
// over when `again`; launch(): the launch's own error; last_error(): reads and clears
// the runtime's.  True when the first or the second attempt was queued without error.
// The last error is read after every attempt, or the first one's would be taken for the
// second's, or, after two, for an unrelated call's.
template <class SetUp, class Launch, class LastError>
bool launch_retry(SetUp set_up, Launch launch, LastError last_error) {
  for (int attempt = 0; attempt < 2; ++attempt) {
    if (!set_up(attempt > 0)) {
      last_error();
      return false;
    }
    const bool queued = launch() == 0;
    if (last_error() == 0 && queued) return true;
  }
  return false;
}

}  // namespace pty
