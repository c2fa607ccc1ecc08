// cluster_small.cu -- which cluster kernel (cluster_small.cuh) a call takes.
#include "cluster_small.cuh"

namespace pty {
namespace csm {

template <int M, int CL>
static int launch_m(int mode, int loss, const FusedArgs& a, cudaStream_t s) {
  if (mode == MODE_INTENSITY) return launch<M, CL, MODE_INTENSITY, 0>(a, s);
  const bool adj = mode == MODE_ADJ;
  if constexpr (M > 64)  // (M = 64: small_batch_max)
    if (loss == PTYCHO_LOSS_FD)
      return adj ? launch<M, CL, MODE_ADJ, PTYCHO_LOSS_FD>(a, s) : launch<M, CL, MODE_LOSS, PTYCHO_LOSS_FD>(a, s);
  if constexpr (M < 256 || CL == 16) {  // (portable clusters: FD and intensities alone)
    switch (loss) {
      case PTYCHO_LOSS_SMOOTH_L1:
        return adj ? launch<M, CL, MODE_ADJ, PTYCHO_LOSS_SMOOTH_L1>(a, s)
                   : launch<M, CL, MODE_LOSS, PTYCHO_LOSS_SMOOTH_L1>(a, s);
      case PTYCHO_LOSS_POISSON:
        return adj ? launch<M, CL, MODE_ADJ, PTYCHO_LOSS_POISSON>(a, s)
                   : launch<M, CL, MODE_LOSS, PTYCHO_LOSS_POISSON>(a, s);
      case PTYCHO_LOSS_INTENSITY_GRAD:
        return adj ? launch<M, CL, MODE_ADJ, PTYCHO_LOSS_INTENSITY_GRAD>(a, s)
                   : launch<M, CL, MODE_LOSS, PTYCHO_LOSS_INTENSITY_GRAD>(a, s);
    }
  }
  return PTYCHO_ERR_UNSUPPORTED_SIZE;
}

}  // namespace csm

bool large_clusters() {
  static PtyDevCache cache;  // 1: no, 2: yes
  int dev = 0, v = cache.get(&dev);
  if (dev < 0) return true;
  if (!v) {
    v = csm::fits<256, 16, MODE_ADJ, PTYCHO_LOSS_FD>() ? 2 : 1;  // the most shared memory and registers of them all
    cache.put(dev, v);
  }
  return v == 2;
}

int launch_small(int M, int mode, int loss, const FusedArgs& a, cudaStream_t s) {
  if (M == 64) return csm::launch_m<64, 4>(mode, loss, a, s);
  if (M == 128) return csm::launch_m<128, 8>(mode, loss, a, s);
  return large_clusters() ? csm::launch_m<256, 16>(mode, loss, a, s) : csm::launch_m<256, 8>(mode, loss, a, s);
}

}  // namespace pty
