// Instantiations and launchers of the runtime-radix pass kernel, one object
// per kind (RX_KIND: 1 C2C, 2 R2C, 3 C2R, 4 real-to-real) and form (RX_BS: 1 for
// Bluestein passes).
#include "rx_kernel.cuh"

namespace pb {

template <int KIND>
using RxFn = void (*)(const RxArgs);

template <typename R>
static RxFn<RX_KIND> rx_pick(const RxArgs& X) {
#if RX_BS
  (void)X;
  return rx_kernel<R, RX_KIND, false, true>;
#else
  if constexpr (RX_KIND == P_C2C) {
    if (X.p.dst_k_contig == 0)
      return X.g.ip ? rx_inplace_kernel<R, RX_KIND, true> : rx_kernel<R, RX_KIND, true, false>;
    return X.g.ip ? rx_inplace_kernel<R, RX_KIND, false> : rx_kernel<R, RX_KIND, false, false>;
  } else if constexpr (RX_KIND == P_R2C) {
    return X.g.ip ? rx_inplace_kernel<R, RX_KIND, false> : rx_kernel<R, RX_KIND, false, false>;
  } else {
    return rx_kernel<R, RX_KIND, false, false>;
  }
#endif
}

// the device's whole shared memory: tiles of any length may be launched
template <typename R>
static cudaError_t rx_allow_smem(const RxArgs& X) {
#if RX_BS
  return pb_allow_smem<rx_kernel<R, RX_KIND, false, true>>(X.g.max_smem);
#else
  if constexpr (RX_KIND == P_C2C || RX_KIND == P_R2C) {
    if (X.g.ip) {
      if constexpr (RX_KIND == P_C2C)
        if (X.p.dst_k_contig == 0) return pb_allow_smem<rx_inplace_kernel<R, RX_KIND, true>>(X.g.max_smem);
      return pb_allow_smem<rx_inplace_kernel<R, RX_KIND, false>>(X.g.max_smem);
    }
  }
  if constexpr (RX_KIND == P_C2C)
    if (X.p.dst_k_contig == 0) return pb_allow_smem<rx_kernel<R, RX_KIND, true, false>>(X.g.max_smem);
  return pb_allow_smem<rx_kernel<R, RX_KIND, false, false>>(X.g.max_smem);
#endif
}

template <int KIND, bool BS>
cudaError_t rx_launch_kind(const RxArgs& X, int real_bytes, int grid, cudaStream_t stream);
template <int KIND, bool BS>
int rx_occupancy_kind(const RxArgs& X, int real_bytes);

template <>
cudaError_t rx_launch_kind<RX_KIND, RX_BS>(const RxArgs& X, int real_bytes, int grid, cudaStream_t stream) {
  const auto kern = real_bytes == 4 ? rx_pick<float>(X) : rx_pick<double>(X);
  const cudaError_t err = real_bytes == 4 ? rx_allow_smem<float>(X) : rx_allow_smem<double>(X);
  if (err != cudaSuccess) return err;
  return pb_launch<RxArgs>(kern, grid, X.g.threads, X.g.smem, stream, X);
}

template <>
int rx_occupancy_kind<RX_KIND, RX_BS>(const RxArgs& X, int real_bytes) {
  const auto kern = real_bytes == 4 ? rx_pick<float>(X) : rx_pick<double>(X);
  int blocks = 0;
  if ((real_bytes == 4 ? rx_allow_smem<float>(X) : rx_allow_smem<double>(X)) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, X.g.threads, X.g.smem) != cudaSuccess)
    return 1;
  return blocks > 0 ? blocks : 1;
}

}  // namespace pb
