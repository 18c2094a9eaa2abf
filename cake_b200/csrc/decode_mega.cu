// decode_mega.cu — the instances of the decode kernel (decode_mega.cuh), a translation unit of their own.  sm_100a only.
// Where the kernel's code lies in its module is worth 1 % of a step (two 8B blocks, in turn on one card, six times each, the same kernel source: 177.4 us; 179.4 with
// more kernels of other kinds in its unit; 177.0 here), and in a unit of its own that does not change with the kernels beside it.
#include "decode_mega.cuh"

#include "../../include/cake_b200.h"

namespace cake {

// (head_dim, query heads per kv head) combinations the kernel is instantiated for
#define MK_FOR_ALL(X) X(16, 2) X(16, 4) X(64, 2) X(64, 4) X(128, 1) X(128, 2) X(128, 4) X(128, 8)
template <typename T> static const void *mk_instance(int head_dim, int group) {
#define MK_CASE(HD, G) \
  if (head_dim == HD && group == G) return (const void *)decode_mega_kernel<T, HD, G>;
  MK_FOR_ALL(MK_CASE)
#undef MK_CASE
  return nullptr;
}
const void *mk_kernel(int dtype, int head_dim, int group) {
  if (dtype == CAKE_B200_F32) return nullptr;
  return dtype == CAKE_B200_F16 ? mk_instance<__half>(head_dim, group) : mk_instance<__nv_bfloat16>(head_dim, group);
}

__global__ void __launch_bounds__(MK_CT) mk_wait_probe_kernel(int what, int fresh, int polls, int *err, int *out) {
  __shared__ __nv_bfloat16 xs[4 * MK_CT];
  __shared__ int gave_up;
  alignas(16) static __device__ uint32_t words[4 * MK_CT];
  const int ct = threadIdx.x;
  const uint32_t tag = 7u;
  if (what < 2) {   // packets with this tag, or the one in front
    for (int i = ct; i < 4 * MK_CT; i += MK_CT) words[i] = what ? (fresh ? tag : tag - 1u) : (fresh ? tag : tag - 1u) << 16;
  } else if (ct < 2) {
    words[ct] = 0u;   // a counter
  }
  __threadfence();
  __syncthreads();
  MkWait w{polls, err};
  for (int i = 0; i < 2; i++) {
    if (ct == 0) gave_up = 0;
    __syncthreads();
    unsigned long long *const ctr = reinterpret_cast<unsigned long long *>(words);
    const long long t0 = clock64();
    if (what == 0) mk_gather<__nv_bfloat16>(xs, nullptr, words, 4 * MK_CT, tag << 16, ct, w);
    else if (what == 1) pk_poll64(reinterpret_cast<uint64_t *>(words) + ct, tag, w);
    else if (what == 2) mk_grid_sync(ctr, (unsigned long long)(i + 1) * (fresh ? 1ULL : 2ULL), ct, w);   // this CTA's arrival is the only one
    else if (ct == 0) mk_inbox_wait(ctr, fresh ? 0ULL : 1ULL, w);
    if (w.left <= 0) gave_up = 1;
    __syncthreads();
    if (ct == 0) {
      out[i] = gave_up ? 0 : 1;
      out[2 + i] = (int)((clock64() - t0) / 1000);
    }
  }
}
cudaError_t mk_wait_probe(cudaStream_t st, int what, int fresh, int polls, int *err, int *out) {
  mk_wait_probe_kernel<<<1, MK_CT, 0, st>>>(what, fresh, polls, err, out);
  return cudaGetLastError();
}

}  // namespace cake
