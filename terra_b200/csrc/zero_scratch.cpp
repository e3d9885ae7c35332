// fp32 scratch that is handed out zeroed and comes back zeroed, because the last kernel that reads it clears it: the sums and block
// counter of GroupNorm's statistics, the tap-major staging of the convolutions' weight gradients. Cleared by a memory operation for every
// call instead, a small layer waits for the host about 5 us longer per buffer (this / that: residual convolution and GroupNorm of 96 x 180 pixels 171 / 186
// us, a training step of a small model 1946 / 2066).
//
// A buffer belongs to one call from `scratch_take` to `scratch_give`, and to one stream for good: its next user is ordered behind its last by
// the stream, whatever other streams and threads do. A call that fails in between does not give it back, as it may not be zero. Inside a
// capture nothing is taken from here or kept: the graph clears buffers of its own.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "check.h"
#include "torch_ops.h"

namespace {

using torch::Tensor;
using Key = std::tuple<c10::DeviceIndex, c10::StreamId, int64_t>;      // device, stream, elements

// Bounds of what lies here unused; where the next buffer would exceed them, all of it goes back to the allocator.
constexpr size_t MAX_BUFFERS = 64, MAX_BYTES = size_t(256) << 20;

struct Pool {
  std::mutex mutex;
  std::map<Key, std::vector<Tensor>> free;
  size_t buffers = 0, bytes = 0;
};
Pool& pool() {
  static Pool* p = new Pool();      // (not destroyed at exit, when CUDA may be gone)
  return *p;
}

bool capturing(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) == cudaSuccess) return status != cudaStreamCaptureStatusNone;
  cudaGetLastError();
  return true;
}

}  // namespace

namespace terra_ops {

Tensor scratch_take(const Tensor& like, at::IntArrayRef sizes) {
  need(like.is_cuda(), "scratch: a CUDA tensor");
  const c10::cuda::CUDAGuard guard(like.device());
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream();
  int64_t elements = 1;
  for (const int64_t s : sizes) elements *= s;
  Tensor t;      // (outlives the lock: the last reference to a tensor that Python has seen takes the interpreter's)
  if (!capturing(stream.stream())) {
    Pool& p = pool();
    const std::lock_guard<std::mutex> lock(p.mutex);
    const auto it = p.free.find(Key{like.device().index(), stream.id(), elements});
    if (it != p.free.end()) {
      t = std::move(it->second.back());
      it->second.pop_back();
      if (it->second.empty()) p.free.erase(it);
      --p.buffers;
      p.bytes -= t.nbytes();
    }
  }
  if (t.defined()) return t.view(sizes);
  t = torch::empty(sizes, like.options().dtype(torch::kFloat32));
  need(cudaMemsetAsync(t.data_ptr(), 0, t.nbytes(), stream.stream()) == cudaSuccess, "scratch: clearing a new buffer");
  return t;
}

void scratch_give(const Tensor& scratch) {
  const c10::cuda::CUDAGuard guard(scratch.device());
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream();
  const size_t bytes = scratch.nbytes();
  if (bytes > MAX_BYTES || capturing(stream.stream())) return;
  Pool& p = pool();
  std::map<Key, std::vector<Tensor>> dropped;      // (likewise)
  const std::lock_guard<std::mutex> lock(p.mutex);
  if (p.buffers == MAX_BUFFERS || p.bytes + bytes > MAX_BYTES) {
    dropped.swap(p.free);
    p.buffers = p.bytes = 0;
  }
  p.free[Key{scratch.device().index(), stream.id(), scratch.numel()}].push_back(scratch);
  ++p.buffers;
  p.bytes += bytes;
}

}  // namespace terra_ops
