// Device memory that calls without memory of their own borrow and that is kept between calls: one list of blocks
// per (device, stream, kind).  A call has its block to itself while it enqueues; it gives it back right after, because what
// the next borrower of the same stream enqueues is ordered behind it.  Threads that share a stream get
// different blocks.  An allocation and a cudaFree per call cost 0.6 ms of a 0.1 ms feed-forward call (16 rows,
// 4096 x 14336); stream-ordered allocations put three more nodes per product into a captured graph.
//
// While a stream is being captured nothing is allocated and the block that the graph will use is set aside: no
// call outside a capture gets it, and it is never exchanged for a larger one.  At most kKeepBytes are kept in all; a
// call beyond that takes stream-ordered memory for its own duration.  tb_release_workspaces gives everything back.
#include <mutex>
#include <vector>

#include "tb_common.cuh"

namespace tb {

namespace {

constexpr size_t kKeepBytes = (size_t)2 << 30;

struct Block {
  int dev;
  cudaStream_t stream;
  int kind;
  void* ptr;
  size_t bytes;
  bool busy, captured, drop;
};
std::mutex g_mu;
std::vector<Block> g_blocks;

size_t kept_bytes() {
  size_t n = 0;
  for (const Block& b : g_blocks) n += b.bytes;
  return n;
}

}  // namespace

tb_status WorkspaceLease::take(cudaStream_t stream, size_t bytes, int kind) {
  stream_ = stream;
  int dev = 0;
  TB_CUDA_TRY(cudaGetDevice(&dev));
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  TB_CUDA_TRY(cudaStreamIsCapturing(stream, &cap));
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  void* old = nullptr;
  bool keep = false;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    Block *fit = nullptr, *small = nullptr;
    for (Block& b : g_blocks) {
      if (b.dev != dev || b.stream != stream || b.kind != kind || b.busy || b.drop) continue;
      if (b.captured && !capturing) continue;
      if (b.bytes >= bytes && (!fit || (b.captured && !fit->captured) || (b.captured == fit->captured && b.bytes < fit->bytes))) fit = &b;
      if (b.bytes < bytes && !b.captured && !small) small = &b;
    }
    if (fit) {
      fit->busy = true;
      fit->captured = fit->captured || capturing;
      ptr_ = fit->ptr;
      return TB_OK;
    }
    if (!capturing && kept_bytes() - (small ? small->bytes : 0) + bytes <= kKeepBytes) {
      keep = true;
      if (small) {   // exchanged for a larger one
        old = small->ptr;
        *small = g_blocks.back();
        g_blocks.pop_back();
      }
    }
  }
  if (old) {   // earlier calls on the stream may still use it
    TB_CUDA_TRY(cudaStreamSynchronize(stream));
    cudaFree(old);
  }
  if (keep && cudaMalloc(&ptr_, bytes) == cudaSuccess) {
    if (kind == kWorkspaceTickets) {   // the tickets start at zero; every launch leaves them zero
      const cudaError_t e = cudaMemsetAsync(ptr_, 0, kWorkspaceTicketBytes, stream);
      if (e != cudaSuccess) {
        cudaFree(ptr_);
        ptr_ = nullptr;
        return fail(TB_ERR_CUDA, "workspace: %s", cudaGetErrorString(e));
      }
    }
    std::lock_guard<std::mutex> lock(g_mu);
    g_blocks.push_back(Block{dev, stream, kind, ptr_, bytes, true, false, false});
    return TB_OK;
  }
  cudaGetLastError();
  ptr_ = nullptr;
  TB_CUDA_TRY(cudaMallocAsync(&ptr_, bytes, stream));
  own_ = true;
  if (kind == kWorkspaceTickets) TB_CUDA_TRY(cudaMemsetAsync(ptr_, 0, kWorkspaceTicketBytes, stream));
  return TB_OK;
}

WorkspaceLease::~WorkspaceLease() {
  if (!ptr_) return;
  if (own_) {
    cudaFreeAsync(ptr_, stream_);
    return;
  }
  void* gone = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    for (Block& b : g_blocks)
      if (b.ptr == ptr_) {
        b.busy = false;
        if (b.drop) {
          gone = b.ptr;
          b = g_blocks.back();
          g_blocks.pop_back();
        }
        break;
      }
  }
  if (gone) {
    cudaStreamSynchronize(stream_);
    cudaFree(gone);
  }
}

void release_workspaces() {
  std::vector<Block> gone;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    for (size_t i = 0; i < g_blocks.size();) {
      if (g_blocks[i].busy) {   // its call gives it back
        g_blocks[i++].drop = true;
        continue;
      }
      gone.push_back(g_blocks[i]);
      g_blocks[i] = g_blocks.back();
      g_blocks.pop_back();
    }
  }
  int cur = 0;
  cudaGetDevice(&cur);
  for (const Block& b : gone) {
    cudaSetDevice(b.dev);
    cudaDeviceSynchronize();
    cudaFree(b.ptr);
  }
  cudaSetDevice(cur);
}

}  // namespace tb
