#include "staging.h"

#include <string.h>

#include <algorithm>

#include <omp.h>

#include "common.cuh"

namespace lmb {

namespace {

constexpr size_t kDirect = 2ull << 20;  // below this one cudaMemcpyAsync is as fast

// Page-locked (or managed) memory moves at full speed by itself.
bool page_locked(const void *p) {
  cudaPointerAttributes at{};
  const bool yes = cudaPointerGetAttributes(&at, p) == cudaSuccess && at.type != cudaMemoryTypeUnregistered;
  cudaGetLastError();  // an ordinary pointer is no error here
  return yes;
}

void copy_piece(void *dst, const void *src, size_t bytes) {
  const size_t part = 512 << 10;
  const long parts = (long)((bytes + part - 1) / part);
  const int nt = std::max(1, std::min(16, omp_get_num_procs()));
#pragma omp parallel for schedule(static) num_threads(nt)
  for (long i = 0; i < parts; i++) {
    const size_t at = (size_t)i * part;
    memcpy(static_cast<char *>(dst) + at, static_cast<const char *>(src) + at, std::min(part, bytes - at));
  }
}

}  // namespace

Staging::~Staging() {
  for (int i = 0; i < kPieces; i++) {
    if (buf_[i]) cudaFreeHost(buf_[i]);
    if (ev_[i]) cudaEventDestroy(ev_[i]);
  }
}

bool Staging::ready() {
  for (int i = 0; i < kPieces; i++) {
    cudaError_t e = cudaSuccess;
    if (!buf_[i]) {
      e = cudaHostAlloc(&buf_[i], kPiece, cudaHostAllocDefault);
      if (e != cudaSuccess) buf_[i] = nullptr;
    }
    if (e == cudaSuccess && !ev_[i]) {
      e = cudaEventCreateWithFlags(&ev_[i], cudaEventDisableTiming);
      if (e != cudaSuccess) ev_[i] = nullptr;
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  }
  return true;
}

int Staging::upload(void *dst, const void *src, size_t bytes, cudaStream_t st) {
  if (bytes <= kDirect || page_locked(src) || !ready()) {
    LMB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
    return LMB_OK;
  }
  for (size_t at = 0; at < bytes; at += kPiece) {
    const size_t len = std::min(kPiece, bytes - at);
    const int b = next_;
    next_ = (next_ + 1) % kPieces;
    LMB_CUDA(cudaEventSynchronize(ev_[b]));  // its last copy is through
    copy_piece(buf_[b], static_cast<const char *>(src) + at, len);
    LMB_CUDA(cudaMemcpyAsync(static_cast<char *>(dst) + at, buf_[b], len, cudaMemcpyHostToDevice, st));
    LMB_CUDA(cudaEventRecord(ev_[b], st));
  }
  return LMB_OK;
}

int Staging::download(void *dst, const void *src, size_t bytes, cudaStream_t st) {
  if (bytes <= kDirect || page_locked(dst) || !ready()) {
    LMB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
    LMB_CUDA(cudaStreamSynchronize(st));
    return LMB_OK;
  }
  int rc = LMB_OK;
  const size_t n = (bytes + kPiece - 1) / kPiece;
  auto piece = [&](size_t i) { return std::min(kPiece, bytes - i * kPiece); };
  auto fetch = [&](size_t i) -> int {
    const int b = (int)((next_ + i) % kPieces);
    LMB_CUDA(cudaEventSynchronize(ev_[b]));
    LMB_CUDA(cudaMemcpyAsync(buf_[b], static_cast<const char *>(src) + i * kPiece, piece(i),
                             cudaMemcpyDeviceToHost, st));
    LMB_CUDA(cudaEventRecord(ev_[b], st));
    return LMB_OK;
  };
  for (size_t i = 0; i < std::min<size_t>(n, kPieces); i++)
    if ((rc = fetch(i))) return rc;
  for (size_t i = 0; i < n; i++) {
    const int b = (int)((next_ + i) % kPieces);
    LMB_CUDA(cudaEventSynchronize(ev_[b]));
    copy_piece(static_cast<char *>(dst) + i * kPiece, buf_[b], piece(i));
    if (i + kPieces < n && (rc = fetch(i + kPieces))) return rc;
  }
  next_ = (int)((next_ + n) % kPieces);
  return LMB_OK;
}

}  // namespace lmb
