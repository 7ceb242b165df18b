// edk_handles.cu — cuBLAS and cuSOLVER handles shared by the bases (entanglement
// spectra) and operators (block Lanczos) of a process.  Creating a pair costs
// milliseconds, more than an entanglement spectrum of 1,024 values, so a call
// borrows one and gives it back; at most kKept idle pairs stay per device, and
// all go when the last object that borrowed one is destroyed.
#include <cublas_v2.h>
#include <cusolverDn.h>

#include <map>

#include "edk_internal.cuh"

namespace edk {

namespace {

constexpr size_t kKept = 4;
std::mutex g_mu;
std::map<int, std::vector<LibHandles>> g_idle;  // by device
int64_t g_users = 0;

void destroy(const LibHandles& h) {
  if (h.blas) cublasDestroy(static_cast<cublasHandle_t>(h.blas));
  if (h.solver) cusolverDnDestroy(static_cast<cusolverDnHandle_t>(h.solver));
}

}  // namespace

HandleLease::~HandleLease() {
  if (!h.blas && !h.solver) return;
  cudaStreamSynchronize(stream);  // (idle already, except after an error)
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto& idle = g_idle[device];
    if (g_users > 0 && idle.size() < kKept) {
      idle.push_back(h);
      return;
    }
  }
  destroy(h);
}

// The calls of one lease run on `st`; they are finished when it ends.
edk_status HandleLease::take(bool& registered, cudaStream_t st) {
  stream = st;
  EDK_TRY_CUDA(cudaGetDevice(&device));
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!registered) {
      registered = true;
      ++g_users;
    }
    auto& idle = g_idle[device];
    if (!idle.empty()) {
      h = idle.back();
      idle.pop_back();
    }
  }
  if (!h.blas) {
    cublasHandle_t b = nullptr;
    if (cublasCreate(&b) != CUBLAS_STATUS_SUCCESS) {
      set_error("cublasCreate failed");
      return EDK_CUDA_ERROR;
    }
    h.blas = b;
  }
  if (cublasSetStream(static_cast<cublasHandle_t>(h.blas), st) != CUBLAS_STATUS_SUCCESS) {
    set_error("cublasSetStream failed");
    return EDK_CUDA_ERROR;
  }
  return EDK_OK;
}

edk_status HandleLease::add_solver() {
  if (!h.solver) {
    cusolverDnHandle_t s = nullptr;
    if (cusolverDnCreate(&s) != CUSOLVER_STATUS_SUCCESS) {
      set_error("cusolverDnCreate failed");
      return EDK_CUDA_ERROR;
    }
    h.solver = s;
  }
  if (cusolverDnSetStream(static_cast<cusolverDnHandle_t>(h.solver), stream) !=
      CUSOLVER_STATUS_SUCCESS) {
    set_error("cusolverDnSetStream failed");
    return EDK_CUDA_ERROR;
  }
  return EDK_OK;
}

void handles_unregister(bool registered) {
  if (!registered) return;
  std::map<int, std::vector<LibHandles>> gone;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (--g_users == 0) gone.swap(g_idle);
  }
  for (auto& kv : gone)
    for (auto& h : kv.second) destroy(h);
}

}  // namespace edk
