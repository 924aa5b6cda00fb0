// What a CUDA call that fails leaves behind: no error for a later launch check to find and, inside a
// recording, no stream in capture. Prints "ok" or what is wrong.
#include <cstdio>
#include <cstring>

#include "common.cuh"

using namespace gpdhg;

__global__ void add_one(int* p) { *p += 1; }

static int failed_allocation() {   // more than there is
  void* p = nullptr;
  try {
    CK(cudaMalloc(&p, (size_t)1 << 60));
    return std::puts("allocated"), 1;
  } catch (const Error&) {
  }
  return cudaGetLastError() != cudaSuccess ? (std::puts("the error is still there"), 1) : 0;
}

static int failed_capture() {
  cudaStream_t s = nullptr;
  int* p = nullptr;
  CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  CK(cudaMalloc(&p, sizeof(int)));
  CK(cudaMemset(p, 0, sizeof(int)));
  try {
    GraphCapture g(s);
    add_one<<<dim3(1, 70000), 1, 0, s>>>(p);   // refused by the runtime: 65,535 at most
    CK_LAUNCH();
    g.finish();
    return std::puts("captured"), 1;
  } catch (const Error&) {
  }
  if (cudaGetLastError() != cudaSuccess) return std::puts("the error is still there"), 1;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusActive;
  CK(cudaStreamIsCapturing(s, &st));
  if (st != cudaStreamCaptureStatusNone) return std::puts("still capturing"), 1;
  GraphCapture g(s);
  CK(cudaEventRecord(g.fork, s));
  CK(cudaStreamWaitEvent(g.side, g.fork, 0));
  add_one<<<1, 1, 0, g.side>>>(p);
  CK(cudaEventRecord(g.join, g.side));
  CK(cudaStreamWaitEvent(s, g.join, 0));
  add_one<<<1, 1, 0, s>>>(p);
  cudaGraphExec_t ex = g.finish();
  CK(cudaGraphLaunch(ex, s));
  int v = 0;
  CK(cudaMemcpyAsync(&v, p, sizeof(int), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  cudaGraphExecDestroy(ex);
  cudaFree(p);
  cudaStreamDestroy(s);
  return v != 2 ? (std::puts("graph did not run"), 1) : 0;
}

int main(int argc, char** argv) {
  try {
    const int rc = argc > 1 && !std::strcmp(argv[1], "capture") ? failed_capture() : failed_allocation();
    if (!rc) std::puts("ok");
    return rc;
  } catch (const std::exception& e) {
    return std::puts(e.what()), 1;
  }
}
