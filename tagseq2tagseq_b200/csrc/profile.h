// Optional CUDA-event bracketing of the main kernels (see ts2ts_profile_enable in include/ts2ts_attn.h).
#pragma once
#include <cuda_runtime.h>

namespace ts2ts {

struct ProfileSlot {
  bool enabled = false;
  bool recorded[2] = {false, false};
  cudaEvent_t start[2] = {nullptr, nullptr};
  cudaEvent_t stop[2] = {nullptr, nullptr};
};

ProfileSlot& profile_slot();  // one per device, defined in api.cu

struct ProfileScope {
  ProfileSlot& s;
  int which;
  cudaStream_t stream;
  bool on;  // not inside a stream capture, where an event cannot be timed
  ProfileScope(int which_, cudaStream_t st) : s(profile_slot()), which(which_), stream(st), on(s.enabled) {
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (on && (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone)) on = false;
    if (on) cudaEventRecord(s.start[which], stream);
  }
  ~ProfileScope() {
    if (on) {
      cudaEventRecord(s.stop[which], stream);
      s.recorded[which] = true;
    }
  }
};

}  // namespace ts2ts
