#pragma once
// Which kernels let their successors in the stream start before they have waited for what is in front of them.
// Plain host code, so that the rules can be walked without a GPU.

namespace yan {

// The quantizer as a call of its own.  What it lets start may be a GEMM that loads weights before its own wait, under the caller's
// promise that the call in front of it does not write them: that call is this quantizer, so whatever lies in front of the
// quantizer has to be complete when the GEMM starts.  Without the promise every GEMM waits before it reads anything.
inline bool cast_releases_early(bool constant_weights) { return !constant_weights; }

}  // namespace yan
