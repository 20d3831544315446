// Arithmetic of rings of buffers: item i of a ring of n buffers is in buffer i % n, and completes phase i / n of its barrier.
// Plain C++, so that it can be looked at without a GPU.
#pragma once
#ifdef __CUDACC__
#define INFLLM_HD __host__ __device__
#else
#define INFLLM_HD
#endif

namespace infllm {

// the last of the first `count` items that is in buffer `b`, -1 if none is
INFLLM_HD constexpr int ring_last(int count, int n, int b) { return count <= b ? -1 : b + (count - 1 - b) / n * n; }
// the parity to wait for until item i has arrived (a barrier passes the parity of the phase that it completed last, and only that)
INFLLM_HD constexpr unsigned ring_parity(int i, int n) { return (unsigned)(i / n) & 1u; }

}  // namespace infllm
