// Turns of the batches of a process on one device that step by grids of
// resident blocks (k_steps): the blocks of a grid wait for one another, so two
// grids that each got part of the SMs would wait for ever.  run() queues its
// steps in pieces, each a turn, at most kTurnsAhead of them ahead of the
// GPU.  Grids run side by side while every block of all of them has room:
// blocks of one form (one shared-memory carve-out) whose sum is within what
// fits the GPU.  A piece that does not fit beside those queued by other batches
// waits for them on the GPU, so two systems that fill it alternate.  Ordinary
// kernels (the step graph) end by themselves and need no turn.
//
// Measured on threads with a system each, per step of all, one grid at a time
// against this: eight of 3,000 beads 109 / 20 us (two 27 / 15), eight of 30,000
// (938 blocks of 1,184) 218 / 216; five steps beside another's long run, 3,000
// beads each, all of that run (1,069 ms) / 0.2 ms, 30,000 each 427 / 51.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

namespace fmd {

constexpr int kTurnsAhead = 2;

// A batch's place among those running on its device.
struct TurnTicket {
  TurnTicket() = default;
  TurnTicket(const TurnTicket&) = delete;
  TurnTicket& operator=(const TurnTicket&) = delete;
  ~TurnTicket();
  // The batch's stream has been waited for: nothing of it is queued any more.
  void finished();

  cudaEvent_t done[kTurnsAhead] = {};  // after each of the last turns
  int64_t turns = 0;
  int device = -1;  // on which it is listed
};

// From construction (the stream ordered behind the grids that this one would
// not fit beside) to destruction the caller queues its launch on the stream.
class Turn {
 public:
  Turn(TurnTicket& t, cudaStream_t st, int form, int blocks, int capacity);
  ~Turn();
  Turn(const Turn&) = delete;
  Turn& operator=(const Turn&) = delete;
  bool alone() const { return alone_; }  // no other batch listed

 private:
  TurnTicket& t_;
  cudaStream_t st_;
  bool alone_ = true;
  std::unique_lock<std::mutex> lock_;  // held until the launch is queued
};

}  // namespace fmd
