#include "turns.h"

#include <algorithm>
#include <vector>

#include "dev_common.cuh"

namespace fmd {
namespace {

// A batch's queued turns: the largest of them, the event after the last.
struct Entry {
  const TurnTicket* owner;
  int form, blocks, capacity;
  cudaEvent_t last;
};

constexpr int kMaxTurnDevices = 64;
struct Device {
  std::mutex mu;
  std::vector<Entry> running;
};
Device g_devices[kMaxTurnDevices];

void remove(std::vector<Entry>& v, const TurnTicket* owner) {
  v.erase(std::remove_if(v.begin(), v.end(), [&](const Entry& e) { return e.owner == owner; }), v.end());
}

}  // namespace

TurnTicket::~TurnTicket() {
  finished();
  for (auto& e : done)
    if (e) cudaEventDestroy(e);
}

void TurnTicket::finished() {
  if (device < 0) return;
  std::lock_guard<std::mutex> lock(g_devices[device].mu);
  remove(g_devices[device].running, this);
  device = -1;
}

Turn::Turn(TurnTicket& t, cudaStream_t st, int form, int blocks, int capacity) : t_(t), st_(st) {
  int dev = 0;
  FMD_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxTurnDevices) throw Error(FMD_ERR_ARG, "device ordinal out of range");
  cudaEvent_t& ev = t.done[t.turns % kTurnsAhead];
  if (ev)
    FMD_CUDA(cudaEventSynchronize(ev));  // kTurnsAhead turns ago
  else
    FMD_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  lock_ = std::unique_lock<std::mutex>(g_devices[dev].mu);
  std::vector<Entry>& running = g_devices[dev].running;
  int64_t sum = blocks;
  int least = capacity;
  bool fits = true;
  for (Entry& e : running) {
    if (e.owner == &t) {
      // still queued: its other turns of this run, or of one that threw
      if (e.form != form) FMD_CUDA(cudaStreamSynchronize(st));
      else blocks = std::max(blocks, e.blocks);
      continue;
    }
    alone_ = false;
    sum += e.blocks;
    least = std::min(least, e.capacity);
    fits = fits && e.form == form;
  }
  // Grids that run at one time: the last of them to be queued saw all the
  // others here and did not wait for them, so their sum was within the
  // smallest capacity, that of the blocks that take most room.
  if (!fits || sum > least)
    for (const Entry& e : running)
      if (e.owner != &t) FMD_CUDA(cudaStreamWaitEvent(st, e.last, 0));
  remove(running, &t);
  running.push_back(Entry{&t, form, blocks, capacity, ev});
  t.device = dev;
}

Turn::~Turn() {
  cudaEventRecord(t_.done[t_.turns % kTurnsAhead], st_);
  ++t_.turns;
}

}  // namespace fmd
