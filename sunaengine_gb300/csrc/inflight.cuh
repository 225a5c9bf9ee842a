// Which engines of this process have substeps on a GPU, for the choice between a
// small world's two routes.
//
// The fused substep takes every SM for itself, so engines that run it take turns,
// while the per-phase launches of several small worlds share the GPU. us for one
// substep of each of N engines on streams of their own, fused / per-phase:
//   2D 4 k    N = 2 162 / 163, 4 324 / 179, 8 648 / 204, 16 1300 / 400
//   2D 16 k   N = 2 186 / 192, 4 374 / 239, 8 747 / 347
//   2D 60 k   N = 2 278 / 303, 4 564 / 462, 8 1132 / 856
//   3D 4 k    N = 2 72 / 87, 4 144 / 96, 8 286 / 110
//   3D 60 k   N = 2 157 / 157, 4 313 / 271, 8 629 / 514
// So an engine takes the fused substep while at most one other is in flight
// (FUSED_PEERS), and once three were, not for CROWD_MS, more than a 60 Hz frame: a
// program that queues the substeps of many engines one after the other would start
// two of them on the fused route each time, and the others would wait for those
// (2D 4 k, N = 4, fifty substeps queued on each: 324 without, 179 with). Results do
// not depend on the route.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <chrono>
#include <mutex>
#include <vector>

namespace sn {

constexpr int FUSED_PEERS = 1;
constexpr long long CROWD_MS = 40;

// One engine's part. Its host thread calls begin, queued, idle and crowded; the
// last looks at every other engine's.
class InFlight {
 public:
  InFlight() = default;
  InFlight(const InFlight&) = delete;
  InFlight& operator=(const InFlight&) = delete;
  ~InFlight() { leave(); }
  // `last`: the event the engine records after what it queues
  void join(int device, cudaEvent_t last) {
    Registry& r = registry();
    std::lock_guard<std::mutex> hold(r.m);
    dev = device;
    done = last;
    r.all.push_back(this);
    joined = true;
  }
  // before the event goes
  void leave() {
    if (!joined) return;
    idle();
    Registry& r = registry();
    std::lock_guard<std::mutex> hold(r.m);
    r.all.erase(std::find(r.all.begin(), r.all.end(), this));
    joined = false;
  }
  // substeps are about to be queued; they have been, the event behind them; the
  // stream has been waited for
  void begin() {
    if (state.exchange(QUEUING) == IDLE) ++registry().busy;
  }
  void queued() { state.store(QUEUED); }
  void idle() {
    if (state.load() != IDLE && state.exchange(IDLE) != IDLE) --registry().busy;
  }
  // Whether more than FUSED_PEERS others have substeps on this device, or had a
  // moment ago. (The count alone says no; the events are asked only when it does
  // not, for engines that nobody has waited for since they finished.)
  bool crowded() {
    Registry& r = registry();
    using clock = std::chrono::steady_clock;
    const int most = r.busy.load() - (state.load() != IDLE ? 1 : 0);
    std::atomic<long long>& until = r.until[(unsigned)dev % Registry::DEVICES];
    const long long was = until.load();
    if (most <= FUSED_PEERS && was == 0) return false;
    const long long now = std::chrono::duration_cast<std::chrono::milliseconds>(clock::now().time_since_epoch()).count();
    if (most > FUSED_PEERS && peers() > FUSED_PEERS) {
      until.store(now + CROWD_MS);
      return true;
    }
    return now < was;
  }

 private:
  enum { IDLE, QUEUING, QUEUED };
  struct Registry {
    static constexpr unsigned DEVICES = 64;
    std::mutex m;
    std::vector<InFlight*> all;
    std::atomic<int> busy{0};  // engines not idle, over all devices
    std::atomic<long long> until[DEVICES] = {};  // ms: the end of a device's crowd
  };
  // Other engines with substeps on this one's device.
  int peers() {
    Registry& r = registry();
    int n = 0;
    std::lock_guard<std::mutex> hold(r.m);
    for (InFlight* e : r.all) {
      if (e == this || e->dev != dev) continue;
      int s = e->state.load();
      if (s == QUEUED && cudaEventQuery(e->done) == cudaSuccess && e->state.compare_exchange_strong(s, IDLE)) --r.busy;
      else n += s != IDLE;
    }
    if (cudaPeekAtLastError() == cudaErrorNotReady) cudaGetLastError();  // an answer, not an error
    return n;
  }
  // never destroyed: an engine may outlive the library's other statics
  static Registry& registry() {
    static Registry* r = new Registry;
    return *r;
  }
  std::atomic<int> state{IDLE};
  int dev = 0;
  cudaEvent_t done = nullptr;
  bool joined = false;
};

}  // namespace sn
