// tf_host.h — host-side helpers of the library that hold no device code: they take the
// runtime calls they make as a parameter, so that a host program can check them.
#pragma once
#include <atomic>
#include <cstddef>
#include <mutex>
#include <vector>

namespace tf {

// A set of launches spread over branch streams.  fork() lets branches 1 .. n - 1 (side) wait
// for the earlier work of the context's stream (branch 0); join() lets that stream wait for
// them.  A scope that is left early, by an error between the two, joins as well: the
// context's next call orders itself after the context's stream alone, so a branch that was
// never joined could still be writing into its buffers.
// Rt: static record(event, stream) and wait(stream, event), both with Status results.
template <typename Rt>
class BranchFork {
  using Stream = typename Rt::Stream;
  using Event = typename Rt::Event;
  using Status = typename Rt::Status;

 public:
  BranchFork(Stream main, const std::vector<Stream>& side, Event fork_ev, const std::vector<Event>& join_ev, int n)
      : main_(main), side_(side), fork_ev_(fork_ev), join_ev_(join_ev), n_(n) {}
  BranchFork(const BranchFork&) = delete;
  BranchFork& operator=(const BranchFork&) = delete;
  ~BranchFork() { join(); }

  Status fork() {
    if (n_ <= 1) return Status{};
    const Status r = Rt::record(fork_ev_, main_);
    if (r != Status{}) return r;
    for (int i = 0; i + 1 < n_; ++i) {
      const Status w = Rt::wait(side_[i], fork_ev_);
      if (w != Status{}) return w;
      forked_ = i + 1;
    }
    return Status{};
  }

  Status join() {
    Status first{};
    for (int i = 0; i < forked_; ++i) {
      Status r = Rt::record(join_ev_[i], side_[i]);
      if (r == Status{}) r = Rt::wait(main_, join_ev_[i]);
      if (first == Status{}) first = r;
    }
    forked_ = 0;
    return first;
  }

 private:
  Stream main_;
  const std::vector<Stream>& side_;
  Event fork_ev_;
  const std::vector<Event>& join_ev_;
  int n_;
  int forked_ = 0;                     // side branches that wait for the context's stream and are not joined yet
};

// Whether a class (la lb|lc ld) has kernel variants to choose from: the thread kernels of up to
// d shells (launch_jk).  The others run one kernel whatever the variant's lower bits.
constexpr bool has_variants(int la, int lb, int lc, int ld) {
  return la <= 2 && (lc + ld == 0 || (lc + ld == 1 && la + lb <= 3) || (lc + ld == 2 && la == 2 && lb == 0));
}

// A value per device, made at the first use on that device: a kernel's launch set-up, which
// holds for one device (function attributes are per device), not for the process.  Several
// threads may ask at once; a value is seen only when it is complete.
template <typename V>
class PerDevice {
  static constexpr int MAX_DEVICES = 64;

 public:
  // make(V&) -> bool: false, it failed (it is tried again at the next use).
  template <typename Make>
  bool get(int device, V& out, Make&& make) {
    if (device < 0 || device >= MAX_DEVICES) return make(out);     // beyond the table: not kept
    if (!ready_[device].load(std::memory_order_acquire)) {
      std::lock_guard<std::mutex> lock(mutex_);
      if (!ready_[device].load(std::memory_order_relaxed)) {
        V v{};
        if (!make(v)) return false;
        value_[device] = v;
        ready_[device].store(true, std::memory_order_release);
      }
    }
    out = value_[device];
    return true;
  }

 private:
  std::mutex mutex_;
  std::atomic<bool> ready_[MAX_DEVICES] = {};
  V value_[MAX_DEVICES] = {};
};

}  // namespace tf
