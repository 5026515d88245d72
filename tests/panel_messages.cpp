// Runs the panel leaf's message rules (panel_msgs.h) on host threads, a CTA each,
// against a model of an mbarrier that reports what the PTX ISA leaves undefined.
//   panel_messages N_CTA COLUMNS LOST RULES
// LOST: -1, or the column whose message from the last CTA to the first never
// arrives.  RULES: 1, or 0 to arm and send whatever happened (the model must object).
// Exit status: 0, 1 undefined use of a barrier, 2 a column of an undisturbed run
// missed, 3 a loss that nobody noticed.
#include <atomic>
#include <barrier>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>

#include "panel_msgs.h"

namespace {

constexpr int  kMessage = 32 * 8 + 16;  // bytes of a candidate
std::chrono::milliseconds budget{40};
std::atomic<bool> undefined{false};

class Mbarrier {
 public:
  void arrive_expect(int bytes) {
    std::lock_guard<std::mutex> l(mu_);
    if(pending_ == 0) undefined = true;  // one arrival per phase
    tx_ += bytes;
    pending_ -= 1;
    settle();
  }
  void complete(int bytes) {
    std::lock_guard<std::mutex> l(mu_);
    tx_ -= bytes;
    settle();
  }
  bool done(unsigned parity) {
    std::lock_guard<std::mutex> l(mu_);
    return (phase_ & 1u) != parity;
  }

 private:
  void settle() {
    if(std::abs(tx_) >= 1 << 20) undefined = true;
    if(pending_ == 0 && tx_ == 0) {
      phase_ += 1;
      pending_ = 1;
    }
  }
  std::mutex mu_;
  int        pending_ = 1, tx_ = 0;
  unsigned   phase_ = 0;
};

struct Ring {
  Mbarrier          full[hplb::kBufs];
  std::atomic<bool> gave_up{false};
  int               ctas = 0, missed = 0;

  bool wait(int buf, unsigned parity) {
    const auto t0 = std::chrono::steady_clock::now();
    while(!full[buf].done(parity)) {
      if(gave_up) return false;
      if(std::chrono::steady_clock::now() - t0 > budget) {
        gave_up = true;
        return false;
      }
      std::this_thread::yield();
    }
    return true;
  }
  bool expired() const { return gave_up; }
  void arm(int buf) { full[buf].arrive_expect(ctas * kMessage); }
};

}  // namespace

int main(int argc, char** argv) {
  if(argc != 5) return 64;
  const int  ctas = std::atoi(argv[1]), columns = std::atoi(argv[2]), lost = std::atoi(argv[3]);
  const bool rules = std::atoi(argv[4]) != 0;
  if(lost < 0) budget = std::chrono::seconds(30);  // nothing should expire
  std::vector<Ring> rings(ctas);
  std::barrier      cluster(ctas);
  for(auto& r : rings) r.ctas = ctas;
  auto cta = [&](int me) {
    Ring& r = rings[me];
    for(int b = 0; b < hplb::kBufs; ++b) r.arm(b);
    cluster.arrive_and_wait();
    auto send = [&](int col) {
      if(rules && !hplb::may_send(r)) return;
      for(int to = 0; to < ctas; ++to)
        if(!(col == lost && me == ctas - 1 && to == 0))
          rings[to].full[col % hplb::kBufs].complete(kMessage);
    };
    for(int k = 0; k < columns; ++k) {
      const bool first = k % 32 == 0, last = k % 32 == 31 || k + 1 == columns;  // leaves of 32
      if(first) send(k);
      const bool arrived = hplb::await_column(r, (unsigned)k);
      r.missed += !arrived;
      if(!last) send(k + 1);
      if(rules)
        hplb::rearm(r, (unsigned)k, arrived);
      else
        r.arm(k % hplb::kBufs);
      if(last) cluster.arrive_and_wait();
    }
  };
  std::vector<std::thread> threads;
  for(int c = 0; c < ctas; ++c) threads.emplace_back(cta, c);
  for(auto& t : threads) t.join();
  int missed = 0;
  for(auto& r : rings) missed += r.missed;
  std::printf("missed %d undefined %d\n", missed, (int)undefined);
  if(undefined) return 1;
  if(lost < 0 && missed != 0) return 2;
  return lost >= 0 && missed == 0 ? 3 : 0;
}
