// ring.h -- parts that arrive in a ring of buffers, emptied by helper threads (host
// only, no CUDA: the device is behind the callbacks).
//
// The calling thread alone sends parts and waits for them; helpers store what has
// arrived. Whoever has to wait looks a bounded number of times and then sleeps, so a
// slow device or a busy host does not have three threads turning. A helper that
// cannot be started, for whatever reason, is done without; with none, the caller stores.
#pragma once
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <mutex>
#include <thread>
#include <vector>

namespace dycg {

constexpr uint32_t RING_HELPERS = 3;
// Yields before a wait sleeps, ~0.3 us each on an idle core: a part of 1 MB takes ~0.02 ms
// to arrive and 0.2-0.3 ms to be stored into fresh pages, so that no wait of a result on
// its way sleeps (at 200 some did, and 8 MB took 0.08 ms more).
constexpr int RING_LOOKS = 2000;

// send(i): queue part i into slot i % slots, 0 or an error; wait(i): until it is
// there, 0 or an error; store(i): take it out of its slot. Returns the first error;
// then what had not arrived was not stored. Only the allocation ahead of the first
// send can throw. Thread: std::thread, or a test's stand-in.
template <class Thread = std::thread, class Send, class Wait, class Store>
int run_ring(uint32_t total, uint32_t slots, Send send, Wait wait, Store store) {
  std::vector<std::atomic<uint8_t>> stored(total);
  for (auto &s : stored) s.store(0, std::memory_order_relaxed);
  std::atomic<uint32_t> arrived{0}, taken{0};
  std::atomic<bool> stop{false};
  std::mutex m;
  std::condition_variable news;
  const auto until = [&](auto ready) {
    for (int k = 0; k < RING_LOOKS; k++) {
      if (ready()) return;
      std::this_thread::yield();
    }
    std::unique_lock<std::mutex> l(m);
    news.wait(l, ready);
  };
  const auto tell = [&]() {
    { std::lock_guard<std::mutex> l(m); }  // (a sleeper looks under the lock)
    news.notify_all();
  };
  const auto store_next = [&]() {  // the next part that nobody has taken; false: none left
    const uint32_t i = taken.fetch_add(1);
    if (i >= total) return false;
    until([&]() { return arrived.load(std::memory_order_acquire) > i || stop.load(); });
    if (arrived.load(std::memory_order_acquire) <= i) return false;
    store(i);
    stored[i].store(1, std::memory_order_release);
    tell();
    return true;
  };
  int x = 0;
  for (uint32_t i = 0; i < slots && i < total && x == 0; i++) x = send(i);
  Thread crew[RING_HELPERS];
  uint32_t helpers = 0;
  try {
    while (helpers < RING_HELPERS && x == 0) {
      crew[helpers] = Thread([&]() {
        while (store_next()) {
        }
      });
      helpers++;
    }
  } catch (...) {
  }
  for (uint32_t i = 0; i < total && x == 0; i++) {
    x = wait(i);
    if (x) break;
    arrived.store(i + 1, std::memory_order_release);
    tell();
    if (!helpers) store_next();
    // slots freed meanwhile (in order) take the parts that follow
    if (i + slots < total) {
      until([&]() { return stored[i].load(std::memory_order_acquire) != 0; });
      x = send(i + slots);
    }
  }
  if (x) stop.store(true);
  tell();
  for (uint32_t t = 0; t < helpers; t++) crew[t].join();
  return x;
}

}  // namespace dycg
