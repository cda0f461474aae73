// Threads that ask for the same device's value at the same time: one works it out, all read that one,
// and nothing is written once it can be read.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

#include "kpx_once.h"

struct Value {
  int a = 0, b = 0;
};

int main() {
  int bad = 0;
  for (int round = 0; round < 50; ++round) {
    kpx::PerDevice<Value> table;
    std::atomic<int> made{0}, wrong{0}, ready{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
      threads.emplace_back([&] {
        ++ready;
        while (ready < 8) std::this_thread::yield();
        const Value* v = table.get(3, [&](Value& x) {
          x.a = ++made;
          std::this_thread::sleep_for(std::chrono::microseconds(200));
          x.b = x.a;
          return true;
        });
        for (int i = 0; i < 100; ++i) {
          if (!v || v->a != 1 || v->b != 1) ++wrong;
          std::this_thread::sleep_for(std::chrono::microseconds(5));
        }
      });
    for (auto& t : threads) t.join();
    if (made != 1 || wrong != 0) bad = 1;
  }
  kpx::PerDevice<Value> table;
  int calls = 0;
  auto failing = [&](Value&) { return ++calls > 1; };
  if (table.get(0, failing) || !table.get(0, failing) || !table.get(0, failing) || calls != 2) bad = 1;
  if (table.get(-1, failing) || table.get(64, failing)) bad = 1;
  if (bad) std::printf("a value was worked out twice, or read unfinished\n");
  return bad;
}
