// copy_pool_check.cpp -- CPU check of cpsz_b200/csrc/copy_pool.h (test
// infrastructure, built and run by tests/test_copy_pool.py): every piece of a
// job is copied once and before wait() returns; jobs of several threads run
// beside one another, also while one owner waits for something else between
// its pieces; idle workers use no processor time; a dropped job leaves none of
// its pieces running.
#include <sys/resource.h>

#include <chrono>
#include <cstdio>
#include <cstring>

#include "copy_pool.h"

using namespace cpsz;
using Clock = std::chrono::steady_clock;

static double ms_since(Clock::time_point t) { return std::chrono::duration<double, std::milli>(Clock::now() - t).count(); }
static double cpu_ms() {
  rusage u;
  getrusage(RUSAGE_SELF, &u);
  return 1e3 * (u.ru_utime.tv_sec + u.ru_stime.tv_sec) + 1e-3 * (u.ru_utime.tv_usec + u.ru_stime.tv_usec);
}

static int fails = 0;
static void expect(bool ok, const char* what) {
  if (!ok) fails++;
  printf("%s %s\n", ok ? "ok" : "FAIL", what);
}

// pieces of `bytes` through a ring of `slots`, opened as the ring has room
static bool ring_job(CopyPool& pool, int pieces, size_t bytes, int slots) {
  std::vector<char> src(pieces * bytes), dst(pieces * bytes, 0), ring(slots * bytes);
  for (size_t i = 0; i < src.size(); i++) src[i] = (char)(i * 31 + i / 4093);
  std::vector<std::atomic<int>> times(pieces);
  for (auto& t : times) t = 0;
  auto work = [&](int k) {
    memcpy(&ring[(k % slots) * bytes], &src[k * bytes], bytes);
    times[k]++;
  };
  CopyPool::Job job(pool, work);
  for (int k = 0; k < pieces; k++) {
    job.open(std::min(pieces, k + slots));
    job.wait(k);
    memcpy(&dst[k * bytes], &ring[(k % slots) * bytes], bytes);
  }
  for (auto& t : times)
    if (t != 1) return false;
  return src == dst;
}

static void all(int workers) {
  CopyPool pool(workers);
  printf("%d workers\n", workers);
  expect(ring_job(pool, 200, 5000, 32), "a job through a ring");
  expect(ring_job(pool, 1, 1, 1), "one byte");

  {  // the owner helps, nothing is left over
    std::atomic<int> n{0};
    auto work = [&](int) { n++; };
    {
      CopyPool::Job job(pool, work);
      job.open(1000);
      job.help();
    }
    expect(n == 1000, "every open piece is copied when the owner helps");
  }
  {  // jobs of four threads beside one another
    std::atomic<int> good{0};
    std::vector<std::thread> t;
    for (int i = 0; i < 4; i++)
      t.emplace_back([&] {
        for (int r = 0; r < 20; r++) good += ring_job(pool, 60, 20000, 32);
      });
    for (auto& x : t) x.join();
    expect(good == 80, "jobs of four threads");
  }
  {  // an owner that waits elsewhere, its job unfinished, holds up nobody and keeps nobody busy
    std::atomic<bool> go{false};
    std::thread waiting([&] {
      auto work = [](int) {};
      CopyPool::Job job(pool, work);
      job.open(1);
      job.wait(0);
      while (!go) std::this_thread::sleep_for(std::chrono::milliseconds(1));
      job.open(2);
      job.wait(1);
    });
    std::this_thread::sleep_for(std::chrono::milliseconds(20));
    bool ok = false;
    std::thread other([&] { ok = ring_job(pool, 100, 5000, 32); });
    const auto t0 = Clock::now();
    std::atomic<bool> done{false};
    std::thread guard([&] {  // lets a held-up job end, so that the check reports instead of hanging
      while (!done && ms_since(t0) < 5000) std::this_thread::sleep_for(std::chrono::milliseconds(5));
      if (!done) go = true;
    });
    other.join();
    const double took = ms_since(t0);
    done = true;
    guard.join();
    expect(ok && took < 2500, "a job beside one whose owner waits");
    const double c0 = cpu_ms();
    std::this_thread::sleep_for(std::chrono::milliseconds(400));
    const double used = cpu_ms() - c0;
    printf("processor time in 400 ms of waiting: %.1f ms\n", used);
    expect(used < 100, "workers sleep while an owner waits");
    go = true;
    waiting.join();
  }
  {  // a dropped job: taken pieces end before the owner goes on, others never run
    std::atomic<int> in{0}, out{0};
    auto work = [&](int) {
      in++;
      std::this_thread::sleep_for(std::chrono::milliseconds(2));
      out++;
    };
    {
      CopyPool::Job job(pool, work);
      job.open(1000);
      std::this_thread::sleep_for(std::chrono::milliseconds(5));
    }
    const int a = in, b = out;
    std::this_thread::sleep_for(std::chrono::milliseconds(20));
    expect(a == b && in == a && a < 1000, "a dropped job leaves nothing running");
  }
}

int main() {
  for (int w : {1, 2, 8}) all(w);
  printf(fails ? "FAILED\n" : "ALL OK\n");
  return fails ? 1 : 0;
}
