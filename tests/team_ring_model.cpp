// CPU threads on team_ring_run (csrc/team_ring.cuh): the warps of the teams,
// buffers with parity barriers and a copy engine whose loads land after given
// delays.  Prints one line for what went wrong; exit status 0 if nothing did.
//   model NB TEAMS TILES LIMIT_MS FLAG_MS DELAY_MS...
// LIMIT_MS bounds a wait for a load; a load of a negative delay never lands (all
// warps then have to end, with the error raised).  FLAG_MS is how much later
// warp 1 of a team reads the abort flag than warp 0 does.
#include <unistd.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>

#include "team_ring.cuh"

using Clock = std::chrono::steady_clock;
static auto ms(int n) { return std::chrono::milliseconds(n); }
constexpr int kWarps = 2;  // of a team; warp 0 leads
constexpr int kLoading = -1;

static std::mutex mu;
static std::condition_variable cv;

[[noreturn]] static void wrong(const char* what, long j, long x) {
  std::printf("%s: tile %ld, %ld\n", what, j, x);
  std::fflush(stdout);
  _exit(1);
}

struct Buffer {
  uint32_t issued = 0, landed = 0;  // completed phases
  int tile = kLoading;  // what it holds
};
struct Barrier {
  int arrived = 0;
  bool any = false, result = false;
  uint32_t round = 0;
};
struct Cta {
  int nb, teams, tiles, limit_ms, flag_ms;
  std::vector<int> delay_ms;
  std::vector<Buffer> buf;
  std::vector<Barrier> team;
  std::vector<int> stored;
  bool abort_flag = false;
  std::vector<std::thread> copies;

  void issue(uint32_t j) {  // mu held
    buf[j % nb].tile = kLoading;
    buf[j % nb].issued++;
    cv.notify_all();
    const int d = j < delay_ms.size() ? delay_ms[j] : 0;
    auto land = [this, j] {
      buf[j % nb].tile = (int)j;
      buf[j % nb].landed++;
      cv.notify_all();
    };
    if (d == 0)
      land();
    else if (d > 0)
      copies.emplace_back([=, this] {
        std::this_thread::sleep_for(ms(d));
        std::lock_guard<std::mutex> lk(mu);
        land();
      });
  }
};

struct Ops {
  Cta& c;
  int t, warp;
  bool wait_parity(const uint32_t& phases, uint32_t parity) {
    std::unique_lock<std::mutex> lk(mu);
    return cv.wait_for(lk, ms(c.limit_ms), [&] { return (phases & 1) != parity; });
  }
  bool wait_issued(uint32_t b, uint32_t parity) { return wait_parity(c.buf[b].issued, parity); }
  bool wait_landed(uint32_t b, uint32_t parity) { return wait_parity(c.buf[b].landed, parity); }
  void gave_up() {
    std::lock_guard<std::mutex> lk(mu);
    c.abort_flag = true;
  }
  void landed(uint32_t) {}
  void issue(uint32_t j) {
    std::lock_guard<std::mutex> lk(mu);
    c.issue(j);
  }
  void transform(uint32_t j, uint32_t b) {
    for (int i = 0; i < 2; i++) {
      std::unique_lock<std::mutex> lk(mu);
      if (!c.abort_flag && c.buf[b].tile != (int)j) wrong("transformed a buffer that holds another tile", j, c.buf[b].tile);
      lk.unlock();
      std::this_thread::sleep_for(std::chrono::microseconds(200));
    }
  }
  bool aborted() {
    if (warp == 1) std::this_thread::sleep_for(ms(c.flag_ms));
    std::lock_guard<std::mutex> lk(mu);
    return c.abort_flag;
  }
  bool any(bool x) {
    std::unique_lock<std::mutex> lk(mu);
    Barrier& bar = c.team[t];
    const uint32_t round = bar.round;
    bar.any |= x;
    if (++bar.arrived == kWarps) {
      bar.arrived = 0;
      bar.result = bar.any;
      bar.any = false;
      bar.round++;
      cv.notify_all();
    } else if (!cv.wait_for(lk, ms(20 * c.limit_ms + 5000), [&] { return bar.round != round; })) {
      wrong("a warp waits for ever at its team's barrier", -1, t);
    }
    return bar.result;
  }
  void store(uint32_t j, uint32_t b) {
    std::lock_guard<std::mutex> lk(mu);
    if (c.buf[b].tile != (int)j) wrong("stored a buffer that holds another tile", j, c.buf[b].tile);
    c.stored[j]++;
  }
  void store_read() {}
};

template <int NB, int TEAMS>
static void run(Cta& c) {
  {
    std::lock_guard<std::mutex> lk(mu);
    for (uint32_t j = 0; j < (uint32_t)NB && (int)j < c.tiles; j++) c.issue(j);
  }
  std::vector<std::thread> warps;
  for (int t = 0; t < TEAMS; t++)
    for (int w = 0; w < kWarps; w++)
      warps.emplace_back([&c, t, w] {
        Ops op{c, t, w};
        omr::team_ring_run<NB, TEAMS>(op, (uint32_t)t, w == 0, (uint32_t)c.tiles);
      });
  for (auto& w : warps) w.join();
  for (auto& x : c.copies) x.join();
}

int main(int argc, char** argv) {
  Cta c;
  c.nb = std::atoi(argv[1]);
  c.teams = std::atoi(argv[2]);
  c.tiles = std::atoi(argv[3]);
  c.limit_ms = std::atoi(argv[4]);
  c.flag_ms = std::atoi(argv[5]);
  for (int i = 6; i < argc; i++) c.delay_ms.push_back(std::atoi(argv[i]));
  c.buf.resize(c.nb);
  c.team.resize(c.teams);
  c.stored.assign(c.tiles, 0);
  if (c.nb == 3 && c.teams == 2)
    run<3, 2>(c);
  else if (c.nb == 1 && c.teams == 1)
    run<1, 1>(c);
  else
    wrong("no such ring", c.nb, c.teams);
  bool lost = false;
  for (int d : c.delay_ms) lost |= d < 0;
  if (c.abort_flag != lost) wrong("abort flag", -1, c.abort_flag);
  for (int j = 0; j < c.tiles; j++)
    if (lost ? c.stored[j] > 1 : c.stored[j] != 1) wrong("not stored once", j, c.stored[j]);
  return 0;
}
