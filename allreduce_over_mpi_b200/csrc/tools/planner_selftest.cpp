// Self-test of the host-only core, meant to be built with sanitizers:
//     g++ -std=c++17 -O1 -g -fsanitize=address,undefined planner_selftest.cpp -o t && ./t
//     g++ -std=c++17 -O1 -g -fsanitize=thread planner_selftest.cpp -o t -lpthread && ./t threads
// It builds the plan of every executable shape up to 24 ranks, runs the static race check and the
// snapshot executor against a double-precision sum, exercises the candidate enumerators and the
// cost models, checks the device tables (and that damaged ones are refused), the one-pass programs of a world on one
// device, every access of the single-GPU reductions and the heap allocator, and (argument "threads") runs the thread-per-rank executor with its flag protocol,
// including a silent rank that must produce time-outs rather than a hang.
// The reference has no sanitizer builds (its flags are -Wall -Wextra only, allreduce_over_mpi/CMakeLists.txt:5).
#include <sys/wait.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "../kernels/nway_layout.h"
#include "../planner/config.hpp"
#include "../planner/cost_model.hpp"
#include "../planner/cpu_executor.hpp"
#include "../planner/policy.hpp"
#include "../planner/proc_world.hpp"
#include "../planner/world_program.hpp"
#include "../runtime/dev_plan.hpp"
#include "../runtime/heap_alloc.hpp"
#include "../runtime/fd_channel.cpp"   // descriptor passing over abstract unix sockets: plain host code, compiled in here

static int fails = 0;
#define EXPECT(c) do { if (!(c)) { std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c); ++fails; } } while (0)

static void plans_and_snapshot() {
  int checked = 0;
  for (int n = 1; n <= 24; ++n)
    for (const ft::Shape& s : ft::executable_shapes(n)) {
      ft::Plan p = ft::build_plan(n, s);
      EXPECT(p.ok());
      EXPECT(ft::check_hazards(p).empty());
      for (uint64_t count : {1ull, 29ull, 257ull}) {
        std::vector<std::vector<double>> data(n, std::vector<double>(count));
        std::vector<double> want(count, 0.0);
        for (int r = 0; r < n; ++r)
          for (uint64_t i = 0; i < count; ++i) { data[r][i] = std::sin(r * 131 + i * 7) ; want[i] += data[r][i]; }
        std::vector<void*> bufs(n);
        for (int r = 0; r < n; ++r) bufs[r] = data[r].data();
        EXPECT(ft::run_plan_snapshot(p, FT_SUM, FT_F64, bufs.data(), count) == FT_OK);
        for (int r = 0; r < n; ++r)
          for (uint64_t i = 0; i < count; ++i) EXPECT(std::fabs(data[r][i] - want[i]) < 1e-9);
        EXPECT(ft::plan_traffic_elems(p, ft::Blocks(count, n)) == 2ull * (n - 1) * count);
      }
      ++checked;
    }
  EXPECT(checked > 150);
  EXPECT(!ft::validate_shape(7, ft::Shape{{2, 2}, 3, false}).empty());
  EXPECT(!ft::parse_topo("2,3", "", 7).ok());
}

// Device tables: every rank of every shape passes the descriptor check, the reduce-scatter half
// leaves each block complete on exactly one rank, and a table damaged in any of the ways the check
// guards against is refused.
static void device_tables() {
  for (int n = 1; n <= 24; ++n)
    for (const ft::Shape& s : ft::executable_shapes(n)) {
      ft::Plan p = ft::build_plan(n, s);
      for (int r = 0; r < n; ++r) EXPECT(ft::check_dev_plan(ft::build_dev_plan(p, r), n, r).empty());
      uint64_t owners = 0;
      for (uint64_t h : ft::rs_holders(p)) { EXPECT(h && !(h & (h - 1))); owners |= h; }
      EXPECT(n == 1 || owners == (1ull << n) - 1);
    }
  const ft::Plan p = ft::build_plan(7, ft::Shape{{2, 3}, 1, false});
  const ft::HostDevPlan good = ft::build_dev_plan(p, 2);
  EXPECT(ft::check_dev_plan(good, 7, 2).empty());
  EXPECT(!good.pulls.empty());
  auto broken = [&](auto&& damage) {
    ft::HostDevPlan d = good;
    damage(d);
    return !ft::check_dev_plan(d, 7, 2).empty();
  };
  EXPECT(broken([](ft::HostDevPlan& d) { d.pulls[0].block = 7; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.pulls[0].src[0] = 9; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.pulls[0].src[0] = 2; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.pulls[0].nsrc = 0; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.pulls[0].nsrc = FT_MAX_FANIN; d.pulls[0].reduce = 1; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.plan.stages[0].sync_mask = 0; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.plan.stages[0].sync_mask |= 1ull << 7; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.plan.stages[1].pull_begin += 1; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.plan.stages[d.plan.nstages - 1].pull_end += 1; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.plan.nstages += 1; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.plan.stages[0].last_rs = 1; }));
  EXPECT(broken([](ft::HostDevPlan& d) { d.plan.end_sync_mask = ~0ull; }));
  EXPECT(!ft::check_dev_plan(good, 7, 7).empty());
}

// Heap offsets: allocations alone are consecutive from zero; live blocks never overlap and stay inside the
// heap under a random mix of alloc and free; everything merges back into one block; two allocators fed the
// same sequence agree (that is what keeps the ranks' heaps symmetric).
static void heap_offsets() {
  ft::HeapAllocator h(1 << 20);
  EXPECT(h.alloc(1) == 0 && h.alloc(256) == 256 && h.alloc(257) == 512 && h.alloc(0) == 1024);
  EXPECT(h.used_bytes() == 256 + 256 + 512 + 256 && h.live_blocks() == 4);
  EXPECT(h.alloc((size_t)1 << 20) == ft::HeapAllocator::kNone);
  EXPECT(h.alloc(~(size_t)0) == ft::HeapAllocator::kNone);
  EXPECT(!h.free(128) && !h.free(4096));
  EXPECT(h.free(256) && !h.free(256));
  EXPECT(h.alloc(300) == 1280);          // the 256-byte hole is too small: first fit moves on
  EXPECT(h.alloc(200) == 256);           // and takes it for something that fits
  h.reset();
  EXPECT(h.largest_free() == (size_t)1 << 20 && h.live_blocks() == 0);

  ft::HeapAllocator a(1 << 22), b(1 << 22);
  std::vector<std::pair<size_t, size_t>> live;   // offset, requested bytes
  uint64_t rng = 12345;
  auto next = [&] { rng = rng * 6364136223846793005ull + 1442695040888963407ull; return (uint32_t)(rng >> 33); };
  for (int step = 0; step < 20000; ++step) {
    if (live.empty() || next() % 3) {
      const size_t want = 1 + next() % 60000;
      const size_t off = a.alloc(want);
      EXPECT(off == b.alloc(want));
      if (off == ft::HeapAllocator::kNone) { EXPECT(a.largest_free() < ((want + 255) / 256) * 256); continue; }
      EXPECT(off % 256 == 0 && off + want <= a.size());
      for (const auto& l : live) EXPECT(off + want <= l.first || l.first + ((l.second + 255) / 256) * 256 <= off);
      live.push_back({off, want});
    } else {
      const size_t k = next() % live.size();
      EXPECT(a.free(live[k].first) && b.free(live[k].first));
      live[k] = live.back();
      live.pop_back();
    }
  }
  for (const auto& l : live) EXPECT(a.free(l.first));
  EXPECT(a.live_blocks() == 0 && a.free_blocks() == 1 && a.largest_free() == a.size());
}

// Process world: five forked children meet in a session, reduce a private buffer (pulled with
// process_vm_readv), a small one (through the segment) and one in the symmetric heap, for a lonely layout.
static void proc_world_forked() {
  {   // some sandboxes filter process_vm_readv out altogether: probe it on this process's own memory
    char src[8] = "probe", dst[8] = {0};
    struct iovec lv{dst, sizeof dst}, rv{src, sizeof src};
    if (process_vm_readv(getpid(), &lv, 1, &rv, 1, 0) != (ssize_t)sizeof src) {
      std::printf("process world not exercised: process_vm_readv is not available here\n");
      return;
    }
  }
  const int n = 5;
  const std::string session = "selftest-" + std::to_string((long)getpid());
  std::vector<pid_t> kids;
  for (int r = 0; r < n; ++r) {
    const pid_t pid = fork();
    if (pid == 0) {
      int bad = 0;
      {
        ft::ProcWorld w;
        if (!w.join(session, r, n, 30.0)) _exit(10);
        const ft::Plan p = ft::build_plan(n, ft::Shape{{2, 2}, 1, false});
        for (uint64_t count : {9ull, 70001ull}) {
          std::vector<double> v(count);
          for (int round = 0; round < 3; ++round) {
            for (uint64_t i = 0; i < count; ++i) v[i] = (double)(r + 1) + (double)(i % 5) + round;
            bad |= w.allreduce(p, FT_SUM, FT_F64, nullptr, v.data(), count).code != FT_OK;
            for (uint64_t i = 0; i < count; ++i) bad |= v[i] != 15.0 + n * ((double)(i % 5) + round);
          }
        }
        bad |= !w.heap_create(1 << 20);
        double* h = bad ? nullptr : (double*)w.heap_alloc(30000 * sizeof(double));
        if (h && w.heap_symmetric(h)) {
          for (int i = 0; i < 30000; ++i) h[i] = (double)(r + 1);
          bad |= w.allreduce(p, FT_SUM, FT_F64, nullptr, h, 30000).code != FT_OK;
          bad |= h[0] != 15.0 || h[29999] != 15.0;
        } else {
          bad = 1;
        }
        bad |= w.barrier().code != FT_OK;
      }
      _exit(bad ? 11 : 0);
    }
    kids.push_back(pid);
  }
  for (pid_t k : kids) {
    int status = 0;
    waitpid(k, &status, 0);
    EXPECT(WIFEXITED(status) && WEXITSTATUS(status) == 0);
  }
}

static void enumerators_and_models() {
  for (int n = 0; n <= 200; ++n) {
    auto a = ft::candidate_shapes(n);
    if (n >= 2) EXPECT(a.size() == ft::count_ordered_factorizations(n) + 1);
    (void)ft::candidate_shapes_legacy(n);
    (void)ft::choose_width(n);
    (void)ft::prime_factors(n);
  }
  EXPECT(ft::shape_to_string(ft::choose_v0(8).widths) == "1*8");
  EXPECT(std::fabs(ft::choose_v0(8).cost - 0.666) < 1e-9);
  ft::V1Params k;
  k.nvls_gbs = 500;
  for (int n = 2; n <= 16; ++n)
    for (uint64_t b : {1024ull, 1ull << 20, 1ull << 30}) EXPECT(std::isfinite(ft::pick_algorithm(n, b, k).us));
}

// The selection policy and its JSON reader under the sanitizers: well-formed, damaged and hostile texts, rows that
// parse but do not apply, and more distinct message sizes than the answer cache holds.
static void policy_and_json() {
  const char* texts[] = {
      "{\"params\": {\"launch_us\": 3.5, \"peer_eff\": {\"2\": 0.5, \"99\": 1.0, \"x\": 2}}, \"table\": {\"8\": [[1024, \"ll\", \"2*4\"], "
      "[1048576, \"nvls\", \"8\"], [4096, \"warp\", \"8\"], [8192, \"staged\", \"3*3\"], [1, 2], \"row\", [65536, \"hybrid-0.8-0.25\", \"8\"]]}}",
      "", "{", "{\"table\": [[[[[[[[[[", "{\"a\": \"\\u12", "{\"a\": 1e99999, \"b\": -}", "[1, 2, 3]", "nul", "{\"params\": 5, \"table\": 7}",
      "{\"table\": {\"8\": {\"not\": \"a list\"}}}"};
  int i = 0;
  for (const char* t : texts) {
    ft::Json root;
    ft::JsonParser jp(t);
    const bool ok = jp.parse(&root);
    EXPECT(ok == (i == 0 || i == 6 || i == 8 || i == 9));
    ++i;
  }
  std::string deep(5000, '[');
  ft::Json root;
  ft::JsonParser jp(deep);
  EXPECT(!jp.parse(&root));
  ft::Policy pol(8);
  EXPECT(pol.add_row(1024, "ll", "2*4") && pol.add_row(1 << 20, "nvls", "8") && pol.add_row(65536, "hybrid-0.8-0.25", "8"));
  EXPECT(!pol.add_row(4096, "warp", "8") && !pol.add_row(8192, "staged", "3*3") && !pol.add_row(8192, "staged", "2**"));
  ft::PolicyChoice c = pol.choose(1024, false, false, 64 << 20, 8 << 10);
  EXPECT(c.algo == "ll" && c.shape.widths.size() == 2 && c.from_table);
  c = pol.choose(1 << 20, true, true, 64 << 20, 8 << 10);
  EXPECT(c.algo == "nvls");
  c = pol.choose(1 << 20, true, false, 64 << 20, 8 << 10);     // the switch is not available: the row does not apply
  EXPECT(c.algo != "nvls" && c.algo != "hybrid");
  for (uint64_t b = 16; b < 16 * 3 * ft::Policy::kCacheEntries; b += 16) {   // the cache starts over instead of growing
    c = pol.choose(b, (b / 16) % 2 == 0, false, 64 << 20, 8 << 10);
    EXPECT(!c.algo.empty() && ft::validate_shape(8, c.shape).empty());
  }
  ft::Shape sh;
  EXPECT(ft::parse_shape_text(" 2 x 2 + 1 ", &sh) && sh.lonely == 1 && sh.widths.size() == 2);
  EXPECT(ft::parse_shape_text("RING8", &sh) && sh.ring);
  EXPECT(!ft::parse_shape_text("2*-4", &sh) && !ft::parse_shape_text("", &sh) && !ft::parse_shape_text("ring", &sh) &&
         !ft::parse_shape_text("99999999*2", &sh));
}

// Descriptor passing (how VMM heaps and multicast objects reach the other ranks): a pipe's read end travels from a thread
// to this one with its tag, the received descriptor reads what the sender wrote, waits run out instead of blocking.
static void fd_passing() {
  const std::string name = "ft-selftest-" + std::to_string((long)getpid());
  const int sock = ft_fd_listen(name.c_str());
  EXPECT(sock >= 0);
  int tag = -1;
  EXPECT(ft_fd_recv(sock, &tag, 50) < 0);                        // nobody sent: the wait is bounded
  EXPECT(ft_fd_send("ft-selftest-nobody-listens", 0, 1, 50) != 0);
  int pipefd[2];
  EXPECT(pipe(pipefd) == 0);
  std::thread sender([&] {
    EXPECT(write(pipefd[1], "heap", 4) == 4);
    EXPECT(ft_fd_send(name.c_str(), pipefd[0], 7, 2000) == 0);
  });
  const int got = ft_fd_recv(sock, &tag, 2000);
  sender.join();
  EXPECT(got >= 0 && tag == 7);
  char buf[8] = {0};
  EXPECT(got >= 0 && read(got, buf, 4) == 4 && !std::memcmp(buf, "heap", 4));
  if (got >= 0) ft_fd_close(got);
  ft_fd_close(pipefd[0]);
  ft_fd_close(pipefd[1]);
  ft_fd_close(sock);
}

static void thread_world(bool with_fault) {
  for (const char* text : {"2,2", "2,3", "2,2,2"}) {
    ft::ShapeConfig cfg = ft::parse_topo(text, std::string(text) == "2,3" ? "1" : "", std::string(text) == "2,2" ? 4 : (std::string(text) == "2,3" ? 7 : 8));
    EXPECT(cfg.ok());
    const int n = cfg.shape.world();
    ft::Plan p = ft::build_plan(n, cfg.shape);
    ft::CpuWorld w(n);
    w.timeout_s = with_fault ? 0.2 : 20.0;
    const uint64_t count = 4099;
    std::vector<std::vector<float>> data(n, std::vector<float>(count));
    std::vector<ft::RankStatus> st(n);
    ft::FaultSpec f;
    f.kind = ft::Fault::NeverSignal; f.rank = 1; f.stage = 1;
    for (int round = 0; round < 3; ++round) {
      for (int r = 0; r < n; ++r) for (uint64_t i = 0; i < count; ++i) data[r][i] = (float)(r + 1);
      std::vector<std::thread> th;
      for (int r = 0; r < n; ++r)
        th.emplace_back([&, r] { st[r] = ft::cpu_allreduce(w, r, p, FT_SUM, FT_F32, nullptr, data[r].data(), count, 0, with_fault ? &f : nullptr); });
      for (auto& t : th) t.join();
      if (with_fault) {
        bool any_timeout = false;
        for (int r = 0; r < n; ++r) any_timeout = any_timeout || st[r].code == FT_ERR_TIMEOUT;
        EXPECT(any_timeout);
        break;   // the world is poisoned after a fault
      }
      for (int r = 0; r < n; ++r) { EXPECT(st[r].code == FT_OK); EXPECT(data[r][count - 1] == (float)(n * (n + 1) / 2)); }
    }
  }
}

// Reduce-scatter and all-gather as calls of their own, three rounds without any host barrier in
// between, with a whole all-reduce after each pair: rendezvous numbers keep growing across the three
// kinds of call and the closing all-rank rendezvous lets every rank overwrite its buffer right away.
static void thread_world_phases() {
  for (const char* text : {"2,2", "2,3", "2,2,2", "1"}) {
    const std::string t = text;
    const int n = t == "2,2" ? 4 : (t == "2,3" ? 7 : (t == "1" ? 5 : 8));
    ft::ShapeConfig cfg = ft::parse_topo(text, t == "2,3" ? "1" : "", n);
    EXPECT(cfg.ok());
    ft::Plan p = ft::build_plan(n, cfg.shape);
    const std::vector<uint64_t> holders = ft::rs_holders(p);
    ft::CpuWorld w(n);
    w.timeout_s = 20.0;
    const uint64_t count = 1031;
    const ft::Blocks g(count, n);
    std::vector<std::vector<double>> data(n, std::vector<double>(count));
    std::vector<int> bad(n, 0);
    std::vector<std::thread> th;
    for (int r = 0; r < n; ++r)
      th.emplace_back([&, r] {
        for (int round = 0; round < 3; ++round) {
          for (uint64_t i = 0; i < count; ++i) data[r][i] = (double)(r + 1 + round);
          bad[r] |= ft::cpu_allreduce(w, r, p, FT_SUM, FT_F64, nullptr, data[r].data(), count, 0, nullptr, 1, 1).code != FT_OK;
          for (int b = 0; b < n; ++b)   // wipe everything this rank does not own
            if (!(holders[b] >> r & 1))
              for (uint64_t i = g.offset(b); i < g.offset(b) + g.length(b); ++i) data[r][i] = -1e300;
          bad[r] |= ft::cpu_allreduce(w, r, p, FT_SUM, FT_F64, nullptr, data[r].data(), count, 0, nullptr, 1, 2).code != FT_OK;
          bad[r] |= ft::cpu_allreduce(w, r, p, FT_SUM, FT_F64, nullptr, data[r].data(), count).code != FT_OK;
          const double want = (double)n * (n * (n + 1) / 2 + n * round);
          for (uint64_t i = 0; i < count; ++i) bad[r] |= data[r][i] != want;
        }
      });
    for (auto& x : th) x.join();
    for (int r = 0; r < n; ++r) EXPECT(!bad[r]);
  }
}

// Host twins of the small-message protocols, mixed with staged calls and single phases, with every rank
// delayed at random before each call.  Neither protocol closes with a rendezvous; what keeps a slow rank's
// reads apart from a fast rank's next write into the same slot (two calls later) is only the argument
// that finishing the call in between needs every rank's contribution.  Under the thread sanitizer a hole
// in that argument is a reported race; in any build it is a wrong sum or a timeout.
static void random_pause(int rank) {
  thread_local uint64_t rng = 0;
  if (!rng) rng = 7777 + 13 * (uint64_t)rank;
  rng = rng * 6364136223846793005ull + 1442695040888963407ull;
  if ((rng >> 60) < 5) std::this_thread::sleep_for(std::chrono::microseconds((rng >> 40) % 400));
}

// Every executable shape up to 9 ranks on real threads that stall at random between a stage's rendezvous and
// its pulls, six calls back to back: in place, through the slots, and as two single phases.  The per-stage rendezvous sets are the
// only thing that orders one rank's writes against another's reads; a set that misses a dependency shows up
// as a race under the thread sanitizer (and usually as a wrong sum).
static void thread_world_all_shapes() {
  int shapes = 0;
  for (int n = 2; n <= 9; ++n)
    for (const ft::Shape& s : ft::executable_shapes(n)) {
      const ft::Plan p = ft::build_plan(n, s);
      ft::CpuWorld w(n);
      w.timeout_s = 30.0;
      w.mid_call_hook = random_pause;
      const uint64_t count = 97;
      const std::vector<uint64_t> holders = ft::rs_holders(p);
      const ft::Blocks g(count, n);
      std::vector<int> bad(n, 0);
      std::vector<std::thread> th;
      for (int r = 0; r < n; ++r)
        th.emplace_back([&, r] {
          std::vector<double> buf(count);
          for (int round = 0; round < 6; ++round) {
            for (uint64_t i = 0; i < count; ++i) buf[i] = (double)(r + 1) * (double)(i + 1) + round;
            ft::RankStatus st;
            if (round % 3 == 0) {
              st = ft::cpu_allreduce(w, r, p, FT_SUM, FT_F64, nullptr, buf.data(), count);
            } else if (round % 3 == 1) {
              st = ft::cpu_allreduce_slots(w, r, p, FT_SUM, FT_F64, nullptr, buf.data(), count);
            } else {   // the two halves as calls of their own, everything not owned wiped in between
              st = ft::cpu_allreduce(w, r, p, FT_SUM, FT_F64, nullptr, buf.data(), count, 0, nullptr, 1, 1);
              for (int b = 0; b < n; ++b)
                if (!(holders[b] >> r & 1))
                  for (uint64_t i = g.offset(b); i < g.offset(b) + g.length(b); ++i) buf[i] = -1e300;
              if (st.code == FT_OK) st = ft::cpu_allreduce(w, r, p, FT_SUM, FT_F64, nullptr, buf.data(), count, 0, nullptr, 1, 2);
            }
            bad[r] |= st.code != FT_OK;
            for (uint64_t i = 0; i < count; ++i) bad[r] |= buf[i] != (double)(n * (n + 1) / 2) * (double)(i + 1) + (double)n * round;
          }
        });
      for (auto& x : th) x.join();
      for (int r = 0; r < n; ++r) EXPECT(!bad[r]);
      ++shapes;
    }
  EXPECT(shapes > 30);
}

static void thread_world_small_message_twins() {
  for (int n : {2, 3, 5, 8}) {
    ft::CpuWorld w(n);
    w.timeout_s = 30.0;
    w.mid_call_hook = random_pause;   // ranks also stall in the middle of a call, between publishing and reading
    const ft::Plan flat = ft::build_plan(n, ft::Shape::flat(n));
    const ft::Plan ring = ft::build_plan(n, ft::Shape::make_ring(n));
    const ft::Plan tree = ft::build_plan(n, n == 8 ? ft::Shape{{2, 4}, 0, false} : (n == 5 ? ft::Shape{{2, 2}, 1, false} : ft::Shape::flat(n)));
    const uint64_t count = 777;
    std::vector<int> bad(n, 0);
    std::vector<std::thread> th;
    for (int r = 0; r < n; ++r)
      th.emplace_back([&, r] {
        uint64_t rng = 99 + r;
        auto jitter = [&] {
          rng = rng * 6364136223846793005ull + 1442695040888963407ull;
          std::this_thread::sleep_for(std::chrono::microseconds((rng >> 40) % 300));
        };
        std::vector<float> buf(count);
        for (int round = 0; round < 120; ++round) {
          for (uint64_t i = 0; i < count; ++i) buf[i] = (float)(r + 1) + (float)(i % 7) + (float)round;
          jitter();
          ft::RankStatus st;
          switch (round % 10) {   // back-to-back calls of the same kind are the ones that lean on the parity rule
            case 0: case 1: case 6: st = ft::cpu_allreduce_ll(w, r, FT_SUM, FT_F32, nullptr, buf.data(), count); break;
            case 2: case 3: case 5: st = ft::cpu_allreduce_oneshot(w, r, FT_SUM, FT_F32, nullptr, buf.data(), count); break;
            case 4: st = ft::cpu_allreduce(w, r, round % 16 == 4 ? flat : ring, FT_SUM, FT_F32, nullptr, buf.data(), count); break;
            case 9: st = ft::cpu_allreduce_push(w, r, FT_SUM, FT_F32, buf.data(), count); break;
            case 8:   // a plan on tagged words, twice in a row (both receive areas), then the flat tagged-word call on the same areas
              st = ft::cpu_allreduce_ll_tree(w, r, round % 20 == 8 ? tree : ring, FT_SUM, FT_F32, nullptr, buf.data(), count);
              if (st.code == FT_OK) {
                for (uint64_t i = 0; i < count; ++i) buf[i] = (float)(r + 1) + (float)(i % 7) + (float)round;
                st = ft::cpu_allreduce_ll_tree(w, r, flat, FT_SUM, FT_F32, nullptr, buf.data(), count);
              }
              break;
            case 7:   // through the slots, twice in a row, with different shapes (no closing rendezvous in this mode)
              st = ft::cpu_allreduce_slots(w, r, round % 16 == 7 ? tree : ring, FT_SUM, FT_F32, nullptr, buf.data(), count);
              if (st.code == FT_OK) {
                for (uint64_t i = 0; i < count; ++i) buf[i] = (float)(r + 1) + (float)(i % 7) + (float)round;
                st = ft::cpu_allreduce_slots(w, r, flat, FT_SUM, FT_F32, nullptr, buf.data(), count);
              }
              break;
            default:
              st = ft::cpu_allreduce(w, r, flat, FT_SUM, FT_F32, nullptr, buf.data(), count, 0, nullptr, 1, 1);
              if (st.code == FT_OK) st = ft::cpu_allreduce(w, r, flat, FT_SUM, FT_F32, nullptr, buf.data(), count, 0, nullptr, 1, 2);
          }
          bad[r] |= st.code != FT_OK;
          for (uint64_t i = 0; i < count; ++i) {
            const float want = (float)(n * (n + 1) / 2) + (float)n * ((float)(i % 7) + (float)round);
            bad[r] |= buf[i] != want;
          }
        }
      });
    for (auto& x : th) x.join();
    for (int r = 0; r < n; ++r) EXPECT(!bad[r]);
  }
}

// One pass over the copies of all ranks, as world_reduce_kernel does it for one element of each block: in place, the
// inputs read as late as the program asks for them, no more values put aside than the program says.
static char rank_copy[ftk::kWorldRanks];   // the ranks' "addresses"
template <int RANKS>
static void run_world_args(const ftk::WorldArgs<RANKS>& a, int entries, int depth, uint16_t (*copy)[ftk::kWorldRanks]) {
  const auto at = [&](const void* rank, int block) -> uint16_t& { return copy[(const char*)rank - rank_copy][block]; };
  for (int e = 0; e < entries; ++e) {
    const ftk::WorldEntry& en = a.entry[e];
    float acc = 0;
    std::vector<float> aside(depth > 0 ? depth : 1, 0.f);
    for (int k = en.first; k < en.first + en.nsteps; ++k) {
      const float v = ft::bf16_to_float({at(a.ptr[k], en.block)});
      if (depth == 0) { acc = k == en.first ? v : acc + v; continue; }
      if (a.code[k] & 1) {
        aside.insert(aside.begin(), acc);
        aside.pop_back();
        acc = v;
      } else {
        acc += v;
      }
      const int rounds = a.code[k] >> 2;
      for (int r = 0; r < rounds; ++r) {
        const ft::bf16_t w = ft::float_to_bf16(acc);
        if (a.store[k][r] != ftk::kNoStore) at(a.ptr[a.kSteps + a.store[k][r]], en.block) = w.bits;
        acc = ft::bf16_to_float(w);
        if (r + 1 < rounds || (a.code[k] & 2)) {
          acc = aside[0] + acc;
          aside.erase(aside.begin());
          aside.push_back(0.f);
        }
      }
    }
    for (int r = 0; r < RANKS; ++r)
      if (en.mask >> r & 1) at(a.ptr[a.kSteps + r], en.block) = ft::float_to_bf16(acc).bits;
  }
}
// The same for the programs that are compiled in: world_tree_kernel's and world_copy_kernel's reading of their parameters.
static void run_tree_args(const ftk::WorldTreeArgs& a, int entries, int tree, uint16_t (*copy)[ftk::kWorldRanks]) {
  const auto at = [&](const void* rank, int block) -> uint16_t& { return copy[(const char*)rank - rank_copy][block]; };
  for (int e = 0; e < entries; ++e) {
    const uint64_t word = a.entry[e];
    const int block = (int)(word >> ftk::kTreeBlock) & 7, n = tree < 0 ? 1 : ftk::kWorldTrees[tree].ranks;
    const uint32_t code = tree < 0 ? 1 : ftk::kWorldTrees[tree].code[word >> ftk::kTreeWhich & 1];
    float v[ftk::kTreeRanks], acc = 0;
    for (int k = 0; k < n; ++k) v[k] = ft::bf16_to_float({at(a.in[word >> (3 * k) & 7], block)});
    std::vector<float> aside;
    for (int k = 0, t = 0; k < n; ++k) {
      if (code >> (4 * k) & 1) {
        if (k) aside.push_back(acc);
        acc = v[k];
      } else {
        acc += v[k];
      }
      EXPECT(aside.size() <= 2);
      const int rounds = (int)(code >> (4 * k) & 15) >> 2;
      for (int r = 0; r < rounds; ++r) {
        const ft::bf16_t w = ft::float_to_bf16(acc);
        EXPECT(t < ftk::kTreeRounds);
        const int to = (int)(word >> (ftk::kTreeStore + 4 * t++)) & 15;
        if (to != 15) at(a.out[to], block) = w.bits;
        acc = ft::bf16_to_float(w);
        if (r + 1 < rounds || (code >> (4 * k) & 2)) {
          acc = aside.back() + acc;
          aside.pop_back();
        }
      }
    }
    EXPECT(aside.empty());
    for (int r = 0; r < ftk::kTreeRanks; ++r)
      if (word >> (ftk::kTreeMask + r) & 1) at(a.out[r], block) = ft::float_to_bf16(acc).bits;
  }
}
static int compiled_programs[ftk::kWorldTreeCount], uncompiled_programs;

template <int RANKS>
static bool world_program_as_plan(int n, const ft::Plan& p, ft::WorldPhase phase) {
  ft::WorldProgram wp = ft::WorldProgramBuilder(n).run(p, phase);
  ft::compact_world_program(n, &wp);
  if (!wp.ok || wp.depth > (RANKS == 8 ? 2 : 3)) return false;
  void* in[ftk::kWorldRanks];
  ftk::WorldArgs<RANKS> a;
  std::memset((void*)&a, 0xab, sizeof a);
  for (int r = 0; r < RANKS; ++r) in[r] = rank_copy + r;
  if (!ft::fill_world_args(wp, n, in, in, &a)) return false;
  for (const ftk::WorldEntry& e : wp.entries)   // the kernel looks up whole groups of steps
    for (int k = e.first; k < e.first + (e.nsteps + ftk::kWorldGroup - 1) / ftk::kWorldGroup * ftk::kWorldGroup; ++k) {
      EXPECT(k < a.kSteps + RANKS);
      EXPECT((a.ptr[k] >= in[0] && a.ptr[k] <= in[n - 1]) || (k >= a.kSteps + n && !a.ptr[k]));
    }
  uint16_t got[ftk::kWorldRanks][ftk::kWorldRanks] = {}, want[ftk::kWorldRanks][ftk::kWorldRanks] = {};
  void* bufs[ftk::kWorldRanks];
  for (int r = 0; r < n; ++r) {
    for (int b = 0; b < n; ++b) want[r][b] = got[r][b] = ft::float_to_bf16((float)std::sin(r * 131 + b * 7 + 1)).bits;
    bufs[r] = want[r];
  }
  const int half = p.num_stages / 2;
  EXPECT(ft::run_plan_snapshot(p, FT_SUM, FT_BF16, bufs, n, 1, phase == ft::WorldPhase::all_gather ? half : 0,
                               phase == ft::WorldPhase::reduce_scatter ? half : -1) == FT_OK);
  if (wp.tree >= 0 || wp.copies) {
    uint16_t compact[ftk::kWorldRanks][ftk::kWorldRanks];
    std::memcpy(compact, got, sizeof got);
    ftk::WorldTreeArgs t;
    ft::fill_tree_args(wp, n, in, in, &t);
    EXPECT(wp.copies == (phase == ft::WorldPhase::all_gather) && wp.words.size() == wp.entries.size());
    run_tree_args(t, (int)wp.words.size(), wp.copies ? -1 : wp.tree, compact);
    EXPECT(!std::memcmp(compact, want, sizeof compact));
    if (!wp.copies) ++compiled_programs[wp.tree];
  } else if (n <= ftk::kTreeRanks) {
    ++uncompiled_programs;
  }
  run_world_args(a, (int)wp.entries.size(), wp.depth, got);
  EXPECT(!std::memcmp(got, want, sizeof got));
  return true;
}
static void world_programs() {
  int shapes = 0, taken = 0;
  for (int n = 2; n <= ftk::kWorldRanks; ++n)
    for (const ft::Shape& s : ft::executable_shapes(n)) {
      const ft::Plan p = ft::build_plan(n, s);
      for (ft::WorldPhase phase : {ft::WorldPhase::all, ft::WorldPhase::reduce_scatter, ft::WorldPhase::all_gather}) {
        ++shapes;
        taken += world_program_as_plan<16>(n, p, phase) && (n > 8 || world_program_as_plan<8>(n, p, phase));
      }
    }
  EXPECT(shapes > 250 && taken == shapes);
  for (int c : compiled_programs) EXPECT(c >= 2);   // every compiled program is some shape's, as a whole and as a reduce-scatter
  EXPECT(uncompiled_programs == 0);
}

// Threads that ask one world for programs at the same time get the same ones; shapes that are none leave nothing behind.
static void world_program_cache() {
  const int n = 12;
  const std::vector<ft::Shape> shapes = ft::executable_shapes(n);
  const ft::WorldPhase phases[] = {ft::WorldPhase::all, ft::WorldPhase::reduce_scatter, ft::WorldPhase::all_gather};
  ft::WorldProgramCache cache;
  std::vector<std::vector<const ft::WorldProgramCache::Entry*>> got(4);
  std::vector<std::thread> th;
  for (int t = 0; t < 4; ++t)
    th.emplace_back([&, t] {
      for (const ft::Shape& s : shapes)
        for (ft::WorldPhase phase : phases)
          got[t].push_back(cache.get(n, ft::WorldForm::plan, phase, s.widths.data(), (int)s.widths.size(), s.lonely, s.ring));
      got[t].push_back(cache.get(n, ft::WorldForm::flat, ft::WorldPhase::all, nullptr, 0, 0, false));
      got[t].push_back(cache.get(n, ft::WorldForm::rotated, ft::WorldPhase::all, nullptr, 0, 0, false));
    });
  for (auto& x : th) x.join();
  for (int t = 0; t < 4; ++t) EXPECT(got[t] == got[0]);
  for (const auto* e : got[0]) EXPECT(e && e->program.ok);
  EXPECT(cache.size() == got[0].size());
  const int wrong[] = {5, 2};
  EXPECT(!cache.get(n, ft::WorldForm::plan, ft::WorldPhase::all, wrong, 2, 0, false) && cache.size() == got[0].size());
}

// Every access of every thread of the single-GPU reductions, for the way the host cuts the vectors: reads inside the
// sources and on the boundaries the instructions need, each element of the result written once.
struct NwayReplay {
  ftk::NwayArgs whole, a;      // before and after the cut
  size_t is, os, len;          // bytes of an element of the sources, of the result; elements
  std::vector<uint8_t> written;
  bool good = true;
  void need(bool ok) { good = good && ok; }
  void read(int k, const void* p, size_t bytes, size_t align) {
    const uintptr_t lo = (uintptr_t)whole.src[k];
    need((uintptr_t)p % align == 0 && (uintptr_t)p >= lo && (uintptr_t)p + bytes <= lo + len * is);
  }
  void write(const void* p, size_t bytes, size_t align) {
    const uintptr_t lo = (uintptr_t)whole.dst;
    const bool in = (uintptr_t)p % align == 0 && (uintptr_t)p >= lo && (uintptr_t)p + bytes <= lo + len * os;
    need(in);
    for (size_t b = 0; in && b < bytes; ++b) need(++written[(uintptr_t)p - lo + b] == 1);
  }
  const unsigned char* src(int k, long long bytes) const { return (const unsigned char*)((uintptr_t)a.src[k] + bytes); }
  const unsigned char* dst(long long bytes) const { return (const unsigned char*)((uintptr_t)a.dst + bytes); }
  void edges(int thread, int threads) {
    for (int e = thread; e < a.edge; e += threads) {
      const long long i = e < a.head ? (long long)e - a.head : (long long)(a.nbody + (e - a.head));
      for (int k = 0; k < a.n; ++k) read(k, src(k, i * (long long)is), is, is);
      write(dst(i * (long long)os), os, os);
    }
  }
  // wide and scaled kernels: 32 bytes of every source a thread, `out` bytes of the result.  `first`: the edges are the
  // first CTA's, as in calls that fetch ahead, else the last one's
  void wide(size_t load, size_t out, size_t store, bool first = false) {
    first = first && a.nvec;   // (such calls are long)
    a.seam.ahead = first;
    const unsigned long long grid = ftk::nway_grid(a, ftk::kWideThreads);
    need(grid > 0);
    for (unsigned long long cta = 0; cta < grid; ++cta)
      for (unsigned t = 0; t < ftk::kWideThreads; ++t) {
        const unsigned long long i = cta * ftk::kWideThreads + t;
        if (i < a.nvec) {
          for (int k = 0; k < a.n; ++k) read(k, src(k, i * 32), 32, load);
          write(dst(i * out), out, store);
        } else if (!first && cta == grid - 1) {
          edges(t, ftk::kWideThreads);
        }
        if (first && cta == 0) edges(t, ftk::kWideThreads);
      }
  }
  void realign(bool first = false) {
    a.seam.ahead = first;
    const unsigned long long grid = ftk::nway_grid(a, ftk::kRealignPerCta);
    need(grid > 0 && a.shift[0] > 0 && a.shift[0] < 32);
    for (unsigned long long cta = 0; cta < grid; ++cta)
      for (unsigned t = 0; t < ftk::kRealignThreads; ++t) {
        const unsigned lane = t & 31;
        const unsigned long long i = cta * ftk::kRealignPerCta + t / 32 * 31 + lane;
        if (i <= a.nvec)
          for (int k = 0; k < a.n; ++k) read(k, src(k, (long long)(i * 32) - a.shift[0]), 32, 32);
        if (lane < 31 && i < a.nvec) write(dst(i * 32), 32, 32);   // from this unit's sum and the next lane's: i + 1 <= nvec
        if (a.edge && cta == (first ? 0 : grid - 1)) edges(t, ftk::kRealignThreads);
      }
  }
  void shift() {
    const unsigned threads = ftk::shift_long(a) ? 64 : 128, unroll = ftk::shift_long(a) ? 2 : 1;
    const unsigned long long grid = ftk::nway_grid(a, threads * unroll);
    need(grid > 0);
    for (unsigned long long cta = 0; cta < grid; ++cta)
      for (unsigned t = 0; t < threads; ++t) {
        for (unsigned u = 0; u < unroll; ++u) {
          const unsigned long long i = cta * threads * unroll + u * threads + t;
          for (int k = 0; k < a.n; ++k) {
            const long long s = a.shift[k];
            if (i < a.nvec || (s && i == a.nvec)) read(k, src(k, (long long)(i * 16) - s), 16, 16);
            if (s && t % 32 == 31 && i < a.nvec) read(k, src(k, (long long)(i * 16 + 16) - s), 16, 16);
          }
          if (i < a.nvec) write(dst(i * 16), 16, 16);
        }
        if (a.edge && cta == grid - 1) edges(t, threads);
      }
  }
  bool done() {
    for (int k = 0; k < a.n; ++k)   // source and result are cut at the same element
      need(((uintptr_t)a.src[k] - (uintptr_t)whole.src[k]) * os == ((uintptr_t)a.dst - (uintptr_t)whole.dst) * is);
    for (uint8_t w : written) need(w == 1);
    return good;
  }
};
static int nway_kernel_seen[5];   // wide, realign, shift, scaled wide, scaled narrow
static bool replay_nway(const ftk::NwayArgs& in, size_t unit, size_t len, bool first = false) {
  NwayReplay r{in, in, unit, unit, len, std::vector<uint8_t>(len * unit)};
  // the order of run_policy() in reduce_nway.cu
  if (ftk::layout_wide(in, len * unit, unit, &r.a)) { ++nway_kernel_seen[0]; r.wide(32, 32, 32, first); }
  else if (ftk::layout_realign(in, len * unit, unit, &r.a)) { ++nway_kernel_seen[1]; r.realign(first); }
  else { ++nway_kernel_seen[2]; ftk::layout_shift(in, len * unit, unit, &r.a); r.shift(); }
  return r.done();
}
static bool replay_scaled(const ftk::NwayArgs& in, bool in_bf16, bool out_bf16, size_t len, bool first) {
  const size_t is = in_bf16 ? 2 : 4, os = out_bf16 ? 2 : 4;
  NwayReplay r{in, in, is, os, len, std::vector<uint8_t>(len * os)};
  bool wide = false;
  if (!ftk::layout_scaled(in, len, in_bf16, out_bf16, &r.a, &wide)) return true;   // an element at a time
  ++nway_kernel_seen[wide ? 3 : 4];
  r.wide(wide ? 32 : 16, 32 / is * os, wide && 32 / is * os >= 32 ? 32 : 16, first);
  return r.done();
}
static void nway_layouts() {
  const auto at = [](int vector, size_t offset) { return (void*)(((uintptr_t)(vector + 1) << 32) + offset); };
  for (size_t unit : {1, 2, 4, 8}) {
    const size_t offsets[] = {0, unit, 16 - unit, 16, 16 + unit, 32 - unit, 32, 96 + unit, 128 - unit};
    std::vector<size_t> lens;
    for (size_t bytes = unit; bytes <= 216; bytes += unit) lens.push_back(bytes / unit);
    for (size_t edge : {2048, 3968, 4096, 7936, 8192})   // CTAs of the kernels, and the size from which a body starts on a line
      for (long long off : {-40, -8, 0, 8, 40, 168}) lens.push_back((size_t)((long long)edge + off) / unit);
    for (size_t d : offsets)
      for (size_t s0 : offsets)
        for (size_t s1 : offsets) {
          ftk::NwayArgs in{};
          in.n = 2;
          in.dst = at(0, d); in.src[0] = at(1, s0); in.src[1] = at(2, s1);
          for (size_t len : lens) EXPECT(replay_nway(in, unit, len) && replay_nway(in, unit, len, true));
          if (unit != 2 && unit != 4) continue;
          for (bool out_bf16 : {false, true})
            if (d % (out_bf16 ? 2 : 4) == 0)
              for (size_t len : lens) EXPECT(replay_scaled(in, unit == 2, out_bf16, len, false) && replay_scaled(in, unit == 2, out_bf16, len, true));
        }
    for (size_t bytes : {(3u << 20) - 40, 3u << 20, (3u << 20) + 56}) {   // where the shifted kernel changes its CTAs
      ftk::NwayArgs in{};
      in.n = 3;
      in.dst = at(0, unit); in.src[0] = at(1, 0); in.src[1] = at(2, 24); in.src[2] = at(3, 16 - unit);
      EXPECT(replay_nway(in, unit, bytes / unit));
    }
  }
  for (int seen : nway_kernel_seen) EXPECT(seen > 1000);
}

// Which CTAs of a call fetch ahead and which ask for the successor.  Asking costs a CTA's time at the chip's front end: no more
// may ask than it takes, or calls whose data lies in L2 get slower (fp32 x2 of 8 M 9.2 us instead of 7.9).
static void seams() {
  for (unsigned long long moved : {1ull, (50ull << 20) - 1}) EXPECT(ftk::seam_of(moved, 8192, 100000).ahead == 0 && ftk::seam_of(moved, 8192, 100000).ask == ftk::kNoCta);
  for (unsigned n : {2, 3, 8, 16})
    for (unsigned long long moved : {50ull << 20, (100ull << 20) - 1, 100ull << 20, 2400ull << 20}) {
      const unsigned fetched = n * ftk::kWideThreads * 32;
      const unsigned long long ctas = moved / (n + 1) / (ftk::kWideThreads * 32), most = moved < (100u << 20) ? 2368 : 2960;
      const ftk::Seam s = ftk::seam_of(moved, fetched, ctas);
      EXPECT(s.ahead > 0 && (unsigned long long)s.ahead * fetched <= (12u << 20));
      EXPECT(s.ask < ctas && ctas - s.ask == std::min(ctas, most));   // the last ones, all of a call that has no more
    }
}

// Gathered copies that L2 holds stay there for whoever reads them.
static void halves_in_l2() {
  for (uint64_t mb : {33, 58, 64, 84, 99}) EXPECT(!ftk::halves_stream(true, mb << 20) && ftk::halves_stream(false, mb << 20));
  for (uint64_t mb : {1, 24, 31}) EXPECT(!ftk::halves_stream(true, mb << 20) && !ftk::halves_stream(false, mb << 20));
  for (uint64_t mb : {126, 200, 4000}) EXPECT(ftk::halves_stream(true, mb << 20) && ftk::halves_stream(false, mb << 20));
}

int main(int argc, char** argv) {
  const bool threads = argc > 1 && !std::strcmp(argv[1], "threads");
  if (!threads) { proc_world_forked(); plans_and_snapshot(); device_tables(); world_programs(); nway_layouts(); seams(); halves_in_l2(); heap_offsets(); enumerators_and_models(); policy_and_json(); fd_passing(); }
  world_program_cache();
  thread_world(false);
  thread_world_phases();
  thread_world_small_message_twins();
  thread_world_all_shapes();
  thread_world(true);
  std::printf(fails ? "%d FAILURES\n" : "selftest ok\n", fails);
  return fails ? 1 : 0;
}
