// What the library's host code asks of the GPU, on the stand-in runtime of
// host_cuda.h.  One check per argument; exit status 0 when it holds.
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "../../exocubed_b200/csrc/exo_internal.h"
#include "../../include/exo_b200.h"
#include "host_cuda.h"

static int fail(const char* what) {
  std::printf("FAIL %s: %s\n", what, exo_last_error());
  return 1;
}
static bool is(const HostLaunch& l, const char* name) {
  return l.kernel.find(name) != std::string::npos;
}
static bool forward(const HostLaunch& l) {
  return is(l, "k_implicit_columns") && !is(l, "_bwd");
}

enum Form { FULL, PARTIAL, NOALLOC };
static int columns(Form form, int ncol, int L, double* scratch, double dt = 60.) {
  static double any[64];  // never read: nothing runs
  const double* a = any;
  if (form == NOALLOC)
    return exo_implicit_columns_noalloc(ncol, L, a, any, a, a, a, a, dt, 1.4, -9.8, nullptr);
  return form == FULL ? exo_implicit_columns(ncol, L, a, any, a, a, a, a, dt, 1.4, -9.8, scratch,
                                             nullptr)
                      : exo_partial_correction_columns(ncol, L, a, any, a, a, a, a, dt, 1.4, -9.8,
                                                       scratch, nullptr);
}

// Two host threads solve columns on one stream with one scratch: the two
// launches of a call, which hand the factors over in the scratch, stand side
// by side in the stream.  Each forward sweep gives the other thread's time to
// get between.
static int check_pairs(Form form) {
  std::mutex m;
  std::condition_variable cv;
  int sweeps = 0;
  host_launches_clear();
  host_on_launch([&](const HostLaunch& l) {
    if (!forward(l)) return;
    std::unique_lock<std::mutex> lk(m);
    const int mine = ++sweeps;
    cv.notify_all();
    cv.wait_for(lk, std::chrono::milliseconds(300), [&] { return sweeps > mine; });
  });
  double scratch[8];
  int rc[2] = {1, 1};
  std::thread a([&] { rc[0] = columns(form, 4, 8, scratch); });
  std::thread b([&] { rc[1] = columns(form, 4, 8, scratch); });
  a.join();
  b.join();
  host_on_launch(nullptr);
  const std::vector<HostLaunch> all = host_launches();
  if (rc[0] || rc[1] || all.size() != 4) return fail("two calls of two launches");
  for (int c = 0; c < 4; c += 2)
    if (!forward(all[c]) || !is(all[c + 1], "_bwd") || all[c].thread != all[c + 1].thread)
      return fail("a call's sweep and back substitution side by side in the stream");
  return 0;
}

// The deepest columns the hooks take (the radial tables of a block stand in its
// shared memory beside the warps' own), and the first ones they refuse.
static int check_levels() {
  double scratch[8];
  for (Form form : {FULL, PARTIAL, NOALLOC})
    for (int L : {1, 250, 4899, 4900, 5518}) {
      host_launches_clear();
      if (columns(form, 3, L, scratch)) return fail("a column solve of this depth");
      const std::vector<HostLaunch> all = host_launches();
      if (all.size() != 2 || all[0].grid * all[0].block < 3) return fail("two launches over 3 columns");
    }
  for (Form form : {FULL, PARTIAL, NOALLOC}) {
    host_launches_clear();
    if (columns(form, 3, 5519, scratch) != EXO_ERR_ARG) return fail("EXO_ERR_ARG past the deepest column");
    if (columns(form, 0, 5519, scratch)) return fail("no columns of any depth");
    if (!host_launches().empty()) return fail("no launch for a refused call");
  }
  return 0;
}

// A bounded wait that gives up inside the back substitution is an error of the
// call that launched it, whole arrays and views alike.
static int check_timeout(int precision, int implicit_flag) {
  exo_config cfg;
  exo_config_default(&cfg, EXO_EQN_IDEAL);
  cfg.N = 6;
  cfg.L = 4;
  cfg.precision = precision;
  cfg.implicit_flag = implicit_flag;
  exo_ctx* c = nullptr;
  if (exo_create(&cfg, &c)) return fail("exo_create");
  const size_t n = (size_t)6 * 5 * 12 * 12 * 10;
  std::vector<double> du(n, 1.), w(n, 1.);
  if (exo_solve_implicit_3d(c, du.data(), w.data(), 60.)) return fail("a solve without a timeout");
  // the kernel's first argument is the batch, whose first member is the view
  host_on_launch([](const HostLaunch& l) {
    if (!is(l, "kb_implicit_bwd")) return;
    const exo::DevView* const* batch = (const exo::DevView* const*)l.args[0];
    batch[0]->sc->timeout = 1;
  });
  const int rc = exo_solve_implicit_3d(c, du.data(), w.data(), 60.);
  host_on_launch(nullptr);
  if (rc != EXO_ERR_TIMEOUT) return fail("EXO_ERR_TIMEOUT from exo_solve_implicit_3d");
  exo_array_view v[6];
  for (int p = 0; p < 6; ++p) {
    v[p] = exo_array_view{};
    v[p].data = w.data() + p * (n / 6);
    v[p].dtype = EXO_DTYPE_F64;
    v[p].nx4 = 5;
    v[p].nx3 = v[p].nx2 = 12;
    v[p].nx1 = 10;
    v[p].stride[0] = 1440;
    v[p].stride[1] = 120;
    v[p].stride[2] = 10;
    v[p].stride[3] = 1;
    v[p].device = -1;
  }
  if (exo_solve_implicit_3d_views(c, v, v, 60.) != EXO_ERR_TIMEOUT)
    return fail("EXO_ERR_TIMEOUT from exo_solve_implicit_3d_views");
  exo_destroy(c);
  return 0;
}

// The mixed 5x5 solve's shared memory leaves its loads enough of L1: not more than 61
// doubles a column beside the radial tables, or four blocks of 64 columns
// within the 196 KB that leave 60 KB of L1 (6 x 8^2 columns, and 6 x 32^2,
// which is more than a block for every second SM).
static int check_fused_smem(int N) {
  for (int L : {1, 32, 96, 99, 100, 250}) {
    exo_config cfg;
    exo_config_default(&cfg, EXO_EQN_IDEAL);
    cfg.N = N;
    cfg.L = L;
    cfg.precision = EXO_PREC_MIXED;
    cfg.implicit_flag = 9;
    exo_ctx* c = nullptr;
    if (exo_create(&cfg, &c)) return fail("exo_create");
    const int nc1 = L + 6;
    std::vector<double> du((size_t)6 * 5 * (N + 6) * (N + 6) * nc1, 1.), w(du);
    for (int tile : {32, 64, 128}) {
      const int tiles[6] = {0, 0, 0, tile, 0, 0};
      if (exo_set_tiles(c, tiles)) return fail("exo_set_tiles");
      host_launches_clear();
      if (exo_solve_implicit_3d(c, du.data(), w.data(), 60.)) return fail("a solve");
      const std::vector<HostLaunch> all = host_launches();
      if (all.size() != 1 || !is(all[0], "kb_implicit_fused") || all[0].block != (unsigned)tile)
        return fail("one launch at the tile");
      const size_t small = (size_t)(61 * tile + 3 * (nc1 + 1)) * sizeof(double);
      const size_t block = (all[0].smem + sizeof(exo::DevView) + 127) / 128 * 128 + 1024;
      if (all[0].smem > small && !(tile == 64 && 4 * block <= 196 * 1024)) {
        std::printf("%d levels, tile %d: %zu bytes\n", L, tile, all[0].smem);
        return fail("shared memory that leaves an L1");
      }
    }
    exo_destroy(c);
  }
  return 0;
}

int main(int argc, char** argv) {
  const char* what = argc > 1 ? argv[1] : "";
  int rc = 2;
  if (!std::strcmp(what, "pairs")) rc = check_pairs(FULL) + check_pairs(PARTIAL) + check_pairs(NOALLOC);
  if (!std::strcmp(what, "levels")) rc = check_levels();
  if (!std::strcmp(what, "fused_smem")) rc = check_fused_smem(8) + check_fused_smem(32);
  if (!std::strcmp(what, "timeout"))
    rc = check_timeout(EXO_PREC_FP64, 9) + check_timeout(EXO_PREC_FP64, 1) +
         check_timeout(EXO_PREC_MIXED, 1) + check_timeout(EXO_PREC_MIXED_F32_SOLVE, 9);
  if (rc == 0) std::printf("%s: ok\n", what);
  return rc;
}
