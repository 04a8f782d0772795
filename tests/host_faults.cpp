// host_faults.cpp -- the engine's host code on a fake CUDA runtime: what a call
// answers when a launch or an allocation fails, and what it does on a stream
// that is being captured.  One check a run (argv[1]); exit status 0 = it holds.
#include "fake_cuda.h"

#include <vector>

#include "mlp_gpu.h"

#define REQUIRE(c)                                                                 \
  do {                                                                             \
    if (!(c)) {                                                                    \
      std::fprintf(stderr, "%s:%d: %s (%s)\n", __FILE__, __LINE__, #c, mlp_last_error()); \
      return 1;                                                                    \
    }                                                                              \
  } while (0)

static mlp_problem_t problem(int n, int dmax) {
  std::vector<int32_t> D((size_t)n * n);
  for (int a = 0; a < n; a++)
    for (int b = 0; b < n; b++) D[(size_t)a * n + b] = a == b ? 0 : 1 + (a * 7 + b * 7) % dmax;
  D[1] = D[n] = dmax;
  mlp_problem_t p = nullptr;
  return mlp_problem_create_matrix(n, D.data(), 1, &p) == 0 ? p : nullptr;
}

static std::vector<int32_t> tour(int n) {
  std::vector<int32_t> t(n + 1, 0);
  for (int q = 0; q < n; q++) t[q] = q;
  return t;
}

// A batch's result is not read when its kernel could not be launched.
static int batch_result() {
  const int n = 50;
  mlp_batch_t b = nullptr;
  mlp_problem_t p = problem(n, 100);
  REQUIRE(p && mlp_batch_create(0, &b) == 0);
  int32_t job = -1;
  const std::vector<int32_t> t = tour(n);
  REQUIRE(mlp_batch_add(b, p, t.data(), n + 1, &job) == 0 && mlp_batch_reset(b) == 0);
  for (const char* what : {"launch_result", "cudaStreamSynchronize"})
    for (const cudaError_t e : {cudaErrorMemoryAllocation, cudaErrorLaunchFailure}) {
      fake::fail(what, e);
      std::vector<int32_t> out(n + 1, -7);
      mlp_dvnd_stats_t st;
      const int want = e == cudaErrorMemoryAllocation ? MLP_ERR_NOMEM : MLP_ERR_CUDA;
      REQUIRE(mlp_batch_result(b, job, out.data(), n + 1, nullptr) == want);
      REQUIRE(mlp_batch_result(b, job, out.data(), n + 1, &st) == want);
      for (int32_t v : out) REQUIRE(v == -7);
      fake::fails.clear();
      REQUIRE(mlp_batch_result(b, job, out.data(), n + 1, &st) == 0);
    }
  mlp_batch_destroy(b);
  mlp_problem_destroy(p);
  return 0;
}

// The sweeps of a solver launch on a capturing stream whatever was switched
// before or during the capture: no tile list is left to be built by a launch.
static int captured_sweeps() {
  const int n = 400;
  mlp_problem_t p = problem(n, 65535);  // 64-bit costs that leave 32 bits
  for (int wide = 0; wide < 2; wide++)
    for (int shape = -1; shape < 14; shape++) {
      mlp_solver_t s = nullptr;
      REQUIRE(p && mlp_solver_create(p, wide, &s) == 0);
      const std::vector<int32_t> t = tour(n);
      REQUIRE(mlp_solver_set_tour(s, t.data(), n + 1) == 0);
      if (shape >= 0) REQUIRE(mlp_solver_set_tile_shape(s, shape) == 0);
      auto sweep = [&] {
        fake::capturing = true;
        const int st = mlp_solver_sweep(s, MLP_NB_ALL, 1, nullptr);
        fake::capturing = false;
        return st;
      };
      REQUIRE(sweep() == 0);
      for (int variant : {0, 1, 0}) {
        REQUIRE(mlp_solver_set_sweep_kernel(s, variant) == 0);
        REQUIRE(sweep() == 0);
      }
      for (int variant : {1, 0, 1}) {
        fake::capturing = true;
        const int st = mlp_solver_set_sweep_kernel(s, variant);
        fake::capturing = false;
        REQUIRE(st == 0 && sweep() == 0);
      }
      for (int on : {1, 0}) {
        REQUIRE(mlp_solver_set_total(s, on) == 0);
        for (int variant : {0, 1}) {
          REQUIRE(mlp_solver_set_sweep_kernel(s, variant) == 0);
          REQUIRE(sweep() == 0);
        }
      }
      // A mask set outside the capture.
      REQUIRE(mlp_solver_sweep(s, 1, 1, nullptr) == 0 && mlp_solver_sweep(s, MLP_NB_ALL, 1, nullptr) == 0);
      REQUIRE(sweep() == 0);
      mlp_solver_destroy(s);
    }
  mlp_problem_destroy(p);
  return 0;
}

// Starts are built whichever allocation of the ordered rows fails; any other
// failing allocation is reported.
static int constructor_memory() {
  const int n = 50;
  mlp_problem_t p = problem(n, 100);
  REQUIRE(p != nullptr);
  const uint32_t seed = 3;
  std::vector<int32_t> t(n + 1);
  fake::calls.clear();
  REQUIRE(mlp_problem_random_tours(p, 1, &seed, 0.5f, t.data()) == 0 && fake::grasp_table != nullptr);
  const int allocs = fake::calls["cudaMallocAsync"], sorts = fake::calls["launch_grasp_sort"];
  REQUIRE(allocs == 5 && sorts == 1);  // tours, tasks, flag; the rows' jobs and table
  for (int k = 0; k < allocs; k++)
    for (bool all : {false, true}) {  // the k-th alone fails, or all from it on
      fake::calls.clear();
      fake::fail("cudaMallocAsync", cudaErrorMemoryAllocation, k);
      fake::once = !all;
      fake::grasp_table = &fake::calls;
      const int st = mlp_problem_random_tours(p, 1, &seed, 0.5f, t.data());
      fake::fails.clear();
      fake::once = false;
      if (k < 3) {
        REQUIRE(st == MLP_ERR_NOMEM && fake::calls["launch_grasp"] == 0);
      } else {
        REQUIRE(st == 0 && fake::grasp_table == nullptr);
        REQUIRE(fake::calls["launch_grasp"] == 1 && fake::calls["launch_grasp_sort"] == 0);
      }
      REQUIRE(fake::held == 0);
    }
  mlp_problem_destroy(p);
  return 0;
}

// Rows are ordered where enough starts use them or few are to be ordered, not
// for a start or two of each of very many matrices.
static int constructor_rule() {
  struct Case {
    int n, matrices, starts;
    bool rows;
  };
  for (const Case c : {Case{60, 1, 1, true}, Case{60, 64, 1, true}, Case{60, 512, 1, true}, Case{60, 1100, 1, false},
                       Case{60, 2000, 1, false}, Case{60, 1100, 4, true}, Case{300, 512, 1, true}, Case{300, 900, 1, false},
                       Case{300, 600, 4, true}}) {
    mlp_batch_t b = nullptr;
    REQUIRE(mlp_batch_create(0, &b) == 0);
    std::vector<mlp_problem_t> ps;
    for (int m = 0; m < c.matrices; m++) {
      ps.push_back(problem(c.n, 100));
      for (int q = 0; q < c.starts; q++) REQUIRE(mlp_batch_add_random(b, ps.back(), q, 0.5f, nullptr) == 0);
    }
    fake::grasp_table = &fake::calls;
    REQUIRE(mlp_batch_reset(b) == 0);
    if ((fake::grasp_table != nullptr) != c.rows) std::fprintf(stderr, "n %d, %d x %d\n", c.n, c.matrices, c.starts);
    REQUIRE((fake::grasp_table != nullptr) == c.rows);
    mlp_batch_destroy(b);
    for (mlp_problem_t p : ps) mlp_problem_destroy(p);
  }
  return 0;
}

// Without the one-launch search (its kernels refused by the device) the iterated
// kernels serve; nothing is refused.
static int no_small_search() {
  const int n = 50;
  mlp_problem_t p = problem(n, 100);
  const std::vector<int32_t> t = tour(n);
  for (bool refused : {false, true}) {
    mlp_solver_t s = nullptr;
    if (refused) fake::fail("configure_small", cudaErrorInvalidValue);
    REQUIRE(p && mlp_solver_create(p, 0, &s) == 0);
    fake::fails.clear();
    REQUIRE(mlp_solver_set_tour(s, t.data(), n + 1) == 0);
    fake::calls.clear();
    REQUIRE(mlp_solver_dvnd_async(s, MLP_NB_ALL, 5) == 0);
    REQUIRE(fake::calls["launch_dvnd_small"] == (refused ? 0 : 1) && fake::calls["launch_merge_one"] == (refused ? 5 : 0));
    mlp_solver_destroy(s);
  }
  mlp_problem_destroy(p);
  return 0;
}

int main(int argc, char** argv) {
  const std::string check = argc > 1 ? argv[1] : "";
  if (check == "batch_result") return batch_result();
  if (check == "captured_sweeps") return captured_sweeps();
  if (check == "constructor_memory") return constructor_memory();
  if (check == "constructor_rule") return constructor_rule();
  if (check == "no_small_search") return no_small_search();
  std::fprintf(stderr, "unknown check\n");
  return 2;
}
