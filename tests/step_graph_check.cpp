// Checks of the capture of steps (tetfit_b200/csrc/step_graph.hpp) against a
// runtime that refuses one of its calls, built and run by
// tests/test_step_graph.py: no graph is left over, the stream is not left
// capturing, and no exception gets out.  Prints "ok", or names the failed check.
#include <cstdio>
#include <cstdlib>
#include <stdexcept>

#include "../tetfit_b200/csrc/step_graph.hpp"

static int fail_at = 0;  // 1 begin, 2 launch, 3 end, 4 end with a graph, 5 instantiate
static bool capturing = false, error = false;
static int graphs = 0, launched = 0;

struct Fake {
  using Stream = int;
  using Graph = int*;
  using Exec = int*;
  static int storage;
  static bool refuse(int call) {
    if (fail_at == call) error = true;
    return fail_at == call;
  }
  static bool begin(Stream) {
    if (refuse(1)) return false;
    capturing = true;
    return true;
  }
  static bool end(Stream, Graph* g) {
    if (!capturing) std::exit(2);
    capturing = false;
    if (refuse(3)) return false;
    *g = &storage;
    graphs++;
    return !refuse(4);
  }
  static bool instantiate(Exec* x, Graph) {
    *x = &storage;
    return !refuse(5);
  }
  static void destroy(Graph) { graphs--; }
  static void clear_error() { error = false; }
};
int Fake::storage = 0;

int main() {
  for (fail_at = 0; fail_at <= 5; fail_at++) {
    launched = 0;
    int* x = nullptr;
    try {
      x = tf::capture_steps<Fake>(0, [] {
        if (Fake::refuse(2)) throw std::runtime_error("refused");
        launched++;
      });
    } catch (...) {
      std::printf("exception at %d\n", fail_at);
      return 1;
    }
    if ((x != nullptr) != (fail_at == 0) || capturing || error || graphs != 0 ||
        launched != (fail_at == 1 || fail_at == 2 ? 0 : 1)) {
      std::printf("state after a refusal at %d\n", fail_at);
      return 1;
    }
  }
  std::printf("ok\n");
  return 0;
}
