// Checks of the resident CG kernels' launch rules
// (tetfit_b200/csrc/resident_choice.hpp), built and run by
// tests/test_resident_choice.py: every choice covers the rows with at most its
// rows a thread and the device's blocks, and nothing is chosen that the device's
// answers do not allow.  Prints "ok" and exits 0, or names the failed check.
#include <cstdio>
#include <cstdlib>

#include "../tetfit_b200/csrc/resident_choice.hpp"

using namespace tf;

static void need(bool ok, const char* what, long long at) {
  if (ok) return;
  std::printf("%s at %lld\n", what, at);
  std::exit(1);
}

int main() {
  const int sms = 148;
  auto room = [](int) { return 18000; };
  auto none = [](int) { return 0; };
  auto fifteen = [] { return 15; };

  // standalone: flat to 20,480 rows, clusters of 8 to 184,320, flat to 606,208
  for (int64_t n = 1; n <= 700000; n += n < 300 ? 1 : 97) {
    const ResidentChoice f = pcg_flat(n, sms, room), c = pcg_clustered(n, fifteen, room);
    need((f.rows > 0) == (n <= 606208), "flat range", n);
    need((c.rows > 0) == (n > 20480 && n <= 184320), "cluster range", n);
    for (const ResidentChoice& q : {f, c}) {
      if (!q.rows) continue;
      need(q.warps >= 8 && q.warps <= kPcgThreads / 32, "warps", n);
      need(q.blocks >= 1 && q.blocks <= sms && q.blocks % q.cluster == 0, "blocks", n);
      // as pcg_launch_resident cuts the rows
      const int64_t slices = (n + 31) / 32, per = (slices + q.blocks - 1) / q.blocks;
      need(per <= (int64_t)q.warps * q.rows, "rows a thread", n);
    }
    need(pcg_flat(n, sms, none).rows == 0, "flat without shared memory", n);
    need(pcg_clustered(n, fifteen, none).rows == 0, "clusters without shared memory", n);
    need(pcg_clustered(n, [] { return 0; }, room).rows == 0, "clusters that do not run", n);
  }
  // a device that gives some of the kernels their shared memory
  auto some = [](int rows) { return rows == 2 ? 0 : 18000; };
  need(pcg_flat(148 * 512 + 1, sms, some).rows == 0 && pcg_flat(148 * 512, sms, some).rows == 1, "refused kernel", 2);

  // groups
  auto clusters = [](int, int, int size) { return size == 16 ? 8 : 15; };
  auto refused = [](int, int, int) { return 0; };
  for (int fp32 = 0; fp32 < 2; fp32++)
    for (int64_t n = 1; n <= 20000; n++) {
      const auto all = group_choices({n}, sms, fp32, room, clusters);
      need(all.empty() == (n > 148 * 16 * 8), "group range", n);
      const bool one = n <= 256, eight = n > 80 * 8 && n <= 120 * 16 * (fp32 ? 4 : 2);
      if (!all.empty()) {
        need(all.size() == (one || eight ? 2u : 1u), "clusters", n);
        need(all.back().cluster == 1 && all.back().blocks == 0, "flat last", n);
      }
      for (const ResidentChoice& q : all) {
        const int64_t blocks = q.blocks ? q.blocks : (n + q.warps * q.rows - 1) / (q.warps * q.rows);
        need(q.warps >= 8 && q.warps <= kCgResidentWarps && q.rows >= 1 && q.rows <= kCgResidentRows, "shape", n);
        need(blocks <= sms && blocks * q.warps * q.rows >= n, "rows a thread", n);
      }
      const auto flat = group_choices({n}, sms, fp32, room, refused);
      need(flat.size() == (all.empty() ? 0u : 1u), "clusters that do not run", n);
      need(group_choices({n}, sms, fp32, none, clusters).empty(), "group without shared memory", n);
    }
  need(group_choices({300, 0}, sms, true, room, clusters).empty(), "member without rows", 0);
  need(group_choices({40, 700, 3000}, sms, false, room, clusters).size() == 1, "several members", 3);
  std::printf("ok\n");
  return 0;
}
