// Queue arithmetic at the ends of its range (ceil_div, beyond_queue of
// xyz_b200/csrc/common.cuh).  Exit code 1 on a failure.
#include <climits>
#include <cmath>

#include "../../xyz_b200/csrc/common.cuh"

using namespace xyzgpu;

int main() {
  bool ok = true;
  for (int per : {1, 32, 128, 4736})
    for (int n : {0, 1, 31, 32, 33, 4735, 4736, 4737, INT_MAX - 4736, INT_MAX - 31, INT_MAX - 1, INT_MAX}) {
      long long const want = (static_cast<long long>(n) + per - 1) / per;
      ok = ok && ceil_div(n, per) == want;
      // items taken by the last of 200,000 lanes once the queue is empty
      for (uint32_t past : {0u, 1u, 31u, 4736u, 200000u})
        ok = ok && beyond_queue(static_cast<int>(static_cast<uint32_t>(n) + past), n);
      ok = ok && (n == 0 || !beyond_queue(n - 1, n)) && (n < 2 || !beyond_queue(0, n));
    }
  return ok ? 0 : 1;
}
