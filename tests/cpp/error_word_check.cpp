// A kernel's report that a wait gave up belongs to the call that launched it
// (xyz_b200/csrc/error_word.h).  Exit code 1 on a failure.
#include "../../xyz_b200/csrc/error_word.h"

using namespace xyzgpu;

int word = 0;

// A call whose kernel sets the word (or not) when the stream is waited for, and
// which fails by itself after the launch (or not): 0, 1 (wait gave up), 2 (own).
int call(bool kernel_gives_up, bool own_failure) {
  ErrorWordUse use(&word, [=] {
    word |= kernel_gives_up;
    return 0;
  });
  if (own_failure) return 2;
  return use.take() ? 1 : 0;
}

int main() {
  bool ok = call(false, false) == 0 && call(true, false) == 1 && call(false, false) == 0;
  ok = ok && call(true, true) == 2 && word == 0 && call(false, false) == 0;
  return ok ? 0 : 1;
}
