// The word of page-locked memory in which a kernel reports that a wait gave up.
// It is cleared by the call whose kernels set it, on every way out: a word left
// set would be reported by the next call that has nothing to do with it.
#pragma once

namespace xyzgpu {

// One call's use of the word.  finish() waits for the call's kernels and returns
// an error code, or 0.
template <class Finish>
class ErrorWordUse {
 public:
  ErrorWordUse(volatile int *word, Finish finish) : word_(word), finish_(finish) {}
  ErrorWordUse(const ErrorWordUse &) = delete;
  ~ErrorWordUse() {
    if (!taken_) take();  // the call returns with an error of its own
  }
  // Waits; whether a kernel of the call set the word, which is cleared.
  bool take() {
    taken_ = true;
    status_ = static_cast<int>(finish_());
    bool const set = *word_ != 0;
    *word_ = 0;
    return set;
  }

  int status() const { return status_; }  // of the wait

 private:
  volatile int *word_;
  Finish finish_;
  int status_ = 0;
  bool taken_ = false;
};

}  // namespace xyzgpu
