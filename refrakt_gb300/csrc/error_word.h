// Error words of the tensor-core kernels (gemm.cu, conv.cu; error_word.cpp).
#pragma once

namespace rfk {

// A word of pinned host memory that a kernel writes only when one of its bounded waits runs out, so the host
// reads it after a synchronisation without a copy (two copies of a device word took 20 us per call).  Each call that
// synchronises, and each denoiser, holds its own: another stream's, thread's or device's failure is not taken for it.
class ErrorWord {
  public:
    ErrorWord() = default;
    ErrorWord(const ErrorWord&) = delete;
    ErrorWord& operator=(const ErrorWord&) = delete;
    ~ErrorWord();
    // takes a word, zero, on any device; false when none can be allocated.  Not during stream capture
    bool acquire();
    int* get() const { return p_; }
    // its value, cleared; after the kernels that were given it have finished (0: no wait ran out)
    int take();

  private:
    int* p_ = nullptr;
};

}  // namespace rfk
