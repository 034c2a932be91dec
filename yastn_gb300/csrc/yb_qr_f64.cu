// The blocked Householder QR (yb_qr.cuh) for FP64 blocks.
#include "yb_qr.cuh"

namespace yb {

int qr_factor_f64(void* work, void* work32, const int64_t* blocks, int n_blocks, int64_t* qctrl,
                  int qctrl_words, cudaStream_t s) {
  return qr_factor<double, float>(work, work32, blocks, n_blocks, qctrl, qctrl_words, s);
}

}  // namespace yb
