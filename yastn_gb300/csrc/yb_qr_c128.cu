// The blocked Householder QR (yb_qr.cuh) for complex128 blocks.
#include "yb_qr.cuh"

namespace yb {

int qr_factor_c128(void* work, void* work32, const int64_t* blocks, int n_blocks, int64_t* qctrl,
                  int qctrl_words, cudaStream_t s) {
  return qr_factor<double2, float2>(work, work32, blocks, n_blocks, qctrl, qctrl_words, s);
}

}  // namespace yb
