// cert_weight.cu -- to_weight_map of the certified mode with the chunked
// pointing (kernels in cert_scatter.cuh).

#include "cert_scatter.cuh"

namespace so3g {

int cert_to_weight_map(int coord, int kind, ScatterArgs &a, int n_det, long long n_seg,
                       long long max_len, cudaStream_t st, void **work) {
    return cx_scatter<true>(coord, kind, a, n_det, n_seg, max_len, st, work);
}

}  // namespace so3g
