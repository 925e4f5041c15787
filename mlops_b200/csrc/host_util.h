// Host-side helpers shared by the C-ABI entry points: status codes, the driver
// entry point used to encode TMA tensor maps (fetched at run time so the library
// links against the CUDA runtime only) and a per-device SM count cache.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

// Return codes of every extern "C" entry point (see include/b200moe.h).
enum : int {
  B200MOE_OK = 0,
  B200MOE_ERR_ARG = -1,        // null pointer, negative size, unsupported combination
  B200MOE_ERR_ALIGN = -2,      // pointer / pitch alignment requirement not met
  B200MOE_ERR_TENSORMAP = -3,  // cuTensorMapEncodeTiled refused the operand
  B200MOE_ERR_LAUNCH = -4,     // kernel launch failed (cudaGetLastError != success)
  B200MOE_ERR_DRIVER = -5,     // driver entry point unavailable
  B200MOE_ERR_LIMIT = -6       // size beyond a documented maximum
};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_tiled();
// Rows of tiles a GEMM walks together (banded_tile): `bytes` is what one row of tiles reads of the
// operand that runs along it (a group's whole weight, or its rows of X in a weight gradient).
int tile_band(long long bytes);
int tile_band(long long bytes, long long rows, int groups);  // ... of a GEMM over `rows` rows in `groups` groups
// b200moe_routing_probability_sum and, with counts (the sort's, int64) and aux, the auxiliary loss of
// the rows as one sequence.
int launch_routing_statistics(const float* logits, long long ld, long long tokens, int experts, int mode,
                              void* workspace, float* probability_sum, const long long* counts, int top_k, float* aux,
                              cudaStream_t s);
// b200moe_routing_gradient, with the gradient written as two bf16 pieces [tokens, experts] as well
// (high + low; both or neither).
int launch_routing_gradient(const float* logits, long long ld, long long tokens, int experts, int top_k, int mode,
                            const int32_t* ids, const float* route_weights, const float* grad_route_weights,
                            const float* grad_aux, const float* frequency, float aux_scale,
                            const float* grad_probability_sum, float* grad_logits, long long ldg, void* high,
                            void* low, cudaStream_t s);
int sm_count_device();      // SM count of the current device (cached per device)
int sm_count();             // CTAs a persistent kernel may launch: the SM count, or the limit below
void set_cta_limit(int n);  // n > 0: persistent kernels launch at most n CTAs; 0: no limit

// Encodes a row-major tensor of `rank` dims.  dims[0] is the innermost (contiguous)
// extent in elements; strides_bytes[i] is the byte pitch of dims[i+1].
int encode_tensor_map(CUtensorMap* map, CUtensorMapDataType dtype, int rank, const void* base,
                      const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box,
                      CUtensorMapSwizzle swizzle);

inline int launch_status() { return cudaGetLastError() == cudaSuccess ? B200MOE_OK : B200MOE_ERR_LAUNCH; }

}  // namespace b200
