#include "host_util.h"

#include <mutex>

namespace b200 {

EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(p);
    }
  });
  return fn;
}

static int g_cta_limit = 0;  // 0 = every SM

int sm_count() {
  const int n = sm_count_device();
  return (g_cta_limit > 0 && g_cta_limit < n) ? g_cta_limit : n;
}

void set_cta_limit(int n) { g_cta_limit = n > 0 ? n : 0; }

// Walked column by column, every row of tiles streams that operand again; while it stays in L2
// beside the rest this costs nothing, above some 50 MB it comes from HBM each time (28.2 GB instead
// of 2.3 GB for 32768 rows through a 28672 x 4096 E4M3 weight of 8 experts).  Bands of 16 rows make
// the tiles in flight on 148 SMs about square.  Measured column order / bands of 16, in us:
//   E4M3 GEMM, K = 4096     17 MB 577 / 576   34 MB 1149 / 1170   50 MB 1763 / 1761   67 MB 2488 / 2344
//                           117 MB 5574 / 4091
//   bf16 GEMM               34 MB 241 / 235   67 MB 512 / 456   117 MB 1006 / 803   235 MB 2257 / 1608
//   weight gradient         34 MB 2368 / 2424   67 MB 1711 / 1583   117 MB 3230 / 2757
// (one threshold for the three; the bf16 GEMM would gain 2% from a lower one).  Bands of 8 to 32 are
// within 3% of one another.
int tile_band(long long bytes) { return bytes > (40LL << 20) ? 16 : 1; }

// Where the groups have less than a whole tile of rows (decoding), nothing is read twice in either order
// and a band only spreads the tiles in flight over sixteen groups' weights.  Eight groups, 28672 x 4096,
// column order / bands, in us, by rows in all:
//   E4M3    128 163 / 167   512 175 / 178   1024 227 / 211   2048 393 / 342
//   bf16    128 308 / 315   512 317 / 327   1024 407 / 359   2048 685 / 534
int tile_band(long long bytes, long long rows, int groups) { return rows >= 128LL * groups ? tile_band(bytes) : 1; }

int sm_count_device() {
  static int cached[64];
  static bool have[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!have[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
    have[dev] = true;
  }
  return cached[dev];
}

int encode_tensor_map(CUtensorMap* map, CUtensorMapDataType dtype, int rank, const void* base,
                      const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box,
                      CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = get_encode_tiled();
  if (fn == nullptr) return B200MOE_ERR_DRIVER;
  cuuint64_t gdim[5];
  cuuint64_t gstr[5];
  cuuint32_t bdim[5];
  cuuint32_t estr[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bdim[i] = box[i];
    estr[i] = 1;
    if (i + 1 < rank) gstr[i] = strides_bytes[i];
  }
  CUresult r = fn(map, dtype, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstr, bdim, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? B200MOE_OK : B200MOE_ERR_TENSORMAP;
}

}  // namespace b200
