// Whole forward of a Linear in one call: the prologue (quantisation, with the rank-32 down-projection where there is a
// branch) and the GEMM, enqueued back to back from one descriptor of the layer's constants.  Nothing is allocated and
// nothing is kept; what it saves is the caller's time between and around the two entry points, which is all the time that a
// small Linear takes: the kernels of 154 x 640 -> 1280 run for 8 us, the call took 28 us as separate entry points with three
// tensors between them and takes 17 us so.
#include "common.cuh"

namespace pq {
bool lowrank_sliced(int64_t K, int R);
namespace {
inline int64_t up256(int64_t v) { return (v + 255) / 256 * 256; }
}  // namespace
}  // namespace pq

using namespace pq;

extern "C" int64_t pq_int8_linear_scratch_bytes(int64_t M, int64_t K, int rank) {
  if (M < 0 || K <= 0 || rank < 0) return 0;
  return up256(M * K) + up256(M * 2 * rank) + up256(M * 4);
}

extern "C" int pq_int8_linear(const pq_linear_desc* d, const void* x, int64_t ldx, int64_t M, void* scratch,
                              int64_t scratch_bytes, void* out, int64_t ldo, void* stream) {
  if (d == nullptr) return PQ_ERR_NULL;
  if (M < 0 || d->N <= 0 || d->K <= 0) return PQ_ERR_SHAPE;
  if (d->rank != 0 && (!lowrank_sliced(d->K, d->rank) || d->lb == nullptr || d->lb_t == nullptr || d->a_t == nullptr))
    return PQ_ERR_UNSUPPORTED;
  if (M == 0) return PQ_OK;
  if (scratch == nullptr) return PQ_ERR_NULL;
  if (!aligned_to(scratch, 256)) return PQ_ERR_ALIGN;
  if (scratch_bytes < pq_int8_linear_scratch_bytes(M, d->K, d->rank)) return PQ_ERR_WORKSPACE;
  unsigned char* b = static_cast<unsigned char*>(scratch);
  int8_t* q = reinterpret_cast<int8_t*>(b);
  void* t = d->rank != 0 ? b + up256(M * d->K) : nullptr;
  float* s = reinterpret_cast<float*>(b + up256(M * d->K) + up256(M * 2 * d->rank));
  int rc;
  if (d->rank != 0)
    rc = pq_quant_rows_lowrank(x, d->K, ldx, nullptr, 0, 0, d->dtype, M, d->a_t, d->K, d->rank, q, s, t, d->rank, d->workspace,
                               d->ws_bytes, stream);
  else
    rc = pq_quant_rows(x, d->dtype, M, d->K, ldx, q, s, stream);
  if (rc != PQ_OK) return rc;
  return pq_int8_gemm(q, d->K, s, d->w, d->ldw, d->s_col, d->bias, t, d->rank, d->rank != 0 ? d->lb : nullptr, d->ldb,
                      d->rank != 0 ? d->lb_t : nullptr, d->rank, d->dtype, out, d->dtype, ldo, M, d->N, d->K, d->workspace,
                      d->ws_bytes, nullptr, stream);
}

extern "C" int64_t pq_int8_linear_g32_scratch_bytes(int64_t M, int64_t K) {
  if (M < 0 || K <= 0) return 0;
  return up256(M * K) + up256(M * (K / 32) * 4);
}

extern "C" int pq_int8_linear_g32(const void* x, int dtype, int64_t ldx, const int8_t* w, int64_t ldw, const float* s_w,
                                  const float* bias, void* scratch, int64_t scratch_bytes, void* out, int64_t ldo, int64_t M,
                                  int64_t N, int64_t K, void* workspace, size_t ws_bytes, void* stream) {
  if (M < 0 || N <= 0 || K <= 0) return PQ_ERR_SHAPE;
  if (K % 128 != 0) return PQ_ERR_UNSUPPORTED;
  if (M == 0) return PQ_OK;
  if (scratch == nullptr) return PQ_ERR_NULL;
  if (!aligned_to(scratch, 256)) return PQ_ERR_ALIGN;
  if (scratch_bytes < pq_int8_linear_g32_scratch_bytes(M, K)) return PQ_ERR_WORKSPACE;
  int8_t* q = static_cast<int8_t*>(scratch);
  float* s_a = reinterpret_cast<float*>(static_cast<unsigned char*>(scratch) + up256(M * K));
  const int rc = pq_quant_rows_g32(x, dtype, M, K, ldx, q, s_a, stream);
  if (rc != PQ_OK) return rc;
  return pq_int8_gemm_g32(q, K, s_a, w, ldw, s_w, bias, out, dtype, ldo, M, N, K, workspace, ws_bytes, stream);
}
