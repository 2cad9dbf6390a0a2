// One call per layer of a decode step: the new rows into the paged cache, attention over it, the merge of its partial results. Three
// launches; what it saves is host time: which kernel serves the shapes, the number of splits, the scratch they need and the layout of q, k
// and v were a dozen calls from Python per layer, 34 us per layer with the launches where the kernels of one short sequence take 13 us; 30 us so
// (14 us replayed from a captured graph, where the host has no part).
#include "common.cuh"

extern "C" {

int mfb_paged_decode_tc_supported(int Hq, int Hkv, int hd, int block_size);
int mfb_paged_decode_tc_splits(int B, int Hkv, int max_len);
int mfb_paged_decode_attention_tc_q(const void* q, long long ld_q, long long ld_head, const void* key_cache, const void* value_cache,
                                    const int* block_tables, const int* context_lens, const int* cu_q, const float* sink, void* out,
                                    void* scratch, int splits, int rows, int B, int Hq, int Hkv, int D, int DV, int num_blocks,
                                    int block_size, int max_blocks, int chunk, int window, int all_values, float scale, float softcap,
                                    long long ld_out, float out_scale, int* status, cudaStream_t stream);
int mfb_paged_decode_int8_supported(int Hq, int Hkv, int hd, int block_size);
int mfb_paged_decode_int8_splits(int B, int Hkv, int max_len);
int mfb_paged_decode_attention_int8(const void* q, long long ld_q, long long ld_head, const void* key_cache, const void* value_cache,
                                    const float* key_scale, const float* value_scale, const int* block_tables, const int* context_lens,
                                    void* out, void* scratch, int splits, int B, int Hq, int Hkv, int hd, int block_size, int max_blocks,
                                    float scale, cudaStream_t stream);
int mfb_reshape_and_cache_int8(const void* key, const void* value, void* key_cache, void* value_cache, float* key_scale,
                               float* value_scale, const int* slot_mapping, long long T, int heads, int hd, long long k_stride,
                               long long v_stride, cudaStream_t stream);
int mfb_reshape_and_cache(const void* key, const void* value, void* key_cache, void* value_cache, const int* slot_mapping, long long T,
                          int row_elems, long long k_stride, long long v_stride, cudaStream_t stream);
long long mfb_paged_decode_scratch_bytes(int B, int Hq, int hd, int splits);

// q [B, Hq, hd], k / v [B, Hkv, hd] bf16, strides in elements; caches [num_blocks, block_size, Hkv, hd] bf16, or int8 with scales
// [num_blocks, block_size, Hkv]; out [B, Hq, hd]. 0: launched. Positive: nothing was launched, that many bytes of scratch are needed.
// -1: nothing was launched, the general path takes the call. -2: likewise, but for contiguous q, k and v. Others: an error of a launch.
long long mfb_paged_decode_step(const void* q, long long q0, long long q1, long long q2, const void* k, long long k0, long long k1,
                                long long k2, const void* v, long long v0, long long v1, long long v2, void* key_cache,
                                void* value_cache, float* key_scale, float* value_scale, const int* slots, const int* tables,
                                const int* lens, void* out, void* scratch, long long scratch_bytes, int B, int Hq, int Hkv, int hd,
                                int num_blocks, int block_size, int max_blocks, float scale, int* status, cudaStream_t stream) {
  const bool i8 = key_scale != nullptr;
  if (B < 1 || (i8 ? !mfb_paged_decode_int8_supported(Hq, Hkv, hd, block_size) : !mfb_paged_decode_tc_supported(Hq, Hkv, hd, block_size))) return -1;
  auto off16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
  if (off16(key_cache) || off16(value_cache)) return -1;
  if (q2 != 1 || k2 != 1 || v2 != 1 || k1 != hd || v1 != hd || q1 < hd || q0 < hd || q1 % 8 || q0 % 8 || k0 % 8 || v0 % 8 ||
      off16(q) || off16(k) || off16(v))
    return i8 ? -1 : -2;
  const int splits = i8 ? mfb_paged_decode_int8_splits(B, Hkv, max_blocks * block_size) : mfb_paged_decode_tc_splits(B, Hkv, max_blocks * block_size);
  const long long need = mfb_paged_decode_scratch_bytes(B, Hq, hd, splits);
  if (scratch_bytes < need) return need;
  int rc = i8 ? mfb_reshape_and_cache_int8(k, v, key_cache, value_cache, key_scale, value_scale, slots, B, Hkv, hd, k0, v0, stream)
              : mfb_reshape_and_cache(k, v, key_cache, value_cache, slots, B, Hkv * hd, k0, v0, stream);
  if (rc) return -100 - rc;
  rc = i8 ? mfb_paged_decode_attention_int8(q, q0, q1, key_cache, value_cache, key_scale, value_scale, tables, lens, out, scratch, splits,
                                            B, Hq, Hkv, hd, block_size, max_blocks, scale, stream)
          : mfb_paged_decode_attention_tc_q(q, q0, q1, key_cache, value_cache, tables, lens, nullptr, nullptr, out, scratch, splits, B, B,
                                            Hq, Hkv, hd, hd, num_blocks, block_size, max_blocks, 0, 0, 0, scale, 0.f, (long long)Hq * hd,
                                            1.f, status, stream);
  return rc ? -200 - rc : 0;
}

int mfb_event_record(cudaEvent_t event, cudaStream_t stream) {
  const cudaError_t rc = cudaEventRecord(event, stream);
  if (rc != cudaSuccess) { mfb_host::set_error("event_record: %s", cudaGetErrorString(rc)); return 2; }
  return 0;
}

// Whether all work in front of an event is done (0; 1: not yet), after waiting for it if wait != 0; other values: an error. The event stands
// outside of whatever this thread is capturing, so the call is harmless to a capture, which forbids it by default.
int mfb_event_done(cudaEvent_t event, int wait) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) { mfb_host::set_error("event_done: capture mode"); return 2; }
  const cudaError_t rc = wait ? cudaEventSynchronize(event) : cudaEventQuery(event);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (rc == cudaSuccess) return 0;
  cudaGetLastError();              // "not ready" would otherwise look like a failed launch
  if (rc == cudaErrorNotReady) return 1;
  mfb_host::set_error("event_done: %s", cudaGetErrorString(rc));
  return 3;
}

}  // extern "C"
