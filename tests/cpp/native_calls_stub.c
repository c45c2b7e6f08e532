/* Stand-ins for the library under native_calls.c: each returns whether the
 * interpreter's lock was held while it ran. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "fbgemm_b200/embedding_c_api.h"

int fbgemm_b200_spmdm_launch(fbgemm_b200_ctx* ctx, const fbgemm_b200_spmdm_config* cfg, int64_t output_size,
                             int64_t index_size, int64_t data_size, const void* input, const void* indices,
                             const void* offsets_or_lengths, const float* weights, void* out,
                             const int32_t* compressed_indices_table, int slot, void* stream) {
  (void)ctx, (void)cfg, (void)output_size, (void)index_size, (void)data_size, (void)input, (void)indices;
  (void)offsets_or_lengths, (void)weights, (void)out, (void)compressed_indices_table, (void)slot, (void)stream;
  return PyGILState_Check();
}

int fbgemm_b200_spmdm(fbgemm_b200_ctx* ctx, const fbgemm_b200_spmdm_config* cfg, int64_t output_size, int64_t index_size,
                      int64_t data_size, const void* input, const void* indices, const void* offsets_or_lengths,
                      const float* weights, void* out, const int32_t* compressed_indices_table, void* stream) {
  return fbgemm_b200_spmdm_launch(ctx, cfg, output_size, index_size, data_size, input, indices, offsets_or_lengths, weights,
                                  out, compressed_indices_table, 0, stream);
}

int fbgemm_b200_table_set_forward(fbgemm_b200_table_set* set, int64_t bags, const void* indices, int64_t index_size,
                                  const void* offsets, const float* weights, void* out, int slot, void* stream) {
  (void)set, (void)bags, (void)indices, (void)index_size, (void)offsets, (void)weights, (void)out, (void)slot, (void)stream;
  return PyGILState_Check();
}

int fbgemm_b200_float_to_fused_8bit_rowwise(const float* input, int64_t rows, int32_t cols, uint8_t* output, void* stream) {
  (void)input, (void)rows, (void)cols, (void)output, (void)stream;
  return PyGILState_Check();
}

int fbgemm_b200_float_to_fused_nbit_rowwise(int32_t bit_rate, const float* input, int64_t rows, int32_t cols, uint8_t* output,
                                            void* stream) {
  (void)bit_rate;
  return fbgemm_b200_float_to_fused_8bit_rowwise(input, rows, cols, output, stream);
}

int fbgemm_b200_pruned_hashmap_lookup(fbgemm_b200_ctx* ctx, int32_t T, int32_t B, const void* indices, const void* offsets,
                                      int32_t index_bytes, int64_t index_size, const void* hash_table, int32_t hash_bytes,
                                      const int64_t* hash_table_offsets, void* dense_indices, int32_t slot, void* stream) {
  (void)ctx, (void)T, (void)B, (void)indices, (void)offsets, (void)index_bytes, (void)index_size, (void)hash_table;
  (void)hash_bytes, (void)hash_table_offsets, (void)dense_indices, (void)slot, (void)stream;
  return PyGILState_Check();
}

int fbgemm_b200_pruned_array_lookup(fbgemm_b200_ctx* ctx, int32_t T, int32_t B, const void* indices, const void* offsets,
                                    int32_t index_bytes, int64_t index_size, const void* index_remappings,
                                    int32_t remapping_bytes, const int64_t* index_remappings_offsets, void* dense_indices,
                                    int32_t slot, void* stream) {
  return fbgemm_b200_pruned_hashmap_lookup(ctx, T, B, indices, offsets, index_bytes, index_size, index_remappings,
                                           remapping_bytes, index_remappings_offsets, dense_indices, slot, stream);
}

int fbgemm_b200_sequence_lookup(fbgemm_b200_ctx* ctx, const void* dev_weights, const fbgemm_b200_sequence_table* tables,
                                int32_t T, int32_t B, int32_t D, const void* indices, const void* offsets,
                                int32_t index_bytes, int64_t index_size, void* out, int32_t out_dtype, int64_t out_row_bytes,
                                int32_t scale_bias_last, int32_t fp8_exponent_bits, int32_t fp8_exponent_bias, int32_t slot,
                                void* stream) {
  (void)ctx, (void)dev_weights, (void)tables, (void)T, (void)B, (void)D, (void)indices, (void)offsets, (void)index_bytes;
  (void)index_size, (void)out, (void)out_dtype, (void)out_row_bytes, (void)scale_bias_last, (void)fp8_exponent_bits;
  (void)fp8_exponent_bias, (void)slot, (void)stream;
  return PyGILState_Check();
}

int fbgemm_b200_sequence_lookup_filled(fbgemm_b200_ctx* ctx, const void* dev_weights, const fbgemm_b200_sequence_table* tables,
                                       int32_t T, int32_t B, int32_t D, const void* indices, const void* offsets,
                                       int32_t index_bytes, int64_t index_size, void* out, int32_t out_dtype,
                                       int64_t out_row_bytes, int32_t scale_bias_last, int32_t fp8_exponent_bits,
                                       int32_t fp8_exponent_bias, int32_t slot, void* stream) {
  return fbgemm_b200_sequence_lookup(ctx, dev_weights, tables, T, B, D, indices, offsets, index_bytes, index_size, out,
                                     out_dtype, out_row_bytes, scale_bias_last, fp8_exponent_bits, fp8_exponent_bias, slot,
                                     stream);
}
