// Cached latents of a step's prompt portions, taken out of their pages into rows of their own.
//
// Row 128 j + i of `out` is the cached vector at position where[3 j + 1] + i of entry where[3 j]; zero
// before position where[3 j + 2] (pages a window has passed), from the entry's end on, and where a page is
// missing (which sets a status bit).  The product that
// expands keys and values for all heads reads these rows (parts/latent_attention.py); upstream has no
// such cache.
#include "attention_common.cuh"

#define LATENT_BLOCK 128

__global__ void __launch_bounds__(256) latent_rows_kernel(const uint4* __restrict__ cache, int pieces, const int* __restrict__ block_table,
                                                          int max_pages, int page_size, int num_pages, const int* __restrict__ where,
                                                          const int* __restrict__ ctx_lens, uint4* __restrict__ out, int* status) {
  pdl_trigger();
  pdl_wait();
  const int entry = where[3 * blockIdx.x], first = where[3 * blockIdx.x + 1], begin = where[3 * blockIdx.x + 2], end = ctx_lens[entry];
  const int* table = block_table + (size_t)entry * max_pages;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = blockIdx.y * 8 + warp; i < LATENT_BLOCK; i += 8 * gridDim.y) {
    const int pos = first + i, logical = pos / page_size;
    int page = -1;
    if (pos >= begin && pos < end) {
      page = logical < max_pages ? table[logical] : -1;
      if (page < 0 || page >= num_pages) {
        if (lane == 0) atomicOr(status, FE_STATUS_BAD_PAGE);
        page = -1;
      }
    }
    const uint4* src = cache + ((size_t)max(page, 0) * page_size + (pos - logical * page_size)) * pieces;
    uint4* dst = out + ((size_t)blockIdx.x * LATENT_BLOCK + i) * pieces;
    for (int c = lane; c < pieces; c += 32) dst[c] = page >= 0 ? src[c] : make_uint4(0u, 0u, 0u, 0u);
  }
}

// `width` bfloat16 numbers per cached vector (a multiple of 8); `blocks` stretches of 128 rows.
FE_EXPORT int fe_latent_rows(const void* cache, int width, const int* block_table, int max_pages, int page_size, int num_pages,
                             const int* where, int blocks, const int* ctx_lens, void* out, int* status, cudaStream_t stream) {
  if (blocks <= 0) return 0;
  if (width < 8 || width % 8) return FE_ERR_BAD_SHAPE;
  if (((uintptr_t)cache | (uintptr_t)out) & 15) return FE_ERR_BAD_ALIGN;
  return fe_launch_dependent(latent_rows_kernel, dim3(blocks, 4), dim3(256), 0, stream, (const uint4*)cache, width / 8, block_table,
                             max_pages, page_size, num_pages, where, ctx_lens, (uint4*)out, status);
}
