// The cached rows of a latent attention as plain rows: of every sequence the positions that the step's tokens see, latents and rotated
// tails apart, for a product that expands them into keys and values.  A copy: 16 bytes a thread, bound by memory.
#include "common.cuh"

MB_DEFINE_LAST_ERROR()

namespace mb {

// grid (ceil(rows_per * pieces / 256), sequences); block 256.  Piece p of a row: 16 bytes of [latent | tail | zeros up to padded].
// A sequence's first row is the position 0, or with a window the multiple of 64 at or before the first position that the step's first
// token sees: what lies before it may be gone from the cache.  Rows behind the sequence's end are left as they are, but for those up to
// the next multiple of 64, which become zeros.
__global__ void __launch_bounds__(256)
latent_gather_kernel(const uint4* __restrict__ pool, int row_pieces, int latent_pieces, int padded_pieces, const int* __restrict__ block_table,
                     int max_blocks, int page_size, const int* __restrict__ cu_q, const int* __restrict__ kv_lens, int window, int rows_per,
                     uint4* __restrict__ latents, uint4* __restrict__ tails) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int seq = blockIdx.y, pieces = latent_pieces + padded_pieces;
    const int i = blockIdx.x * 256 + threadIdx.x, row = i / pieces, piece = i % pieces;
    const int length = kv_lens[seq], seen = window > 0 ? length - (cu_q[seq + 1] - cu_q[seq]) - window + 1 : 0;
    const int position = (seen > 0 ? seen / 64 * 64 : 0) + row;
    if (row >= rows_per || position >= (length + 63) / 64 * 64) return;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (position < length && piece < row_pieces) {
        const size_t page = block_table[(size_t)seq * max_blocks + position / page_size];
        v = pool[(page * page_size + position % page_size) * row_pieces + piece];
    }
    const size_t to = (size_t)seq * rows_per + row;
    if (piece < latent_pieces) latents[to * latent_pieces + piece] = v;
    else tails[to * padded_pieces + piece - latent_pieces] = v;
}

}  // namespace mb

using namespace mb;

// pool: bfloat16 [pages][page_size][latent + turned]; latents [sequences * rows_per][latent], tails [sequences * rows_per][padded] (null
// without a tail).  Sizes in numbers, multiples of 8; rows_per a multiple of 64 that holds what any sequence's step sees (window 0: all
// of the longest sequence; n: n - 1 positions, the step's tokens and what the multiple of 64 adds).
MB_EXPORT int mb_latent_gather(const void* pool, int latent, int turned, int padded, const int* block_table, int max_blocks, int page_size,
                               const int* cu_q, const int* kv_lens, int sequences, int window, int rows_per, void* latents, void* tails,
                               cudaStream_t stream) {
    if (sequences <= 0 || rows_per <= 0) return 0;
    if (latent <= 0 || latent % 8 || turned % 8 || padded % 8 || padded < turned || (turned > 0 && !tails) || ((uintptr_t)pool & 15) ||
        ((uintptr_t)latents & 15) || ((uintptr_t)tails & 15) || rows_per % 64 || window < 0 || (window > 0 && !cu_q) || sequences > 65535 || (long long)max_blocks * page_size < rows_per)
        return fail("latent_gather: rows of %d and %d numbers (%d with zeros), %d of each of %d sequences", latent, turned, padded, rows_per, sequences);
    const int pieces = (latent + (turned > 0 ? padded : 0)) / 8;
    const long long blocks = ((long long)rows_per * pieces + 255) / 256;
    if (blocks > 0x7fffffff) return fail("latent_gather: %d rows exceed the grid", rows_per);
    MB_LAUNCH("latent_gather", latent_gather_kernel, dim3((unsigned)blocks, sequences), dim3(256), 0, stream, true, (const uint4*)pool,
              (latent + turned) / 8, latent / 8, turned > 0 ? padded / 8 : 0, block_table, max_blocks, page_size, cu_q, kv_lens, window, rows_per, (uint4*)latents,
              (uint4*)tails);
    return check_launch("latent_gather");
}
