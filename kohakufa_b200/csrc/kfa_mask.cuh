// Boolean attention masks, packed for the kernels: 32 keys per 32-bit word along each query row
// (`words`, read by the forward and the dQ kernel, whose threads own query rows) and 32 queries per word
// along each key row (`words_t`, read by the dK / dV kernel, whose threads own key rows). Bit c % 32 of
// word c / 32 is key (query) c; rows are padded with zero bits to whole 128-wide tiles, so a tile's four
// words never run past a row and padded keys / queries are hidden without a length check.
// Same word format as the reference's packing (src/kohakufa/mask.py:32-72). Instead of the reference's
// per-tile any / all classes and host-built tile lists (mask.py:74-122) the packing marks, in one int per
// (128 queries x 128 keys) tile, whether the tile holds any visible pair; every CTA builds the list of
// tiles it visits from that table in shared memory, and a warp whose bits are all set skips the masking
// code.
// Included at the end of kfa_api.cu (uses its helpers).
#pragma once

namespace kfa {

// One CTA packs a 128 x 128 tile, one warp each of its 32 x 32 blocks (warp = 4 * row block + column block): a lane
// reads one key's column of 32 queries (32 independent loads; neighbouring lanes neighbouring keys), which IS that
// key's transposed word; 32 ballots give the rows' words. Rows and columns past the ends read as hidden, so the
// padding words come out zero, and the tile's flag is one vote of the CTA: no zero fills, no atomics. (Row after row
// with a ballot and a store each, every load waited for: with the fills 15.2 -> 9.0 us at 2048 x 2048, 42.6 -> 25.2 at
// 4096 x 4096, 11.3 -> 5.3 at 128 x 128, allocations in a graph included. Bound by the 4-byte stores of the words.)
// Grid: (key tiles, query tiles, slices).
__global__ void __launch_bounds__(512) kfa_pack_mask_kernel(const uint8_t* __restrict__ mask, long long m_sb, long long m_sh,
                                                            long long m_sr, long long m_sc, int Hm, int Sq, int Skv,
                                                            int* __restrict__ words, int wq /*ints per row of words*/,
                                                            int* __restrict__ words_t, int wk /*ints per row of words_t*/,
                                                            int* __restrict__ tiles) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cb = blockIdx.x * 4 + (warp & 3);   // 32-key block
  const int rb = blockIdx.y * 4 + (warp >> 2);  // 32-query block
  const long long slice = blockIdx.z;
  const int b = blockIdx.z / Hm, h = blockIdx.z % Hm;
  const int col = cb * 32 + lane;
  const int rows = min(Sq - rb * 32, 32);  // of this block (may be <= 0)
  const uint8_t* src = mask + b * m_sb + h * m_sh + static_cast<long long>(rb) * 32 * m_sr + col * m_sc;
  uint32_t mine = 0;  // bit r: query rb * 32 + r sees key `col`
  if (col < Skv) {
#pragma unroll
    for (int r = 0; r < 32; ++r)
      if (r < rows && src[r * m_sr] != 0) mine |= 1u << r;
  }
  uint32_t row_word = 0;  // lane r: the word of query row rb * 32 + r
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const uint32_t w = __ballot_sync(0xffffffffu, (mine >> r) & 1u);
    if (lane == r) row_word = w;
  }
  if (lane < rows) words[(slice * Sq + rb * 32 + lane) * wq + cb] = static_cast<int>(row_word);
  if (col < Skv) words_t[(slice * Skv + col) * wk + rb] = static_cast<int>(mine);
  const int some = __syncthreads_or(mine != 0);
  if (tiles != nullptr && threadIdx.x == 0)
    tiles[(slice * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = some ? 1 : 0;
}

}  // namespace kfa

extern "C" int kfa_pack_mask(const void* mask, const int64_t* mask_stride, int mask_batch, int mask_heads, int Sq,
                             int Skv, int32_t* words, int32_t* words_t, int32_t* tiles, void* stream) {
  if (!mask || !mask_stride || !words || !words_t) return fail(KFA_ERR_ARG, "kfa_pack_mask: null pointer");
  if (mask_batch < 1 || mask_heads < 1 || Sq < 1 || Skv < 1) return fail(KFA_ERR_ARG, "kfa_pack_mask: empty mask");
  const int wq = 4 * ((Skv + 127) / 128), wk = 4 * ((Sq + 127) / 128);
  const int slices = mask_batch * mask_heads;
  if (slices > 65535 || (Sq + 31) / 32 > 65535) return fail(KFA_ERR_ARG, "kfa_pack_mask: mask too large for one launch");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  dim3 grid(wq / 4, wk / 4, slices);
  kfa::kfa_pack_mask_kernel<<<grid, 512, 0, s>>>(static_cast<const uint8_t*>(mask), mask_stride[0], mask_stride[1],
                                                 mask_stride[2], mask_stride[3], mask_heads, Sq, Skv, words, wq,
                                                 words_t, wk, tiles);
  KFA_CUDA(cudaGetLastError());
  return KFA_OK;
}
