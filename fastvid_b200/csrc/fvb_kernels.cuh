// fvb_kernels.cuh -- launch shapes and kernel declarations shared by the
// kernel files and the host orchestration (fvb_api.cu).
#pragma once

#include <type_traits>

#include "fvb_common.cuh"

namespace fvb {

constexpr int kWarpsPerCta = 4;    // warps per CTA of the warp-per-item kernels
constexpr int kSrcStride = 66;     // u16 ring row stride: 64 columns + 2 (33 words: conflict-free)
constexpr int kFoldStride = 65;    // u32 ring row stride: 64 columns + 1 (conflict-free)
constexpr int kFastMaxW = 512;     // widest tile of the register-wavefront path
constexpr int kDefaultWavefrontBlock = 8;  // steps of a 32-step wavefront block unrolled (4, 8, 16, 32)
constexpr int kDefaultTileWarps = 1;       // warps per tile of the wavefront kernels (1 or 2)

// Whether a warp pair splits a tile's bands (the predictor and the
// reconstruction alike): at least two bands, and at least four wavefront
// blocks per band -- the second warp runs two blocks behind the first, and
// the band below needs the band above's last row up to one block ahead of
// it, which the schedule provides once a band has four blocks.
__host__ __device__ inline bool pair_splits(int w, int h) { return ((h + 31) >> 5) >= 2 && ((w + 62) >> 5) >= 4; }

// ---------------------------------------------------------------------------
// The folded-symbol intermediate (predictor residuals, zigzag-folded, in
// tile-raster order) is held as u32, or as u16 when every frame of a batch
// has a bit depth below 16 or a quality below 100 (fold16).  Then the
// encoder's symbols are below 2^16: at depth <= 15 |q| <= 2^15 - 1, and a
// 16-bit frame below quality 100 has a step of at least 12.  The decoder
// accepts symbols up to 2 * max_sample (decode.cu bounds), which at depth 16
// can exceed 16 bits in a valid stream; such a symbol is stored as 65534 or
// 65535 by parity (fold_value), i.e. a residual of +32767 or -32768 steps,
// which clamps to the same sample as the original since the step is >= 12.
template <typename T>
using FoldPiece = std::conditional_t<sizeof(T) == 2, uint2, uint4>;  // four symbols

template <typename T>
__device__ __forceinline__ uint32_t ldf(const T* p) {
  return static_cast<uint32_t>(__ldg(p));
}
//
// The decoder's u16 intermediate of a frame of depth 12 or less holds, in
// place of the symbol, what the reconstruction adds to the prediction: the
// unfolded residual times the step, as a signed 16-bit value.  The residual
// is first clamped to +-ceil(max_sample / step), beyond which the sample
// saturates whatever the prediction is, so the product stays below
// 2 * max_sample.  The rANS decoder does this once per table entry.
struct FoldMap {
  int32_t step, lim;  // lim 0: symbols are stored as they are
};
__device__ __forceinline__ FoldMap fold_map(const FrameDesc& f, bool fold16) {
  if (!fold16 || f.bit_depth > 12) return FoldMap{1, 0};
  return FoldMap{f.step0, (f.max_sample + f.step0 - 1) / f.step0};
}
template <typename T>
__device__ __forceinline__ T fold_value(uint32_t v, const FoldMap& m) {
  if constexpr (sizeof(T) == 2) {
    if (m.lim) return static_cast<T>(max(-m.lim, min(m.lim, unzigzag(v))) * m.step);
    return static_cast<T>(min(v, 65534u | (v & 1u)));
  } else {
    return v;
  }
}
// The residuals times the step of a decoded frame's samples, for the kernels
// that reconstruct sample by sample and read neighbours back from the planes.
// What they depend on is held here, and they are read by plain loads: read-only
// loads made the same kernels slower by a third to twice (a 1080p yuv422 10-bit
// frame as one tile 7.2 and 5.6 ms; 7.9 with the descriptor read per sample).
struct Deltas {
  const void* folded;
  int32_t step;
  bool u16, products;
  __device__ Deltas(const FrameDesc& f, const void* folded_, int fold16)
      : folded(folded_), step(f.step0), u16(fold16 != 0), products(fold16 && f.bit_depth <= 12) {}
  __device__ __forceinline__ int32_t operator[](int64_t i) const {
    if (!u16) return unzigzag(static_cast<const uint32_t*>(folded)[i]) * step;
    const uint16_t v = static_cast<const uint16_t*>(folded)[i];
    return products ? static_cast<int16_t>(v) : unzigzag(v) * step;
  }
};
__device__ __forceinline__ void unpack_piece(const uint4& p, uint32_t (&x)[4]) {
  x[0] = p.x;
  x[1] = p.y;
  x[2] = p.z;
  x[3] = p.w;
}
__device__ __forceinline__ void unpack_piece(const uint2& p, uint32_t (&x)[4]) {
  x[0] = p.x & 0xffffu;
  x[1] = p.x >> 16;
  x[2] = p.y & 0xffffu;
  x[3] = p.y >> 16;
}
__device__ __forceinline__ void cp_async_piece(uint4* smem, const uint4* gmem) { cp_async16(smem, gmem); }
__device__ __forceinline__ void cp_async_piece(uint2* smem, const uint2* gmem) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// encoder (counts of pass `pass` from dims); `folded` is u16 when fold16
__global__ void enc_init_kernel(const FrameDesc* frames, FrameState* state, const BatchDims* dims);
// frames of step 1 (pass 0 only)
void enc_lossless_launch(bool fold16, int64_t tiles, int max_ctas, cudaStream_t stream, const FrameDesc* frames,
                         FrameState* state, const BatchDims* dims, ShardInfo* shards, void* folded);
// the other frames; u16 symbols: by warp pairs or single warps; u32 symbols: a wavefront block of `unroll` steps (4, 8, 16,
// 32) and `tile_warps` (1, or 2: a warp pair splits each tile's bands)
void enc_predict_launch(int unroll, int tile_warps, bool fold16, bool pairs, int grid, cudaStream_t stream,
                        const FrameDesc* frames, FrameState* state, const BatchDims* dims, int pass,
                        ShardInfo* shards, void* folded, int* queue);
cudaError_t enc_predict_set_smem();
__global__ void enc_predict_wide_kernel(const FrameDesc* frames, FrameState* state, const BatchDims* dims, int pass,
                                        void* folded, uint16_t* recon, int fold16);
void enc_analyze_launch(bool fold16, int grid, cudaStream_t stream, const FrameDesc* frames, FrameState* state,
                        const BatchDims* dims, int pass, ShardInfo* shards, const void* folded,
                        uint8_t* rans_scratch);
void enc_rans_launch(bool fold16, int64_t nshards, cudaStream_t stream, const FrameDesc* frames,
                     const FrameState* state, const BatchDims* dims, int pass, ShardInfo* shards, int32_t* sizes,
                     const void* folded, uint8_t* rans_scratch);
__global__ void enc_scan_kernel(const FrameDesc* frames, FrameState* state, const BatchDims* dims, int pass,
                                ShardInfo* shards, const int32_t* sizes, uint8_t* prefix, int64_t* results);
// Records of one encoder region: pass 0's, or the later pass's (region b,
// indexed like pass 0's for the frames that took part in it).
struct EmitRegion {
  const ShardInfo* shards;
  const void* folded;
  const uint8_t* rans_scratch;
  int64_t count;  // shards 0 .. count-1 have records in this region
};
// The frames' headers and directories, copied by `ctas` CTAs a frame.
struct EmitHeads {
  const FrameDesc* descs;
  const uint8_t* prefix;
  const uint8_t* prefix_b;
  int frames, ctas;
};
// `only_out`: the output of a batch of one frame (null: the table `outs`)
void enc_emit_launch(bool fold16, int grid, size_t smem, cudaStream_t stream, const FrameState* state, EmitRegion a,
                     EmitRegion b, int64_t total_shards, EmitHeads heads, uint8_t* const* outs, uint8_t* only_out);
cudaError_t enc_emit_set_smem(int bytes);
// decoder: shards binned by mode (0 rANS, 1 Rice, 2 zero-run, 3 block pack, 4
// Rice shards of up to kRiceSmall symbols); counts from dims (entry 0).  A list's
// items lie one after another from list * (shards of the batch) on, the small
// Rice shards' downwards from the end of list 1's room.
struct DecodeLists {
  int32_t count[5];
  int32_t next_group;       // dec_other work counter
  int32_t next_group_rans;  // dec_rans work counter
  int32_t pad;
};
struct RansTable;
__global__ void dec_parse_kernel(const FrameDesc* frames, FrameState* state, const BatchDims* dims,
                                 ShardInfo* shards, DecodeLists* lists, int32_t* list_items);
__global__ void dec_rans_tables_kernel(const FrameDesc* frames, FrameState* state, const ShardInfo* shards,
                                       const DecodeLists* lists, const int32_t* list_items, RansTable* tables,
                                       int fold16);
// `few` shards: one warp for two shards, tables of all slots; `roomy`: entries
// and values of up to 170 symbols in shared memory
void dec_rans_launch(bool fold16, bool few, bool roomy, int grid, cudaStream_t stream, const FrameDesc* frames,
                     FrameState* state, const ShardInfo* shards, DecodeLists* lists, const int32_t* list_items,
                     const RansTable* tables, void* folded);
cudaError_t dec_rans_set_smem();
void dec_other_launch(bool fold16, int grid, cudaStream_t stream, const FrameDesc* frames, FrameState* state,
                      const ShardInfo* shards, const BatchDims* dims, DecodeLists* lists, const int32_t* list_items,
                      void* folded);
// u32 symbols: `unroll` and `tile_warps` as for enc_predict
// (every reconstruction kernel also writes the frames' statuses to `results`)
void dec_reconstruct_launch(int unroll, int tile_warps, bool fold16, bool pairs, int grid, cudaStream_t stream,
                            const FrameDesc* frames, const FrameState* state, const BatchDims* dims,
                            const void* folded, int* queue, int64_t* results);
cudaError_t dec_other_set_smem();
cudaError_t dec_reconstruct_set_smem();
__global__ void dec_reconstruct_wide_kernel(const FrameDesc* frames, const FrameState* state, const BatchDims* dims,
                                            const void* folded, int fold16);
__global__ void dec_reconstruct_serial_kernel(const FrameDesc* frames, const FrameState* state,
                                              const BatchDims* dims, const void* folded, int fold16,
                                              int64_t* results);

size_t enc_predict_smem(bool fold16);
size_t enc_emit_smem();
size_t dec_reconstruct_smem(bool fold16);
size_t dec_rans_table_bytes();

}  // namespace fvb
