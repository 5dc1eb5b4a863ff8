// fvb_wave.cuh -- the wavefront of the predictor and of the reconstruction:
// two rows per lane, packed 16-bit arithmetic, bands of 64 rows.
//
// A warp sweeps a tile in bands of 64 rows, lane r holding rows 2r and 2r+1
// of the band; row k handles column t - skew(k) at step t.  For bit depths
// up to 12 the two rows' values share one register, and the predictor and
// the reconstruction run on packed signed 16-bit halves (vmin/vmax/vsub and
// the fused add-min-max of the DPX set, one instruction each on sm_100); a
// row's upper neighbour is the other half of the lane's own previous step
// (odd rows) or of the lane below in rank (even rows: one shuffle).
//
// Samples go through shared-memory windows of five 16-byte chunks per row,
// updated in place: block b of 32 steps consumes 32 columns of every row --
// positions off .. off + 31 of the row's window, where `off` in 0..7 keeps
// the window chunks on 16-byte boundaries of global memory although the rows
// are skewed by single samples.  Chunks 1..4 of the next window are fetched
// by cp.async while a block runs (chunk 0 is the straddling chunk 4 of the
// window before, copied by the row's own lane), and a finished window's
// chunks 0..3 leave with 16-byte stores.  Columns left of the tile are zero
// filled, which makes every value there zero by itself (prediction 0,
// residual 0), so no step has an edge case; columns right of the tile hold
// values that nothing inside the tile reads.
#pragma once

#include "fvb_common.cuh"
#include "fvb_kernels.cuh"

namespace fvb {

constexpr int kBandRows = 64;
constexpr int kWinChunks = 5;
// Row k's window starts at chunk 5k + k / 8.  One instruction reads a word of
// the 32 even (or odd) rows; with a skew of 2 a lane, lanes four apart read
// the same word of their 16-byte chunks, and those chunks, 41 apart, differ
// modulo 8: no bank is hit twice.
constexpr int kWinVecs = kWinChunks * kBandRows + kBandRows / 8;
constexpr int kCarryPad = 128;  // columns kept left of the tile: above the largest skew
constexpr int kCarryCols = kCarryPad + kFastMaxW + 160;

struct alignas(16) WaveSm {
  uint4 win[2][kWinVecs];
  uint16_t carry[kCarryCols];  // row above the band, column c at index c + kCarryPad
};

// Row k runs one step behind the row above it: the shortest sweep (W + 63 steps
// a band), with the shuffle on the chain from step to step.  (Four steps a lane
// instead of two take the shuffle off the chain for 62 steps more a band: 2 us
// less of 35 for the reconstruction of a 1080p frame, 2 to 4 us more for its
// prediction, 6 to 20 % more for batches.)
constexpr int kSkew = 2;  // per lane, two rows
__host__ __device__ constexpr int wave_skew(int row) { return row; }
constexpr int kWinHop = 8 * kWinChunks + 1;  // chunks from row k to row k + 8
__device__ __forceinline__ int win_row(int row) { return kWinChunks * row + (row >> 3); }

// 16 bytes, or zeros where the source is to be ignored (it is not read then)
__device__ __forceinline__ void cp_async16_or_zero(void* smem, const void* gmem, bool ignore) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int z = ignore;
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %2, 0;\n cp.async.cg.shared.global [%0], [%1], 16, p;\n}\n" ::"r"(s),
      "l"(gmem), "r"(z)
      : "memory");
}

// Bits lo .. hi (none when hi < lo; bits 0..31)
__device__ __forceinline__ uint32_t bit_range(int lo, int hi) {
  return (hi < 0 ? 0u : 0xffffffffu >> (31 - min(hi, 31))) & (lo > 31 ? 0u : 0xffffffffu << max(lo, 0));
}

// a - b of packed halves in 0..32767, as signed halves: the low half cannot
// borrow from the high one once its top bit is set.  (The packed subtraction is
// a negation and an addition.)
__device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) { return (a + 0x8000u - b) ^ 0x8000u; }

__device__ __forceinline__ uint32_t pair2(int32_t v) { return static_cast<uint32_t>(v & 0xffff) * 0x10001u; }

// Loads and stores of one warp's windows over the bands of a tile.  Chunks of
// global memory are copied as they lie, so a row's first chunk may hold up to
// seven samples left of the tile, cleared by fix_edge().  CHECK: a chunk may
// reach outside [lo, hi), the memory that may be read.
// ROWS: how rows that are not aligned alike are stored (see store_whole).
template <bool CHECK, bool ROWS>
struct WaveIo {
  static constexpr int kShift = 3;  // rows eight apart: columns 1 << kShift apart
  static_assert(4 * kSkew == 1 << kShift, "skew of eight rows");
  WaveSm& sm;
  const int lane;
  const int W;
  const uint16_t* __restrict__ in;  // row 0 of the band, column 0
  const int64_t in_pitch;
  uint16_t* __restrict__ out;
  const int64_t out_pitch;
  const uint16_t* lo;
  const uint16_t* hi;
  bool at_edge;  // the band touches the plane's first or last chunk
  int nrows, nblk, row_top;  // row_top: the last i with row lr + 8 i in the band
  int a_in, a_step;  // alignment (samples modulo 8) of row 0, and its change per row
  int store_mode;    // 0: single samples, 1: pairs, 2: 16-byte chunks
  bool ragged;       // rows have partial chunks
  // chunk role: chunk lj of rows lr, lr + 8, ...; c_first: the column of chunk
  // lj of row lr in window 0
  int lr, lj, c_first;
  int64_t in_hop, out_hop;  // from row lr + 8 i to the next, one window column
  // own rows 2 lane, 2 lane + 1
  int off0, off1;

  // a row start on an odd sample delays the whole sweep by a step, so that the
  // even rows' window positions are even
  __device__ int skew(int row) const { return wave_skew(row) + (a_in & 1); }
  __device__ int align_of(int row) const { return (a_in + row * a_step) & 7; }
  __device__ int off_of(int row) const { return (align_of(row) - skew(row)) & 7; }

  __device__ WaveIo(WaveSm& sm_, int lane_, int W_, const uint16_t* in_, int64_t in_pitch_, uint16_t* out_,
                    int64_t out_pitch_, const uint16_t* lo_, const uint16_t* hi_)
      : sm(sm_), lane(lane_), W(W_), in(in_), in_pitch(in_pitch_), out(out_), out_pitch(out_pitch_), lo(lo_),
        hi(hi_) {
    a_in = static_cast<int>(reinterpret_cast<uintptr_t>(in) >> 1) & 7;
    a_step = static_cast<int>(in_pitch & 7);
    const int d_in = static_cast<int>(reinterpret_cast<uintptr_t>(out) >> 1) & 7;
    const int d_step = static_cast<int>(out_pitch & 7);
    // whole chunks may be stored when input and output rows are aligned alike
    if (d_in == a_in && d_step == a_step) store_mode = 2;
    else store_mode = ((d_in | d_step | a_in | a_step | W) & 1) ? 0 : 1;
    ragged = ((a_in | a_step | W) & 7) != 0;
    lr = lane >> 2;
    lj = lane & 3;
    c_first = -skew(lr) - off_of(lr) + 8 * lj;
    in_hop = 8 * in_pitch - 4 * kSkew;
    out_hop = 8 * out_pitch - 4 * kSkew;
    off0 = off_of(2 * lane);
    off1 = off_of(2 * lane + 1);
  }
  __device__ void band(int rows_left) {
    nrows = min(kBandRows, rows_left);
    at_edge = CHECK && (in - 7 < lo || in + (nrows - 1) * in_pitch + W + 7 > hi);
    row_top = ((nrows - lr + 7) >> 3) - 1;
    nblk = (W + skew(nrows - 1) + 31) >> 5;
  }
  __device__ void next_band() {
    in += kBandRows * in_pitch;
    out += kBandRows * out_pitch;
  }

  __device__ void fetch_chunk(uint4* dst, const uint16_t* src, int c, bool valid) {
    if (CHECK && at_edge) {
      if (valid && (src < lo || src + 8 > hi)) {  // the plane's first or last chunk
        uint16_t* d = reinterpret_cast<uint16_t*>(dst);
#pragma unroll 1
        for (int e = 0; e < 8; ++e) d[e] = (c + e >= 0 && c + e < W) ? src[e] : 0;
        return;
      }
    }
    cp_async16_or_zero(dst, src, !valid);
  }
  // Starts the fetch of window b (chunks 1..4 of every row; chunk 0 too for
  // the first window of a band).
  __device__ void fetch(int b) {
    uint4* w = sm.win[b & 1];
    const int c = c_first + 32 * b + 8;
    const uint16_t* src = in + lr * in_pitch + c;
    uint4* dst = w + kWinChunks * lr + 1 + lj;
    // rows whose chunk, at column c - (i << kShift), holds a column of the tile
    const uint32_t valid = bit_range((c - W + (1 << kShift)) >> kShift, min((c + 7) >> kShift, row_top));
    if (CHECK && at_edge) {
#pragma unroll 1
      for (int i = 0; i < 8; ++i)
        fetch_chunk(dst + kWinHop * i, src + i * in_hop, c - (i << kShift), valid & (1u << i));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        cp_async16_or_zero(dst + kWinHop * i, src, !(valid & (1u << i)));
        src += in_hop;
      }
    }
    if (b == 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = 2 * lane + h;
        const int c0 = -skew(row) - (h ? off1 : off0);
        fetch_chunk(w + win_row(row), in + row * in_pitch + c0, c0, row < nrows && c0 > -8);
      }
    }
    cp_async_commit();
  }
  // Window b is complete after this (the fetch of window b + 1, or an empty
  // group in its place, was committed).
  __device__ void wait() {
    cp_async_wait<1>();
    __syncwarp();
  }
  // Clears the samples left of the tile in the chunk that holds column 0, and
  // (TAIL) those right of it in the last, where row starts are unaligned.
  template <bool TAIL>
  __device__ void fix_edge(int b) {
    if (((a_in | a_step) & 7) == 0 && !(TAIL && (W & 7))) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = 2 * lane + h;
      const int a = align_of(row), sk = skew(row), off = h ? off1 : off0;
      const int base = 32 * b - sk - off;  // column of the window's first position
      uint16_t* w = reinterpret_cast<uint16_t*>(sm.win[b & 1] + win_row(row));
      // chunk 0 was cleared as chunk 4 of the window before, except in the first
      const int k0 = b ? 1 : 0;
      const int zk = (-a - base) >> 3;  // chunk that starts at column -a
      if (a && zk >= k0 && zk < kWinChunks)
        for (int e = 0; e < a; ++e) w[8 * zk + e] = 0;
      if constexpr (TAIL) {
        const int p = W - base;  // first position right of the tile
        const int tk = p >> 3;
        if ((p & 7) && tk >= k0 && tk < kWinChunks)
          for (int e = p & 7; e < 8; ++e) w[8 * tk + e] = 0;
      }
    }
  }
  // The straddling chunk of window b - 1 becomes chunk 0 of window b.
  __device__ void move_head(int b) {
    const uint4* o = sm.win[(b - 1) & 1];
    uint4* w = sm.win[b & 1];
    const int i = win_row(2 * lane);
    const uint4 x = o[i + 4], y = o[i + kWinChunks + 4];  // win_row(2 lane + 1) = win_row(2 lane) + 5
    w[i] = x;
    w[i + kWinChunks] = y;
  }

  // A chunk whose columns c .. c + 7 all lie in the tile: one store where input
  // and output rows are aligned alike, else four or eight.  Those take a quarter
  // of the instructions of storing row by row, but touch every 32-byte sector
  // eight or sixteen times: the better way while a lone warp's instructions
  // decide (warp pairs: 43 us for an odd 1437x811 frame, 90 row by row), the
  // worse one when the GPU is full (4 1921x1081 rgb10 frames in 64x64
  // tiles, whole decode: 382 us, 326 us row by row).
  __device__ void store_whole(uint16_t* dst, const uint4 v) const {
    if (store_mode == 2) {
      *reinterpret_cast<uint4*>(dst) = v;
      return;
    }
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (store_mode == 1) {
        reinterpret_cast<uint32_t*>(dst)[e] = w[e];
      } else {
        dst[2 * e] = static_cast<uint16_t>(w[e]);
        dst[2 * e + 1] = static_cast<uint16_t>(w[e] >> 16);
      }
    }
  }
  __device__ void store_edge(uint16_t* dst, const uint4* src, int c) const {
    const uint16_t* s = reinterpret_cast<const uint16_t*>(src);
    for (int e = max(0, -c); e < min(8, W - c); ++e) dst[e] = s[e];
  }
  // Positions 0..31 of window b, row by row: a warp's stores lie side by side.
  template <typename T>
  __device__ void flush_rows(int b) {
    constexpr int kPer = sizeof(T) / 2;             // samples a lane
    constexpr int kSide = kPer;                     // rows side by side, 64 / kSide apart
    constexpr int kRows = 8 / kSide;                // of the eight rows k, k + 8, ...
    const int side = kSide == 2 ? lane >> 4 : 0, p = kPer * (kSide == 2 ? lane & 15 : lane);
#pragma unroll 1
    for (int r = 0; r < 8; ++r) {
      const int row = r + side * (kBandRows / 2);
      int c = 32 * b + p - skew(row) - off_of(row);
      uint16_t* dst = out + row * out_pitch + c;
      const uint16_t* src = reinterpret_cast<const uint16_t*>(sm.win[b & 1] + win_row(row)) + p;
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        if (row + 8 * i < nrows && static_cast<unsigned>(c) < static_cast<unsigned>(W))
          *reinterpret_cast<T*>(dst) = *reinterpret_cast<const T*>(src);
        dst += out_hop;
        src += 8 * kWinHop;
        c -= 1 << kShift;
      }
    }
  }
  // Positions 0..31 of window b, all rows, to the output.
  __device__ void flush(int b) {
    if (ROWS && store_mode != 2) {
      if (store_mode == 1) flush_rows<uint32_t>(b);
      else flush_rows<uint16_t>(b);
      return;
    }
    const int c = c_first + 32 * b;
    uint16_t* dst = out + lr * out_pitch + c;
    const uint4* src = sm.win[b & 1] + kWinChunks * lr + lj;
    // rows whose chunk lies in the tile as a whole
    const uint32_t whole = bit_range((c + 8 - W + (1 << kShift) - 1) >> kShift, min(c >> kShift, row_top));
    if (ROWS || store_mode == 2) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (whole & (1u << i)) *reinterpret_cast<uint4*>(dst + i * out_hop) = src[kWinHop * i];
    } else {
#pragma unroll 2
      for (int i = 0; i < 8; ++i)
        if (whole & (1u << i)) store_whole(dst + i * out_hop, src[kWinHop * i]);
    }
    if (ragged) {
      const uint32_t part = bit_range((c - W + (1 << kShift)) >> kShift, min((c + 7) >> kShift, row_top)) & ~whole;
#pragma unroll 1
      for (int i = 0; i < 8; ++i)
        if (part & (1u << i)) store_edge(dst + i * out_hop, src + kWinHop * i, c - (i << kShift));
    }
  }
  // After the last block: its positions 0..31, and the straddling chunk.
  __device__ void flush_last() {
    const int b = nblk - 1;
    flush(b);
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      const int row = 2 * lane + h;
      const int c = 32 * b + 32 - skew(row) - (h ? off1 : off0);
      if (row < nrows && c > -8 && c < W) {
        const uint4* src = sm.win[b & 1] + win_row(row) + 4;
        uint16_t* dst = out + row * out_pitch + c;
        if (c >= 0 && c + 8 <= W) store_whole(dst, *src);
        else store_edge(dst, src, c);
      }
    }
  }
};

// Group of eight steps of one row's window words.  A row whose first position
// is even has steps 2i and 2i+1 in word i; one whose first position is odd
// has steps 2i-1 and 2i there, so the group spans five words, the first kept
// from the group before.  Rows 2r start even; rows 2r + 1, one step later,
// start odd, unless the row pitch is odd.
template <bool ODD>
struct WaveWords {
  uint32_t w[5];
  __device__ void first(const uint32_t* p) { if (ODD) w[0] = p[0]; }
  __device__ void after(const WaveWords& o) { if (ODD) w[0] = o.w[4]; }
  __device__ void load(const uint32_t* p, int g) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i + (ODD ? 1 : 0)] = p[4 * g + i + (ODD ? 1 : 0)];
  }
  __device__ uint32_t word(int j) const { return w[ODD ? (j + 1) >> 1 : j >> 1]; }
  static __device__ constexpr bool high(int j) { return ODD ? !(j & 1) : (j & 1); }  // step j's half of word(j)
  __device__ uint32_t sample(int j) const { return high(j) ? word(j) >> 16 : word(j) & 0xffffu; }
};

// Both rows' samples of step j in one register.
template <bool O1>
__device__ __forceinline__ uint32_t wave_pack(const WaveWords<false>& x, const WaveWords<O1>& y, int j) {
  const uint32_t sel = (WaveWords<false>::high(j) ? 0x32u : 0x10u) | (WaveWords<O1>::high(j) ? 0x7600u : 0x5400u);
  return __byte_perm(x.word(j), y.word(j), sel);
}

// Pointers of one window block of a lane, and the stores of its results: two
// steps a word, over the samples they came from.
template <bool O1>
struct WaveBlock {
  uint32_t* p0;
  uint32_t* p1;
  const uint16_t* crow;  // lane 0: the carry row, column of the block's first step
  uint32_t* cout;        // lane 31: where the last row of the band goes
  int lane;
  // `above`: the carry row that the band above wrote (its own, or the partner's)
  __device__ WaveBlock(WaveSm& sm, const uint16_t* above, int b, int lane_, int off0, int off1) : lane(lane_) {
    uint4* win = sm.win[b & 1] + win_row(2 * lane);
    p0 = reinterpret_cast<uint32_t*>(win) + (off0 >> 1);
    p1 = reinterpret_cast<uint32_t*>(win + kWinChunks) + (off1 >> 1);
    crow = above + kCarryPad + 32 * b;
    cout = reinterpret_cast<uint32_t*>(sm.carry + kCarryPad + 32 * b - 1 - wave_skew(kBandRows - 1));
  }
  // Results of step j of group g, packed (even row low), and those of the
  // step before; the carry row takes the reconstruction's.
  __device__ void put(int g, int j, uint32_t was, uint32_t now, uint32_t last_was, uint32_t last_now) {
    const int i = 4 * g + (j >> 1);
    if (j & 1) p0[i] = __byte_perm(was, now, 0x5410);
    if (O1 == !(j & 1)) p1[i] = __byte_perm(was, now, 0x7632);
    if (!(j & 1) && lane == 31) cout[i] = __byte_perm(last_was, last_now, 0x7632);
  }
  // after step 31: the half word that the next block's first word completes
  __device__ void finish(uint32_t now, uint32_t last_now) {
    if (O1) *reinterpret_cast<uint16_t*>(p1 + 16) = static_cast<uint16_t>(now >> 16);
    if (lane == 31) *reinterpret_cast<uint16_t*>(cout + 16) = static_cast<uint16_t>(last_now >> 16);
  }
};

// A warp pair's sweep of a tile, for launches that leave most of the
// GPU's warps idle: band j runs on warp j % 2, three blocks behind band j - 1, whose
// last row has then reached the columns that the block reads (row 63 is two
// blocks behind row 0), in lock-step at the pair's barrier after every block.  A
// carry row is overwritten by the band after next, at least three blocks behind
// its reader.  Band j starts in slot wave_start(j, blocks).
__device__ __forceinline__ int wave_start(int j, int blocks) {
  return blocks >= 6 ? (j >> 1) * blocks + (j & 1) * 3 : 3 * j;
}
__device__ __forceinline__ void wave_pair_sync(int warp) {
  asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");
}

// Sweeps a tile: begin() at each of the warp's bands, block(b) for its blocks,
// end() after the last, by one warp or a pair.
template <bool PAIR, typename Io, typename Begin, typename Block, typename End>
__device__ __forceinline__ void wave_sweep(Io& io, int height, int warp, Begin begin, Block block, End end) {
  if constexpr (!PAIR) {
    for (int y = 0; y < height; y += kBandRows, io.next_band()) {
      io.band(height - y);
      begin();
      for (int b = 0; b < io.nblk; ++b) block(b);
      end();
    }
  } else {
    const int bands = (height + kBandRows - 1) / kBandRows;
    io.band(kBandRows);
    const int full = io.nblk;
    io.band(height - (bands - 1) * kBandRows);
    const int slots = wave_start(bands - 1, full) + io.nblk;  // the last band ends last
    int j = warp & 1;
    if (j) io.next_band();
    for (int slot = 0; slot < slots; ++slot) {
      if (j < bands) {
        const int b = slot - wave_start(j, full);
        if (b == 0) {
          io.band(height - j * kBandRows);
          begin();
        }
        if (b >= 0) {
          block(b);
          if (b == io.nblk - 1) {
            end();
            j += 2;
            io.next_band();
            io.next_band();
          }
        }
      }
      wave_pair_sync(warp);
    }
  }
}

struct WaveCarry {
  uint32_t up[4];  // eight columns of the carry row
  __device__ void load(const uint16_t* crow, int g) {
    const uint4 c = *reinterpret_cast<const uint4*>(crow + 8 * g);
    up[0] = c.x;
    up[1] = c.y;
    up[2] = c.z;
    up[3] = c.w;
  }
};

// What a lane keeps from step to step, packed (even row in the low half).
struct WavePacked {
  uint32_t rec = 0, above = 0;
  __device__ uint32_t packed() const { return rec; }

  // The upper neighbours of this step: the even row's from the lane below in
  // rank (lane 0: the carry row), the odd row's from the lane's last step.
  __device__ uint32_t neighbours(uint32_t carry, int odd_step, int lane) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, rec, 1);
    const uint32_t sel = (lane == 0 && !odd_step) ? 0x5410u : 0x5432u;
    return __byte_perm(lane == 0 ? carry : up, rec, sel);
  }
  template <bool MED>
  __device__ uint32_t predict(uint32_t a, uint32_t maxs2) {
    const uint32_t d = sub2(a, above);
    if (MED) {
      const uint32_t mn = __vmins2(rec, a), mx = __vmaxs2(rec, a);
      return __vmaxs2(mn, __viaddmin_s16x2(rec, d, mx));
    }
    return __viaddmin_s16x2_relu(rec, d, maxs2);
  }
};

// The same in 32 bits a row (depth 16).
struct WaveWide {
  int32_t rec0 = 0, rec1 = 0, above0 = 0, above1 = 0;
  __device__ uint32_t packed() const { return __byte_perm(rec0, rec1, 0x5410); }

  __device__ void neighbours(uint32_t carry, int odd_step, int lane, int32_t& a0, int32_t& a1) {
    const int32_t up = __shfl_up_sync(0xffffffffu, rec1, 1);
    a0 = lane == 0 ? static_cast<int32_t>(odd_step ? carry >> 16 : carry & 0xffffu) : up;
    a1 = rec0;
  }
  template <bool MED>
  static __device__ int32_t predict(int32_t l, int32_t a, int32_t ul, int32_t maxs) {
    if (MED) return predict_med(l, a, ul);
    return __viaddmin_s32_relu(l, a - ul, maxs);
  }
};

}  // namespace fvb
