// fvb_decode.cu -- sm_100a decoder kernels for the fastvid intra codec.
//
//   dec_parse        : thread-per-tile directory + shard-header walk
//                      (reference decode.cu:131-220)
//   dec_rans_tables, dec_rans, dec_other : entropy decode of every mode with
//                      every rejection rule of the reference (decode.cu:222-550)
//   dec_reconstruct  : warp-per-tile (or warp-pair) wavefront, the mirror of
//                      enc_predict (decode.cu:552-606)
//   dec_reconstruct_serial : one thread per tile, raster order
//                      (decode.cu:608-656; the predictor="serial" diagnostic)
// A frame whose parse failed is skipped by the later kernels, so they never
// read shard records that were not written.
#include "fvb_common.cuh"
#include "fvb_kernels.cuh"
#include "fvb_wave.cuh"

namespace fvb {

namespace {
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ int frame_of_tile(const FrameDesc* frames, int nframes, int64_t t) {
  int lo = 0, hi = nframes - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (frames[mid].tile_base <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ uint32_t rd16(const uint8_t* p) { return p[0] | (static_cast<uint32_t>(p[1]) << 8); }
__device__ __forceinline__ uint32_t rd32(const uint8_t* p) {
  return p[0] | (static_cast<uint32_t>(p[1]) << 8) | (static_cast<uint32_t>(p[2]) << 16) |
         (static_cast<uint32_t>(p[3]) << 24);
}
__device__ __forceinline__ uint64_t rd64(const uint8_t* p) {
  return rd32(p) | (static_cast<uint64_t>(rd32(p + 4)) << 32);
}
constexpr int kRiceSmall = 1024;  // see rice_shard
__device__ __forceinline__ int list_of(int mode, int count) {
  return mode == kModeOrder0 ? 0 : (mode >= 1 && mode <= 17) ? (count > kRiceSmall ? 1 : 4) : mode == 0 ? 2 : 3;
}
__device__ __forceinline__ int64_t list_slot(int list, int64_t pos, int64_t total_shards) {
  return list == 4 ? 2 * total_shards - 1 - pos : list * total_shards + pos;
}
}  // namespace

// ---------------------------------------------------------------------------
// dec_parse: directory entry checks (status 10) and shard header walk
// (status 11), one thread per tile.

__global__ void dec_parse_kernel(const FrameDesc* __restrict__ frames, FrameState* __restrict__ state,
                                 const BatchDims* __restrict__ dims, ShardInfo* __restrict__ shards,
                                 DecodeLists* __restrict__ lists, int32_t* __restrict__ list_items) {
  const int nframes = dims->frames_p[0];
  const int64_t total_tiles = dims->tiles_p[0], total_shards = dims->shards_p[0];
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total_tiles;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int fi = frame_of_tile(frames, nframes, t);
    const FrameDesc& f = frames[fi];
    FrameState& st = state[fi];
    const int64_t lt = t - f.tile_base;
    const TileGeo g = tile_geo(f, lt);
    const uint8_t* enc = f.stream;
    const int64_t size = f.stream_len;
    const int64_t dir_end = kHeaderBytes + f.ntiles * kDirBytes;
    const uint8_t* e = enc + kHeaderBytes + lt * kDirBytes;
    if (e[0] != g.plane || e[1] != kModeOrder0 || e[2] != kPredictTag || e[3] != 0 ||
        rd32(e + 4) != static_cast<uint32_t>(g.x) || rd32(e + 8) != static_cast<uint32_t>(g.y) ||
        rd32(e + 12) != static_cast<uint32_t>(g.w) || rd32(e + 16) != static_cast<uint32_t>(g.h)) {
      set_status(&st.status, 10);
      continue;
    }
    const uint64_t off_u = rd64(e + 20);
    if (off_u > static_cast<uint64_t>(size)) {
      set_status(&st.status, 10);
      continue;
    }
    const int64_t off = static_cast<int64_t>(off_u);
    const int64_t plen = rd32(e + 28);
    if (plen > size - off) {
      set_status(&st.status, 10);
      continue;
    }
    if (lt == 0) {
      if (off != dir_end) {
        set_status(&st.status, 10);
        continue;
      }
    } else {
      const uint64_t poff = rd64(e - kDirBytes + 20);
      const uint64_t plen2 = rd32(e - kDirBytes + 28);
      if (poff > static_cast<uint64_t>(size) || plen2 > static_cast<uint64_t>(size) - poff || off_u != poff + plen2) {
        set_status(&st.status, 10);
        continue;
      }
    }
    if (lt + 1 == f.ntiles && off + plen != size) {
      set_status(&st.status, 10);
      continue;
    }
    const int64_t samples = static_cast<int64_t>(g.w) * g.h;
    const int64_t tile_end = off + plen;
    int64_t cursor = off, decoded = 0;
    bool ok = true;
    for (int j = 0; j < g.shard_count; ++j) {
      if (cursor > tile_end - 3) {
        ok = false;
        break;
      }
      const int mode = enc[cursor];
      const int64_t bl = rd16(enc + cursor + 1);
      const int64_t bo = cursor + 3;
      if (mode > 19 || bl > tile_end - bo) {
        ok = false;
        break;
      }
      const int64_t cnt = min(static_cast<int64_t>(kShardSymbols), samples - decoded);
      ShardInfo& si = shards[f.shard_base + g.first_shard + j];
      si.mode = mode;
      si.offset = bo;
      si.body = static_cast<int32_t>(bl);
      si.count = static_cast<int32_t>(cnt);
      si.sample_base = f.sample_base + g.sample_base + decoded;
      si.frame = fi;
      decoded += cnt;
      cursor = bo + bl;
    }
    if (!ok || decoded != samples || cursor != tile_end) {
      set_status(&st.status, 11);
      continue;
    }
    // bin the tile's shards by entropy mode for dec_shards; the lanes that
    // bin into the same list together take their slots with one atomic
    // (every shard of a batch lands on one of four counters)
    const int lane = static_cast<int>(threadIdx.x & 31);
    for (int j = 0; j < g.shard_count; ++j) {
      const int64_t s = f.shard_base + g.first_shard + j;
      const int list = list_of(shards[s].mode, shards[s].count);
      const unsigned active = __activemask();
      const unsigned peers = __match_any_sync(active, list);
      const int leader = __ffs(peers) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(&lists->count[list], __popc(peers));
      base = __shfl_sync(peers, base, leader);
      const int pos = base + __popc(peers & ((1u << lane) - 1u));
      list_items[list_slot(list, pos, total_shards)] = static_cast<int32_t>(s);
    }
  }
}

// ---------------------------------------------------------------------------
// Entropy decode (decode.cu:222-550).  dec_parse bins shards by mode; then
//   dec_rans_tables  a warp per rANS shard parses its order-0 table
//                    (decode.cu:456-517) into a table record
//   dec_rans         four threads per rANS shard, one on each of its lanes
//                    (decode.cu:530-549), through the record's bucket table or
//                    (few shards) a table of all slots
//   dec_other        a CTA per Rice shard (decode.cu:297-340), a warp per
//                    zero-run (decode.cu:237-295) or block shard
//                    (decode.cu:342-396)

constexpr int kBucketShift = 4;   // a bucket covers 16 slots
constexpr int kBuckets = (1 << kRansTableLog) >> kBucketShift;

// One parsed order-0 table (decode.cu:456-517).  Symbol i covers slots
// cum_i .. cum_i + freq_i - 1 of the 4096-slot ring.  data holds
//  * per symbol, an entry: freq - 1 in bits 31..20, cum in bits 19..8, and in
//    bits 7..0 what the symbol stores (its value as u16, or fold_value of it)
//    when every symbol's, as a signed number, fits eight bits (narrow), else
//    the symbol's index;
//  * per symbol, what it stores, as u16;
//  * for up to kBucketSymbols symbols, a bucket table: word u = (four times
//    the symbol holding slot 16u) << 16, with bit i set for every symbol that
//    starts at slot 16u + i (i = 1..15).  The symbol holding a slot is then
//    the bucket's first plus the starts at or below the slot inside the
//    bucket: one load and a population count, no search.
constexpr int kBucketSymbols = 170;
struct RansTable {
  int32_t lane_start[4], lane_len[4];
  uint32_t state[4];
  int32_t nsym, valid, narrow;
  int32_t pad;
  uint32_t data[512];
  __host__ __device__ static int entries_at(int nsym) { return nsym <= kBucketSymbols ? kBuckets : 0; }
  __host__ __device__ static int values_at(int nsym) { return entries_at(nsym) + nsym; }
};
static_assert(kBuckets + kBucketSymbols + (kBucketSymbols + 1) / 2 <= 512 && 255 + 128 <= 512, "table record");
static_assert(sizeof(RansTable) == 2112, "the scratch limit of the allocation-free decode counts on it");

size_t dec_rans_table_bytes() { return sizeof(RansTable); }

// Varint tokens of a byte string, 32 bytes a step, by a warp.  A byte without
// the 0x80 bit ends a token (ballot); the lane holding a token's last byte
// gathers the token's bytes from the lanes before it by shuffles, with the
// bytes of a token begun in an earlier step carried over.  `bad` covers the
// varint rules: at most five bytes, the fifth at most 0x0f, canonical length.
struct TokenReader {
  uint32_t pend_val = 0;  // value bits of a token begun in an earlier step
  int pend_used = 0;      // its bytes so far (capped at 6)
  bool pend_bad = false;  // its fifth byte was above 0x0f, or it is too long
  uint32_t endm;          // this step: lanes holding a token's last byte
  __device__ uint32_t step(uint32_t byte, bool vld, int nvalid, int lane, bool& bad) {
    endm = __ballot_sync(kFull, vld && !(byte & 0x80u));
    const uint32_t below = endm & ((1u << lane) - 1u);
    const int prev = below ? 31 - __clz(below) : -1;  // the previous token's end in this step
    const bool carried = prev < 0;                    // the token began in an earlier step
    const int here = lane - prev;                     // its bytes in this step
    const int cu = carried ? pend_used : 0;
    uint32_t tok = carried ? pend_val : 0u;
    bad = carried && pend_bad;
#pragma unroll
    for (int t = 0; t < 5; ++t) {
      const uint32_t bt = __shfl_sync(kFull, byte, max(lane - t, 0));
      const int p = cu + here - 1 - t;  // position of byte lane - t in the token
      if (t < here && p < 5) {
        tok |= (bt & 0x7fu) << (7 * p);
        if (p == 4 && bt > 0x0fu) bad = true;
      }
    }
    if (cu + here > 5) bad = true;
    if (!bad && cu + here != varint_len(tok)) bad = true;
    // bytes after the step's last token end begin (or continue) a token
    const int last_end = endm ? 31 - __clz(endm) : -1;
    const int tail = nvalid - 1 - last_end;
    if (tail > 0) {
      const int c0 = endm ? 0 : pend_used;
      uint32_t v = endm ? 0u : pend_val;
      bool pb = endm ? false : pend_bad;
#pragma unroll
      for (int t = 0; t < 5; ++t) {
        const uint32_t bt = __shfl_sync(kFull, byte, min(last_end + 1 + t, 31));
        const int p = c0 + t;
        if (t < tail && p < 5) {
          v |= (bt & 0x7fu) << (7 * p);
          if (p == 4 && bt > 0x0fu) pb = true;
        }
      }
      pend_val = v;
      pend_used = min(c0 + tail, 6);
      pend_bad = pb || c0 + tail > 5;
    } else {
      pend_val = 0;
      pend_used = 0;
      pend_bad = false;
    }
    return tok;
  }
};

__device__ __forceinline__ uint32_t scan_add(uint32_t v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

struct TableSm {
  uint16_t starts[kBuckets];  // bit i of word u: a symbol starts at slot 16u + i
  uint32_t entry[256];
  uint16_t value[256];
};

// Order-0 table of one shard, parsed by a warp (decode.cu:456-517).  Tokens:
// the symbol count n, then per symbol the value's delta and its frequency
// (none for the last).  Values and cumulative frequencies are warp prefix sums
// over the tokens of a step, in 32-bit arithmetic like the serial parser's
// running sums; a table is rejected exactly when one of the serial parser's
// checks fails at some symbol.
__device__ bool rans_parse_warp(const uint8_t* __restrict__ body, int blen, uint32_t maxf, const FoldMap& fm,
                                bool fold16, RansTable& t, TableSm& sm, int lane) {
#pragma unroll
  for (int i = 0; i < kBuckets / 64; ++i) reinterpret_cast<uint32_t*>(sm.starts)[32 * i + lane] = 0;
  __syncwarp();
  if (blen < 1 || body[0] != kRansTableLog) return false;
  TokenReader tr;
  int tokens = 0, n = 0;  // tokens of the steps so far; symbols, once known
  uint32_t val0 = 0, cum0 = 0;
  int cursor = 1;
  bool wide = false;
  for (;;) {
    if (cursor >= blen) return false;
    const bool vld = cursor + lane < blen;
    const uint32_t byte = vld ? body[cursor + lane] : 0u;
    bool bad;
    const uint32_t tok = tr.step(byte, vld, min(32, blen - cursor), lane, bad);
    const bool is_end = (tr.endm >> lane) & 1u;
    const int at = tokens + __popc(tr.endm & ((1u << lane) - 1u));  // this token's number
    if (tokens == 0 && tr.endm) {
      const int first = __ffs(tr.endm) - 1;
      const uint32_t count = __shfl_sync(kFull, tok, first);
      if (__shfl_sync(kFull, bad, first) || count == 0 || count > 255) return false;
      n = static_cast<int>(count);
    }
    const int i = (at - 1) >> 1;
    const bool is_sym = is_end && at > 0 && i < n;
    const bool is_freq = is_sym && !(at & 1);   // even numbers from 2: frequencies
    const bool is_delta = is_sym && (at & 1);
    const bool last = i == n - 1;
    const bool use = is_delta || (is_freq && !last);
    const uint32_t vals = scan_add(is_delta ? tok : 0u, lane) + val0;
    const uint32_t cums = scan_add(is_freq && !last ? tok : 0u, lane) + cum0;
    bool no = use && bad;
    if (is_delta) no |= (i != 0 && tok == 0) || vals > maxf;
    const bool whole = (is_freq && !last) || (is_delta && last);  // the symbol's frequency is known
    const uint32_t fr = last ? (1u << kRansTableLog) - cums : tok;
    const uint32_t cum = last ? cums : cums - tok;
    if (is_freq && !last) no |= fr == 0 || fr >= (1u << kRansTableLog) - cum;
    if (__any_sync(kFull, no)) return false;
    if (whole) {
      const uint32_t store = fm.lim ? fold_value<uint16_t>(vals, fm) : vals & 0xffffu;
      sm.value[i] = static_cast<uint16_t>(store);
      // (u32 symbols are not sign-extended to 16 bits but to 32)
      wide |= static_cast<int16_t>(store) != static_cast<int8_t>(store) || (!fold16 && store > 127u);
      sm.entry[i] = ((fr - 1u) << 20) | (cum << 8);
      // two buckets a word
      atomicOr(reinterpret_cast<uint32_t*>(sm.starts) + (cum >> 5), 1u << (cum & 31u));
    }
    const int count_here = __popc(tr.endm);
    if (n && tokens + count_here >= 2 * n) {  // the last delta is in this step
      const uint32_t lastm = __ballot_sync(kFull, is_delta && last);
      cursor += __ffs(lastm);
      break;
    }
    tokens += count_here;
    val0 = __shfl_sync(kFull, vals, 31);
    cum0 = __shfl_sync(kFull, cums, 31);
    cursor += 32;
  }
  // three lane lengths, four states (each at least kRansL); the fourth lane
  // takes the rest
  if (cursor + 28 > blen) return false;
  const uint32_t w = lane < 7 ? rd32(body + cursor + 4 * lane) : 0u;
  cursor += 28;
  const bool no = (lane < 3 && w >= (1u << 31)) || (lane >= 3 && lane < 7 && w < kRansL);
  if (__any_sync(kFull, no)) return false;
  int64_t start = cursor;
  int64_t len[4];
  for (int l = 0; l < 3; ++l) len[l] = __shfl_sync(kFull, w, l);
  len[3] = blen - start - len[0] - len[1] - len[2];
  if (len[3] < 0) return false;
  wide = __any_sync(kFull, wide);
  __syncwarp();
  if (lane < 4) {
    for (int l = 0; l < lane; ++l) start += len[l];
    t.lane_start[lane] = static_cast<int32_t>(start);
    t.lane_len[lane] = static_cast<int32_t>(len[lane]);
  }
  if (lane >= 3 && lane < 7) t.state[lane - 3] = w;
  if (lane == 0) {
    t.nsym = n;
    t.narrow = !wide;
  }
  uint32_t* entries = t.data + RansTable::entries_at(n);
  uint16_t* values = reinterpret_cast<uint16_t*>(t.data + RansTable::values_at(n));
  for (int i = lane; i < n; i += 32) {
    entries[i] = sm.entry[i] | (wide ? static_cast<uint32_t>(i) : sm.value[i] & 0xffu);
    values[i] = sm.value[i];
  }
  if (n <= kBucketSymbols) {
    // lane l: buckets 8l .. 8l + 7
    const uint4 m = reinterpret_cast<const uint4*>(sm.starts)[lane];
    const uint32_t w4[4] = {m.x, m.y, m.z, m.w};
    const uint32_t mine = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
    uint32_t before = scan_add(mine, lane) - mine;  // symbols that start in earlier buckets
    uint32_t b[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t m16 = (k & 1) ? w4[k >> 1] >> 16 : w4[k >> 1] & 0xffffu;
      b[k] = ((before + (m16 & 1u) - 1u) << 18) | (m16 & 0xfffeu);
      before += __popc(m16);
    }
    uint4* o = reinterpret_cast<uint4*>(t.data) + 2 * lane;
    o[0] = make_uint4(b[0], b[1], b[2], b[3]);
    o[1] = make_uint4(b[4], b[5], b[6], b[7]);
  }
  return true;
}

// A warp per rANS shard.  (A thread per shard, its serial parser waiting for
// every token, took 18 us for a 1080p frame, this takes 4 us; 16 4K rgb frames
// take 90 us, 13 more than that parser, but with the bucket tables that every
// dec_rans group used to build for itself.)
__global__ void __launch_bounds__(128)
dec_rans_tables_kernel(const FrameDesc* __restrict__ frames, FrameState* __restrict__ state,
                       const ShardInfo* __restrict__ shards, const DecodeLists* __restrict__ lists,
                       const int32_t* __restrict__ list_items, RansTable* __restrict__ tables, int fold16) {
  __shared__ __align__(16) TableSm sm_all[4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int count = lists->count[0];
  for (int p = blockIdx.x * 4 + warp; p < count; p += gridDim.x * 4) {
    const ShardInfo& si = shards[list_items[p]];
    FrameState& st = state[si.frame];
    RansTable& t = tables[p];
    bool ok = false;
    if (__any_sync(kFull, st.status == 0)) {  // a failed parse may have left shard records unwritten
      const FrameDesc& f = frames[si.frame];
      ok = rans_parse_warp(f.stream + si.offset, si.body, static_cast<uint32_t>(f.max_sample) * 2u,
                           fold_map(f, fold16), fold16 != 0, t, sm_all[warp], lane);
      if (!ok && lane == 0) set_status(&st.status, 5);
    }
    if (lane == 0) t.valid = ok;
    __syncwarp();
  }
}

// A lane's byte stream through a private ring of four 16-byte chunks in shared
// memory, fed by cp.async: all four before the first read, then one with
// every second eight-byte read (feed()).  Eight steps take at most 13 bytes, so
// the read position enters at most one new chunk between two feeds and the ring
// stays full whatever the data.  A feed may leave the newest two copies in
// flight: a chunk is copied when the read position is three chunks before it
// and read when it is one chunk before, at least two feeds later.  Of the
// lane's last chunk only the bytes up to the lane's end are copied (reading past
// them is an overrun that the byte count check reports).
template <int LANES>
struct LaneRing {
  static constexpr int kChunks = 4;
  uint32_t ring;          // shared address of slot 0 of this lane (slots LANES chunks apart)
  const uint8_t* next;    // global address of the next chunk to copy
  int at;                 // bit position of the next unread byte, from the first chunk's start
  int last, last_bytes;   // last chunk holding a lane byte (-1: none), and its bytes
  int fetched;            // number of the next chunk to copy

  __device__ void issue(int upto) {
    const uint32_t s = ring + (fetched & (kChunks - 1)) * (LANES * 16);
    const int ok = fetched <= min(last, upto);
    const int n = fetched == last ? last_bytes : 16;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %3, 0;\n @p cp.async.cg.shared.global [%0], [%1], 16, %2;\n}\n" ::"r"(s),
        "l"(next), "r"(n), "r"(ok)
        : "memory");
    fetched += ok;
    next += ok ? 16 : 0;
  }
  __device__ void init(uint4* ring_smem, const uint8_t* p, int len) {
    const int head = static_cast<int>(reinterpret_cast<uintptr_t>(p) & 15);
    next = p - head;
    at = 8 * head;
    ring = static_cast<uint32_t>(__cvta_generic_to_shared(ring_smem));
    last = len > 0 ? (head + len - 1) >> 4 : -1;
    last_bytes = ((head + len - 1) & 15) + 1;
    fetched = 0;
#pragma unroll
    for (int i = 0; i < kChunks; ++i) issue(kChunks - 1);
    cp_async_commit();
  }
  __device__ __forceinline__ void feed() {
    issue((at >> 7) + kChunks - 1);
    cp_async_commit();
    cp_async_wait<2>();
  }
  // The next eight bytes, first byte in the top bits of hi, the last four in lo.
  __device__ __forceinline__ void window(uint32_t& hi, uint32_t& lo) const {
    const uint32_t q = static_cast<uint32_t>(at) >> 6;  // pair of words holding the first byte
    auto pair = [&](uint32_t i) { return ring + ((i >> 1) & (kChunks - 1)) * (LANES * 16) + (i & 1) * 8; };
    uint32_t w0, w1, w2, w3;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w0), "=r"(w1) : "r"(pair(q)));
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w2), "=r"(w3) : "r"(pair(q + 1)));
    const bool upper = at & 32;
    const uint32_t a = upper ? w1 : w0, b = upper ? w2 : w1, c = upper ? w3 : w2;
    const uint32_t sel = 0x0123u + 0x1111u * ((static_cast<uint32_t>(at) >> 3) & 3u);
    hi = __byte_perm(a, b, sel);
    lo = __byte_perm(b, c, sel);
  }
};

// Shared memory of one dec_rans warp: eight shards' tables (bucket words, then
// the entries of up to kSymbols symbols; a shard with more reads its entries from
// its table record) and the lanes' byte rings; ROOMY: the symbols' values too, of
// any shard whose record has a bucket table.
constexpr int kGroups = 8;  // shards per warp, four lanes each
template <bool ROOMY>
struct alignas(16) RansWarpSm {
  // 36: five CTAs on an SM, 758 us for 16 4K rgb10 frames, 854 us with 64 and four
  static constexpr int kSymbols = ROOMY ? kBucketSymbols : 36;
  static constexpr int kWords = (kBuckets + kSymbols + 3) / 4 * 4;  // copied by 16 bytes
  static constexpr int kValueWords = ROOMY ? (kSymbols + 7) / 8 * 4 : 0;
  uint32_t table[kGroups][kWords + kValueWords];
  uint4 rings[LaneRing<32>::kChunks][32];
};
static_assert(RansWarpSm<true>::kSymbols <= kBucketSymbols && RansWarpSm<false>::kSymbols <= kBucketSymbols,
              "entries are copied with the bucket words");

template <bool ROOMY>
constexpr size_t dec_rans_smem() { return sizeof(RansWarpSm<ROOMY>) * kWarpsPerCta; }

// Bucket table of a shard of more than kBucketSymbols symbols, by its four
// lanes: lane l writes buckets 64l .. 64l + 63.
__device__ __forceinline__ void build_buckets(uint32_t* b, const uint32_t* entries, int nsym, int my_l) {
  constexpr uint32_t kSlots = 1u << kRansTableLog;
  auto start = [&](int i) { return i < nsym ? ((entries[i] >> 8) & (kSlots - 1u)) : kSlots; };
  int s = 0;
  uint32_t next = start(1);  // first slot of symbol s + 1
  for (int k = 0; k < kBuckets / 4; ++k) {
    const uint32_t u = static_cast<uint32_t>(my_l * (kBuckets / 4) + k);
    const uint32_t lo = u << kBucketShift;
    while (next <= lo) next = start(++s + 1);
    uint32_t w = static_cast<uint32_t>(s) << 18;
    for (int i = s + 1; next < lo + (1u << kBucketShift);) {
      w |= 1u << (next - lo);
      next = start(++i);
    }
    next = start(s + 1);
    b[u] = w;
  }
}

// The entry of the state's slot, through a shard's bucket table.
struct BucketLookup {
  const uint32_t* buckets;
  const uint32_t* entries;
  // x' = freq * (x >> 12) + slot - cum
  __device__ __forceinline__ uint32_t operator()(uint32_t& x) const {
    const uint32_t slot = x & ((1u << kRansTableLog) - 1u), xh = x >> kRansTableLog;
    const uint32_t bw = buckets[slot >> kBucketShift];
    // starts at offsets 1..r of the bucket survive the shift by 31 - r
    const uint32_t more = __popc(bw << ((slot & ((1u << kBucketShift) - 1u)) ^ 31u));
    const uint32_t e = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(entries) + (bw >> 16) + 4 * more);
    x = (e >> 20) * xh + (xh + slot - ((e >> 8) & 0xfffu));
    return e;
  }
};

// Through a table of all 4096 slots: entries with slot - cum in place of cum.
struct SlotLookup {
  const uint32_t* slots;
  __device__ __forceinline__ uint32_t operator()(uint32_t& x) const {
    const uint32_t xh = x >> kRansTableLog;
    const uint32_t e = slots[x & ((1u << kRansTableLog) - 1u)];
    x = (e >> 20) * xh + (xh + ((e >> 8) & 0xfffu));
    return e;
  }
};

// Bytes of b by prmt selector; a selector digit with its top bit set repeats
// the byte's sign (__byte_perm ignores that bit).
template <int SEL>
__device__ __forceinline__ uint32_t sign_bytes(uint32_t b) {
  uint32_t r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(b), "n"(SEL));
  return r;
}

template <typename FoldT>
__device__ __forceinline__ FoldT rans_value(uint32_t byte, bool narrow, const uint16_t* values) {
  const uint32_t v = narrow ? static_cast<uint32_t>(static_cast<int8_t>(byte)) : values[byte];
  return static_cast<FoldT>(v);
}

// The state map's renormalisation: after it x >= 2^11, so one byte comes in
// when x < 2^23 and a second when x < 2^15 (decode.cu:540-545).
__device__ __forceinline__ uint32_t rans_shift(uint32_t x) {
  const uint32_t sh = x < kRansL ? 8u : 0u;
  return x < (kRansL >> 8) ? 16u : sh;
}

// Four steps of a lane; byte k of the result is the low byte of step k's
// entry.  The bytes come from the top of an eight-byte window, as many as four
// steps can use; reading past the lane is an error, found by the byte count.
// `aside0`, `aside1` and `aside2` run between the steps, where the warp would
// wait for its lookups.
template <int LANES, typename Lookup, typename A0, typename A1, typename A2>
__device__ __forceinline__ uint32_t rans_four(const Lookup lookup, LaneRing<LANES>& ring, uint32_t& x, A0 aside0,
                                              A1 aside1, A2 aside2) {
  uint32_t hi, lo;
  ring.window(hi, lo);
  aside0();
  const uint32_t e0 = lookup(x);
  const uint32_t s0 = rans_shift(x);
  x = __funnelshift_l(hi, x, s0);
  aside1();
  const uint32_t e1 = lookup(x);
  const uint32_t s1 = rans_shift(x);
  x = __funnelshift_l(__funnelshift_l(lo, hi, s0), x, s1);
  const uint32_t half = s0 + s1;  // at most 32
  hi = __funnelshift_lc(lo, hi, half);
  lo = half < 32 ? lo << half : 0u;
  aside2();
  const uint32_t e2 = lookup(x);
  const uint32_t s2 = rans_shift(x);
  x = __funnelshift_l(hi, x, s2);
  const uint32_t e3 = lookup(x);
  const uint32_t s3 = rans_shift(x);
  x = __funnelshift_l(__funnelshift_l(lo, hi, s2), x, s3);
  ring.at += half + s2 + s3;
  return __byte_perm(__byte_perm(e0, e1, 0x0040), __byte_perm(e2, e3, 0x0040), 0x5410);
}

// Decode lane `my_l` of one shard: n symbols from this lane's byte ring,
// initial state x; lane l decodes symbols l, l + 4, ...  Returns the final
// state; the ring's position tells the bytes consumed.  Four steps' symbols of
// the four lanes, one byte each, are transposed among the lanes by two
// shuffles, so each lane stores four consecutive symbols at once.
template <typename FoldT, int LANES, typename Lookup>
__device__ __forceinline__ void rans_decode_lane(const Lookup lookup, bool narrow, const uint16_t* values,
                                                 LaneRing<LANES>& ring, FoldT* __restrict__ out, int n, int my_l,
                                                 unsigned group, uint32_t& x) {
  const uint32_t sel1 = my_l < 2 ? 0x5410u : 0x3276u, sel2 = (my_l & 1) ? 0x3715u : 0x6240u;
  out += 4 * my_l;
  // b: byte k is the byte of step my_l of lane k, i.e. of symbol 4 my_l + k of
  // sixteen
  auto put = [&](FoldT* o, uint32_t b) {
    if constexpr (sizeof(FoldT) == 2) {
      uint2 v;
      if (narrow) {
        v = make_uint2(sign_bytes<0x9180>(b), sign_bytes<0xb3a2>(b));
      } else {
        v.x = values[b & 0xffu] | (static_cast<uint32_t>(values[(b >> 8) & 0xffu]) << 16);
        v.y = values[(b >> 16) & 0xffu] | (static_cast<uint32_t>(values[b >> 24]) << 16);
      }
      *reinterpret_cast<uint2*>(o) = v;
    } else {
      uint4 v;
      if (narrow) {
        v = make_uint4(sign_bytes<0x8880>(b), sign_bytes<0x9991>(b), sign_bytes<0xaaa2>(b), sign_bytes<0xbbb3>(b));
      } else {
        v = make_uint4(values[b & 0xffu], values[(b >> 8) & 0xffu], values[(b >> 16) & 0xffu], values[b >> 24]);
      }
      *reinterpret_cast<uint4*>(o) = v;
    }
  };
  auto none = [] {};
  int left = n;
  // the bytes of the last 32 symbols (byte k: this lane's step k) are
  // transposed and stored while the next ones are decoded
  uint32_t b0 = 0, b1 = 0, t0 = 0, t1 = 0;
  auto swap2 = [&] {
    t0 = __shfl_xor_sync(group, b0, 2);
    t1 = __shfl_xor_sync(group, b1, 2);
  };
  auto swap1 = [&] {
    b0 = __byte_perm(b0, t0, sel1);
    b1 = __byte_perm(b1, t1, sel1);
    t0 = __shfl_xor_sync(group, b0, 1);
    t1 = __shfl_xor_sync(group, b1, 1);
  };
  auto store = [&] {
    put(out - 32, __byte_perm(b0, t0, sel2));
    put(out - 16, __byte_perm(b1, t1, sel2));
  };
  if (left >= 32) {
    ring.feed();
    b0 = rans_four<LANES>(lookup, ring, x, none, none, none);
    b1 = rans_four<LANES>(lookup, ring, x, none, none, none);
    left -= 32;
    out += 32;
    for (; left >= 32; left -= 32, out += 32) {
      ring.feed();
      const uint32_t n0 = rans_four<LANES>(lookup, ring, x, swap2, swap1, store);
      const uint32_t n1 = rans_four<LANES>(lookup, ring, x, none, none, none);
      b0 = n0;
      b1 = n1;
    }
    swap2();
    swap1();
    store();
  }
  if (left >= 16) {
    ring.feed();
    b0 = rans_four<LANES>(lookup, ring, x, none, none, none);
    swap2();
    swap1();
    put(out, __byte_perm(b0, t0, sel2));
    left -= 16;
    out += 16;
  }
  if (left > 0) {  // at most 15 symbols: at most four steps a lane
    ring.feed();
    uint32_t hi, lo;
    ring.window(hi, lo);
    out -= 4 * my_l;
    for (int i = my_l; i < left; i += 4) {
      out[i] = rans_value<FoldT>(lookup(x) & 0xffu, narrow, values);
      const uint32_t sh = rans_shift(x);
      x = __funnelshift_l(hi, x, sh);
      hi = __funnelshift_l(lo, hi, sh);
      lo <<= sh;
      ring.at += sh;
    }
  }
  cp_async_wait<0>();
}

// A warp takes eight rANS shards at a time (all shards but the last of a tile
// have 1,024 steps a lane), copies their tables into shared memory and decodes
// their 32 lanes.
//
// Bound by the chain of a step -- two dependent shared-memory lookups and a
// population count -- and, with 16 to 20 warps an SM, by the shared-memory pipe
// (12 cycles a step: the lookups hit about three banks twice) and issue (42
// instructions).  16 4K rgb10 frames: 1117 us with a lookup and a store of two
// bytes for every symbol's value and tables built by four lanes while the rest
// of the warp waited; 861 us with the value in the entry, 16-byte transposed
// stores and tables made once by dec_rans_tables; 750 us with 20 warps an SM.
// ROOMY is for launches that leave the SMs room (roomy_rans_shards).
template <typename FoldT, bool ROOMY>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
dec_rans_kernel(const FrameDesc* __restrict__ frames, FrameState* __restrict__ state,
                const ShardInfo* __restrict__ shards, DecodeLists* __restrict__ lists,
                const int32_t* __restrict__ list_items, const RansTable* __restrict__ tables,
                FoldT* __restrict__ folded) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  using Sm = RansWarpSm<ROOMY>;
  Sm& sm = reinterpret_cast<Sm*>(smem_raw)[warp];
  const int j = lane >> 2, my_l = lane & 3;
  const unsigned group = 0xfu << (4 * j);
  const int count = lists->count[0];
  for (;;) {
    int p0 = 0;
    if (lane == 0) p0 = atomicAdd(&lists->next_group_rans, kGroups);
    p0 = __shfl_sync(kFull, p0, 0);
    if (p0 >= count) break;
    const int p = p0 + j;
    const bool live = p < count && tables[p].valid;
    const RansTable& t = tables[live ? p : p0];
    const int nsym = live ? t.nsym : 0;
    const bool local = nsym <= Sm::kSymbols;
    LaneRing<32> ring;
    const ShardInfo* si = nullptr;
    const FrameDesc* f = nullptr;
    if (live) {
      si = &shards[list_items[p]];
      f = &frames[si->frame];
      ring.init(&sm.rings[0][lane], f->stream + si->offset + t.lane_start[my_l], t.lane_len[my_l]);
    }
    // the bucket words and the local entries, 16 bytes a copy
    const uint32_t* entries = t.data + RansTable::entries_at(nsym);
    if (live) {
      uint32_t* to = sm.table[j];
      if (nsym <= kBucketSymbols) {
        const int chunks = (kBuckets + (local ? nsym : 0) + 3) / 4;  // the entries follow the buckets
        for (int i = my_l; i < chunks; i += 4) cp_async16(to + 4 * i, t.data + 4 * i);
        if (ROOMY && !t.narrow)
          for (int i = my_l; i < (nsym + 1) / 2; i += 4) cp_async4(to + Sm::kWords + i, t.data + RansTable::values_at(nsym) + i);
      } else {
        build_buckets(to, entries, nsym, my_l);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();  // the four lanes of a shard read what each other copied or built; a vote orders no memory
    const bool all_local = __all_sync(kFull, local);
    if (live) {
      const uint16_t* values = reinterpret_cast<const uint16_t*>(t.data + RansTable::values_at(nsym));
      FoldT* out = folded + si->sample_base;
      uint32_t x = t.state[my_l];
      const int from = ring.at;
      const uint32_t* at = local ? sm.table[j] + kBuckets : entries;
      if (all_local)
        rans_decode_lane<FoldT, 32>(BucketLookup{sm.table[j], sm.table[j] + kBuckets}, t.narrow,
                                    ROOMY ? reinterpret_cast<const uint16_t*>(sm.table[j] + Sm::kWords) : values, ring,
                                    out, si->count, my_l, group, x);
      else
        rans_decode_lane<FoldT, 32>(BucketLookup{sm.table[j], at}, t.narrow, values, ring, out, si->count, my_l,
                                    group, x);
      if (ring.at - from != 8 * t.lane_len[my_l] || x != kRansL) set_status(&state[si->frame].status, 5);
    }
    __syncwarp();
  }
}

// Few shards: the chain of a step decides, not the number of lanes in flight.
// A warp of its own takes two shards and spreads their tables over all 4096
// slots (16 KB each), which leaves one lookup a step: a 1080p rgb10 frame of
// 1,539 shards takes 94 us here, 125 us in dec_rans_kernel's small tables.
constexpr int kSlotGroups = 2;
struct alignas(16) RansSlotSm {
  uint32_t slots[kSlotGroups][1 << kRansTableLog];
  uint4 rings[LaneRing<4 * kSlotGroups>::kChunks][4 * kSlotGroups];
  uint32_t entry[256];
  uint32_t bucket[kBuckets];
};
size_t dec_rans_slots_smem() { return sizeof(RansSlotSm); }

template <typename FoldT>
__global__ void __launch_bounds__(32)
dec_rans_slots_kernel(const FrameDesc* __restrict__ frames, FrameState* __restrict__ state,
                      const ShardInfo* __restrict__ shards, DecodeLists* __restrict__ lists,
                      const int32_t* __restrict__ list_items, const RansTable* __restrict__ tables,
                      FoldT* __restrict__ folded) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RansSlotSm& sm = *reinterpret_cast<RansSlotSm*>(smem_raw);
  const int lane = threadIdx.x;
  const int j = lane >> 2, my_l = lane & 3;
  const int count = lists->count[0];
  for (int p0 = blockIdx.x * kSlotGroups; p0 < count; p0 += gridDim.x * kSlotGroups) {
    const int p = p0 + j;
    const bool live = j < kSlotGroups && p < count && tables[p].valid;
    const RansTable& mine = tables[live ? p : p0];
    LaneRing<4 * kSlotGroups> ring;
    const ShardInfo* si = nullptr;
    if (live) {
      si = &shards[list_items[p]];
      ring.init(&sm.rings[0][lane], frames[si->frame].stream + si->offset + mine.lane_start[my_l],
                mine.lane_len[my_l]);
    }
    for (int g = 0; g < kSlotGroups && p0 + g < count; ++g) {
      const RansTable& t = tables[p0 + g];
      if (!t.valid) continue;
      const int nsym = t.nsym;
      const uint32_t* entries = t.data + RansTable::entries_at(nsym);
      __syncwarp();
      for (int i = lane; i < nsym; i += 32) sm.entry[i] = entries[i];
      if (nsym <= kBucketSymbols)
        for (int i = lane; i < kBuckets; i += 32) sm.bucket[i] = t.data[i];
      else if (lane < 4)
        build_buckets(sm.bucket, entries, nsym, lane);
      __syncwarp();
#pragma unroll 4
      for (int i = lane; i < (1 << kRansTableLog); i += 32) {
        const uint32_t bw = sm.bucket[i >> kBucketShift];
        const uint32_t e = sm.entry[(bw >> 18) + __popc(bw << ((i & ((1 << kBucketShift) - 1)) ^ 31))];
        sm.slots[g][i] = (e & 0xfff000ffu) | ((static_cast<uint32_t>(i) - ((e >> 8) & 0xfffu)) << 8);
      }
    }
    cp_async_wait<0>();
    __syncwarp();
    if (live) {
      const uint16_t* values = reinterpret_cast<const uint16_t*>(mine.data + RansTable::values_at(mine.nsym));
      uint32_t x = mine.state[my_l];
      const int from = ring.at;
      rans_decode_lane<FoldT, 4 * kSlotGroups>(SlotLookup{sm.slots[j]}, mine.narrow, values, ring,
                                               folded + si->sample_base, si->count, my_l, 0xfu << (4 * j), x);
      if (ring.at - from != 8 * mine.lane_len[my_l] || x != kRansL) set_status(&state[si->frame].status, 5);
    }
    __syncwarp();
  }
}

// Rice shards (decode.cu:297-340): a CTA of four warps per shard, 32 threads
// on each of its four Rice lanes.  A lane's codes can only be found one after
// another, so each thread takes a 32nd of the lane's bits and guesses where
// its first code starts: it reads codes from a little before its part, and
// such a reading falls in step with the true one after a few codes
// (Weissenberger & Schmidt, "Massively parallel Huffman decoding on GPUs",
// ICPP 2018).  Each thread then counts the codes of its part and hands the
// end of its last one to the next thread; where that differs from the guess,
// the part is read again from there.  Thread 0 starts at the true place, so
// after at most 32 rounds -- almost always one -- every start is the true one,
// and the codes are read once more for their values, now that their places
// are known from the counts.  The body is staged in shared memory, and the
// symbols leave from there in 16-byte stores.  Bound by the chain of one code
// (about 30 instructions and 180 cycles in a lone warp): one thread a lane
// read 1,024 of them in series, 100 us for the smallest frame with Rice
// shards; eight threads a lane (a warp per shard) took 28 us, 32 take 12 us.
//
// Small shards (kRiceSmall) go a warp each, eight threads a lane, when there are
// more than CTAs: with a few codes a thread a CTA's barriers and its other lead-ins
// cost more than the codes.  4 4K gray8 frames in 32x32 tiles (32,640 shards of
// 1,024 symbols) take 131 us so and 216 a CTA each, in 16x16 tiles 275 and 746;
// one 720p frame in 32x32 tiles (920 shards) 27 and 17, in 32x16 tiles (1,800) 23
// and 21, in 16x16 tiles (3,600) 19 and 29.  Shards of 2,048 symbols do as well
// either way.
constexpr int kOtherWarps = 4;
constexpr int kRiceStage = 8832;    // bytes of a body held in shared memory: above any that the encoder writes
constexpr int kRiceWave = 148 * 12;  // CTAs on the GPU at once
constexpr int kRiceNone = 0x7fffffff;

// The threads that decode a shard together: a CTA, or one of its warps with a
// quarter of the CTA's shared memory.
template <int WARPS>
struct RiceGroup {
  static constexpr int kThreads = 32 * WARPS;
  static constexpr int kParts = 8 * WARPS;  // threads per Rice lane
  static constexpr int kStage = kRiceStage * WARPS / kOtherWarps;
  static constexpr int kSymbols = kShardSymbols * WARPS / kOtherWarps;
  static constexpr int kBodyWords = (kStage + 48) / 4;
  static __device__ __forceinline__ void sync() {
    if (WARPS == 1) __syncwarp();
    else __syncthreads();
  }
  // whether any thread's is true; orders shared memory as sync() does
  static __device__ __forceinline__ bool any(bool b) {
    if (WARPS > 1) return __syncthreads_or(b);
    __syncwarp();
    return __any_sync(kFull, b);
  }
};
static_assert(RiceGroup<1>::kSymbols >= kRiceSmall, "a small shard's symbols");

template <typename FoldT>
struct alignas(16) RiceSm {
  uint32_t body[kOtherWarps * RiceGroup<1>::kBodyWords];
  FoldT out[kShardSymbols];
  int32_t stop[32 * kOtherWarps];
  int32_t total[kOtherWarps][4];
};
static_assert(kOtherWarps * RiceGroup<1>::kBodyWords >= RiceGroup<kOtherWarps>::kBodyWords &&
                  RiceGroup<1>::kBodyWords % 4 == 0, "staging");

// Words of a body, in shared memory or (a longer one) in global memory, where
// only words that hold a byte of it are read; words past the end are zero.
struct RiceBody {
  const uint32_t* words;
  int last;  // last word holding a byte of the body (global)
  bool staged;
  __device__ uint32_t operator[](int i) const {
    if (staged) return words[i];
    return i <= last ? __ldg(words + i) : 0u;
  }
};

// Reads codes from bit `pos` while they start before `lim`, in a lane that
// ends at bit `end`: emit(quotient, remainder, index) for each.  Returns the
// bit after the last code, or kRiceNone when no further code was found (`rest`
// is then where the search began; `bad`, which emit may share, is set when the
// lane ends within a code and never cleared).  The number of codes is added to n.
template <typename Emit>
__device__ __forceinline__ int rice_read(const RiceBody& body, int pos, int lim, int end, int k, int& n, int& rest,
                                         bool& bad, Emit emit) {
  const uint32_t mask = (1u << k) - 1u;
  const uint32_t ones = 0xffffffffu >> (k + 1);  // a one bit here ends a code of at most 31 bits
  while (pos < lim) {
    const int w = pos >> 5;
    const uint32_t a = body[w], b = body[w + 1], c = body[w + 2];
    uint32_t lo = __funnelshift_r(a, b, pos), hi = __funnelshift_r(b, c, pos);  // shift taken modulo 32
    // codes of at most 31 bits wholly inside these 64 bits and the lane
    const int avail = min(64, end - pos);
    const int enough = avail - (lim - pos);  // bits left when the part is done
    int left = avail;
    uint32_t hit;
    while ((hit = lo & ones) != 0) {
      const int z = __clz(__brev(hit)), tot = z + 1 + k;
      if (tot > left) break;
      emit(static_cast<uint32_t>(z), (lo >> z >> 1) & mask, n);
      ++n;
      lo = __funnelshift_r(lo, hi, tot);
      hi >>= tot;
      left -= tot;
      if (left <= enough) break;
    }
    pos += avail - left;
    if (left < avail) continue;
    // a longer code, or the end of the lane
    int p = pos;
    uint32_t x = lo;
    while (x == 0 && p < end) {
      p += 32;
      x = __funnelshift_r(body[p >> 5], body[(p >> 5) + 1], p);
    }
    p += x ? __ffs(x) - 1 : 0;
    if (p + 1 + k > end) {  // no further one bit in the lane, or one whose code would run past it
      rest = pos;
      bad |= p < end;
      return kRiceNone;
    }
    const int r = p + 1;
    emit(static_cast<uint32_t>(p - pos), __funnelshift_r(body[r >> 5], body[(r >> 5) + 1], r) & mask, n);
    ++n;
    pos = r + k;
  }
  return pos;
}

// A Rice shard by thread t of a group (of a CTA's warp w, when the group is a
// warp); returns whether it is valid (every thread the same).
template <int WARPS, typename FoldT>
__device__ bool rice_shard(int w, int t, const uint8_t* __restrict__ body, int blen, int n, int k, uint32_t maxf,
                           const FoldMap& fm, FoldT* __restrict__ out, RiceSm<FoldT>& sm) {
  using G = RiceGroup<WARPS>;
  uint32_t* const stage = sm.body + w * G::kBodyWords;
  FoldT* const sout = sm.out + w * G::kSymbols;
  int32_t* const stops = sm.stop + w * G::kThreads;
  const int warp = t >> 5, lane = t & 31;
  const int lc = min(4, n);
  const int table = (lc - 1) * 4;
  if (table > blen) return false;
  // the body, from a 16-byte boundary at or before it (the stream's header
  // lies before every body)
  const int head = static_cast<int>(reinterpret_cast<uintptr_t>(body) & 15);
  const uint8_t* from = body - head;
  const int bytes = head + blen;
  RiceBody rb;
  rb.staged = bytes <= G::kStage;
  rb.last = (bytes - 1) >> 2;
  if (rb.staged) {
    for (int i = 16 * t; i < bytes + 32; i += 16 * G::kThreads) {
      const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(stage)) + i;
      const int have = max(0, min(16, bytes - i));  // the rest of the 16 bytes is zeroed
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(have ? from + i : from), "r"(have)
                   : "memory");
    }
    cp_async_commit();
    rb.words = stage;
  } else {
    rb.words = reinterpret_cast<const uint32_t*>(from);
  }
  cp_async_wait<0>();
  G::sync();
  // thread: Rice lane rl, part `part` of its bits (bit positions from `from`)
  const int rl = t & 3, part = t >> 2;
  const bool live = rl < lc;
  bool bad = false;
  int64_t off = table, len = 0;
  for (int i = 0; i < lc - 1; ++i) {
    const int64_t v = rd32(body + 4 * i);
    if (i < rl) off += v;
    else if (i == rl) len = v;
  }
  if (rl == lc - 1) len = blen - off;
  if (off > blen || len < 0 || len > blen - off) bad = live;
  if (G::any(bad)) return false;
  const int nl = live ? (n - rl + lc - 1) / lc : 0;  // codes of the lane
  const int begin = 8 * (head + static_cast<int>(off)), end = live ? begin + 8 * static_cast<int>(len) : begin;
  const int size = end - begin;
  const int lo = begin + static_cast<int>(static_cast<int64_t>(size) * part / G::kParts);
  const int lim = begin + static_cast<int>(static_cast<int64_t>(size) * (part + 1) / G::kParts);
  auto skip = [](uint32_t, uint32_t, int) {};
  int start = begin, stop, count = 0, rest = begin;
  if (part) {
    start = rice_read(rb, max(begin, lo - (8 + k) * (k + 2)), lo, end, k, count, rest, bad, skip);
    if (start == kRiceNone) start = lo;
  }
  bool reread = true;
  for (int round = 0; round < G::kParts; ++round) {
    if (reread) {
      count = 0;
      bad = false;
      stop = start;
      if (start != kRiceNone) stop = rice_read(rb, start, lim, end, k, count, rest, bad, skip);
    }
    stops[t] = stop;
    G::sync();
    const int before = part ? stops[t - 4] : start;
    reread = before != start;
    start = before;
    if (!G::any(reread)) break;
  }
  int at = count;  // codes of the parts up to this one
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(kFull, at, o);
    if (lane >= o) at += v;
  }
  if constexpr (WARPS > 1) {
    if (lane >= 28) sm.total[warp][rl] = at;
    G::sync();
    for (int v = 0; v < warp; ++v) at += sm.total[v][rl];
  }
  // exactly the lane's codes, and fewer than eight bits left, all zero
  if (start != kRiceNone && stop == kRiceNone) bad |= end - rest > 7;
  if (part == G::kParts - 1) bad |= at != nl;
  at -= count;
  if (G::any(bad)) return false;
  if (start != kRiceNone) {
    int m = 0;
    rice_read(rb, start, lim, end, k, m, rest, bad, [&](uint32_t q, uint32_t r, int i) {
      const uint64_t v = (static_cast<uint64_t>(q) << k) + r;
      bad |= v > maxf;
      sout[(at + i) * lc + rl] = fold_value<FoldT>(static_cast<uint32_t>(v), fm);
    });
  }
  if (G::any(bad)) return false;
  constexpr int kPer = 16 / sizeof(FoldT);
  uint4* o4 = reinterpret_cast<uint4*>(out);  // shards start on 16-byte boundaries
  for (int i = t; i < n / kPer; i += G::kThreads) o4[i] = reinterpret_cast<const uint4*>(sout)[i];
  for (int i = n / kPer * kPer + t; i < n; i += G::kThreads) out[i] = sout[i];
  return true;
}

// A zero-run shard (decode.cu:237-295) decoded by the whole warp, 32 body
// bytes per step, one per lane: the step's tokens (TokenReader) are placed by
// a warp prefix sum of the symbols they stand for.  Every check of the serial
// parser is made -- the varint rules, a run no longer than the symbols left, a
// value in 1..maxf, no token after the last symbol, no partial token and no
// missing symbol at the end -- so a stream is accepted exactly when the serial
// parser accepts it.  The shard's symbols are zeroed first; value tokens then
// write theirs.  Warp-collective: every lane calls it with the same arguments.
// Returns whether the shard is valid.
template <typename FoldT>
__device__ bool zero_run_warp(const uint8_t* __restrict__ body, int64_t blen, int n, uint32_t maxf,
                              const FoldMap& fm, FoldT* __restrict__ out, int lane) {
  for (int i = lane; i < n; i += 32) out[i] = 0;
  __syncwarp();
  int produced = 0;  // symbols of the steps so far (warp-uniform)
  TokenReader tr;
  bool bad = false;
  for (int64_t base = 0; base < blen && !bad; base += 32) {
    const bool vld = base + lane < blen;
    const uint32_t byte = vld ? body[base + lane] : 0u;
    bool tb;
    const uint32_t tok = tr.step(byte, vld, static_cast<int>(min(static_cast<int64_t>(32), blen - base)), lane, tb);
    const bool is_end = (tr.endm >> lane) & 1u;
    uint32_t cnt = 0;
    if (is_end) {
      if (tok & 1u) {
        const uint32_t value = (tok + 1u) >> 1;  // u32 arithmetic as in the reference
        if (value == 0u || value > maxf) tb = true;
        cnt = 1;
      } else {
        cnt = min((tok >> 1) + 1u, static_cast<uint32_t>(n) + 1u);  // a run; longer than n fails below
      }
    }
    const uint32_t inc = scan_add(cnt, lane);
    const uint32_t start = static_cast<uint32_t>(produced) + inc - cnt;
    if (is_end) {
      if (start + cnt > static_cast<uint32_t>(n)) tb = true;  // a run past the end, or a token after it
      if (!tb && (tok & 1u)) out[start] = fold_value<FoldT>((tok + 1u) >> 1, fm);
    }
    bad = __any_sync(kFull, is_end && tb);
    produced += static_cast<int>(__shfl_sync(kFull, inc, 31));
  }
  return !bad && tr.pend_used == 0 && produced == n;
}

struct OtherGroupSm {
  int32_t boff[32], bwidth[32];
  int32_t valid;
};

template <typename FoldT>
struct OtherSm {
  RiceSm<FoldT> rice;
  OtherGroupSm block[kOtherWarps];
  int claimed;
};

size_t dec_other_smem(bool fold16) { return fold16 ? sizeof(OtherSm<uint16_t>) : sizeof(OtherSm<uint32_t>); }

// A CTA takes a large Rice shard, or four small ones, zero-run or block shards
// (one a warp).
template <typename FoldT>
__global__ void __launch_bounds__(32 * kOtherWarps)
dec_other_kernel(const FrameDesc* __restrict__ frames, FrameState* __restrict__ state,
                 const ShardInfo* __restrict__ shards, const BatchDims* __restrict__ dims,
                 DecodeLists* __restrict__ lists, const int32_t* __restrict__ list_items,
                 FoldT* __restrict__ folded) {
  const int64_t total_shards = dims->shards_p[0];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  OtherSm<FoldT>& osm = *reinterpret_cast<OtherSm<FoldT>*>(smem_raw);
  OtherGroupSm& sm = osm.block[warp];
  // work items: the large Rice shards, the small ones, the others
  const bool lone = lists->count[4] <= kRiceWave;  // small Rice shards go a CTA each, too
  int ends[5], items[5] = {0, 1, 4, 2, 3};
  ends[0] = 0;
#pragma unroll
  for (int i = 1; i < 5; ++i) {
    const int n = lists->count[items[i]];
    ends[i] = ends[i - 1] + (i == 1 || (i == 2 && lone) ? n : (n + kOtherWarps - 1) / kOtherWarps);
  }
  for (;;) {
    __syncthreads();  // the CTA's last shard is done, its claim read
    if (threadIdx.x == 0) osm.claimed = atomicAdd(&lists->next_group, 1);
    __syncthreads();
    int g = osm.claimed;
    if (g >= ends[4]) break;
    const int list = g < ends[1] ? 1 : g < ends[2] ? 4 : g < ends[3] ? 2 : 3;
    const bool cta = list == 1 || (list == 4 && lone);
    g -= list == 1 ? 0 : list == 4 ? ends[1] : list == 2 ? ends[2] : ends[3];
    if (!cta) g = g * kOtherWarps + warp;
    if (g >= lists->count[list]) continue;
    const ShardInfo& si = shards[list_items[list_slot(list, g, total_shards)]];
    const int fi = si.frame;
    // a failed parse may have left shard records unwritten.  (Only the parse
    // writes status 10 and 11; one set meanwhile by another shard must not
    // split the CTA or the warp, so they decide together.)
    const int failed = state[fi].status != 0;
    if (cta ? __syncthreads_or(failed) : __any_sync(kFull, failed)) continue;
    const FrameDesc& f = frames[fi];
    const int mode = si.mode, n = si.count, blen = si.body;
    const uint8_t* body = f.stream + si.offset;
    FoldT* out = folded + si.sample_base;
    const uint32_t maxf = static_cast<uint32_t>(f.max_sample) * 2u;
    const FoldMap fm = fold_map(f, sizeof(FoldT) == 2);
    if (cta) {
      if (!rice_shard<kOtherWarps>(0, threadIdx.x, body, blen, n, mode - 1, maxf, fm, out, osm.rice) && threadIdx.x == 0)
        set_status(&state[fi].status, 2);
    } else if (list == 4) {
      if (!rice_shard<1>(warp, lane, body, blen, n, mode - 1, maxf, fm, out, osm.rice) && lane == 0)
        set_status(&state[fi].status, 2);
    } else if (list == 2) {
      if (!zero_run_warp(body, blen, n, maxf, fm, out, lane) && lane == 0) set_status(&state[fi].status, 1);
    } else {
      const int nblk = (n + kBlockSymbols - 1) / kBlockSymbols;
      const int maxw = 32 - __clz(maxf);
      if (lane == 0) {
        int64_t cursor = 0;
        int ok = 1;
        for (int b = 0; b < nblk; ++b) {
          if (cursor >= blen) {
            ok = 0;
            break;
          }
          const int w = body[cursor++];
          if (w > maxw) {
            ok = 0;
            break;
          }
          const int64_t nb = min(static_cast<int64_t>(kBlockSymbols), static_cast<int64_t>(n) - static_cast<int64_t>(b) * kBlockSymbols);
          const int64_t pay = (nb * w + 7) / 8;
          if (pay > blen - cursor) {
            ok = 0;
            break;
          }
          sm.boff[b] = static_cast<int32_t>(cursor);
          sm.bwidth[b] = w;
          const int64_t bits = nb * w;
          if ((bits & 7) != 0) {
            const uint8_t mask = static_cast<uint8_t>(~((1u << (bits & 7)) - 1u));
            if (body[cursor + pay - 1] & mask) {
              ok = 0;
              break;
            }
          }
          cursor += pay;
        }
        if (ok && cursor != blen) ok = 0;
        sm.valid = ok;
        if (!ok) set_status(&state[fi].status, 3);
      }
      __syncwarp();
      if (sm.valid) {
        int bad = 0;
        for (int b = 0; b < nblk; ++b) {
          const int w = sm.bwidth[b];
          const uint8_t* pay = body + sm.boff[b];
          const int nb = min(kBlockSymbols, n - b * kBlockSymbols);
          for (int i = lane; i < nb; i += 32) {
            uint32_t v = 0;
            if (w) {
              const int64_t bit = static_cast<int64_t>(i) * w;
              const int64_t byte0 = bit >> 3;
              const int64_t lastb = (bit + w - 1) >> 3;
              uint64_t acc = 0;
              for (int64_t j = byte0; j <= lastb; ++j) acc |= static_cast<uint64_t>(pay[j]) << (8 * (j - byte0));
              v = static_cast<uint32_t>((acc >> (bit & 7)) & ((1ull << w) - 1));
            }
            if (v > maxf) bad = 1;
            out[static_cast<int64_t>(b) * kBlockSymbols + i] = fold_value<FoldT>(v, fm);
          }
        }
        if (__any_sync(kFull, bad) && lane == 0) set_status(&state[fi].status, 3);
      }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------------------
// dec_reconstruct: warp per tile, lane = row of a 32-row band, column c of
// row i at step c + i; the folded tile streams through a 64-column ring and
// the reconstruction is flushed to the output plane 32 columns at a time.

// Mirror of enc_tile_fast: the folded residuals stream in through a skewed
// 64-column ring, the reconstruction goes out through another and is flushed
// to the output plane 32 columns at a time (decode.cu:552-606).

struct RecWarpSmem {
  static constexpr int kFS = kFoldStride;
  uint32_t fold[32 * kFS];             // folded-residual ring (skewed)
  uint16_t out[32 * kSrcStride];    // reconstruction ring (u16, skewed)
  uint16_t carry[kFastMaxW + 128];  // row above the band, column c at index c + 32
};

size_t dec_reconstruct_smem(bool fold16) {
  return (fold16 ? sizeof(WaveSm) : sizeof(RecWarpSmem)) * kWarpsPerCta;
}

template <bool MED, bool STEP1, bool EDGE, int UNROLL, bool SPLIT>
__device__ __forceinline__ void rec_block(RecWarpSmem& sm, const uint16_t* carry_in, uint16_t* carry_out, int lane,
                                          int t0, int W, int32_t maxs, int32_t step, bool band0, int32_t& rec,
                                          int32_t& a_prev) {
  const uint32_t* frow = sm.fold + lane * RecWarpSmem::kFS + (t0 & 32);
  uint16_t* orow = sm.out + lane * kSrcStride + (t0 & 32);
  const uint16_t* crow_in = carry_in + 32 - lane + t0;  // lane 0: column t0 + u
  // one warp per tile reads and writes the same row: one pointer
  uint16_t* crow_out = SPLIT ? carry_out + 32 - lane + t0 : const_cast<uint16_t*>(crow_in);      // lane 31: column t0 + u - 31
#pragma unroll UNROLL
  for (int u = 0; u < 32; ++u) {
    const uint32_t fv = frow[u];
    int32_t a = __shfl_up_sync(0xffffffffu, rec, 1);
    const int32_t above0 = crow_in[u];
    if (lane == 0) a = band0 ? 0 : above0;
    const int32_t pred = MED ? predict_med(rec, a, a_prev) : predict_grad(rec, a, a_prev, maxs);
    const int32_t q = unzigzag(fv);
    int32_t rn = max(0, min(maxs, STEP1 ? pred + q : pred + q * step));
    if (EDGE) {
      const int c = t0 + u - lane;
      if (c < 0) rn = 0;
      if (lane == 31 && c >= 0 && c < W) crow_out[u] = static_cast<uint16_t>(rn);
    } else {
      if (lane == 31) crow_out[u] = static_cast<uint16_t>(rn);
    }
    orow[u] = static_cast<uint16_t>(rn);
    a_prev = a;
    rec = rn;
  }
}

// One warp's sweep of one 32-row band of a tile, block by block: begin()
// stages the first folded chunks, block(k) runs wavefront block k (staging
// the chunk ahead and flushing the reconstruction two chunks behind), end()
// flushes the rest.  Lane 0 reads the row above the band from carry_in;
// lane 31 writes the band's last row to carry_out (one warp per tile: the
// same row, read before it is overwritten).
template <bool MED, bool STEP1, int UNROLL, bool SPLIT>
struct RecBand {
  static constexpr int kFS = RecWarpSmem::kFS;
  RecWarpSmem& sm;
  int lane;
  uint16_t* __restrict__ plane;
  int64_t pitch;
  int W, H, x0, y0;
  int32_t maxs, step;
  int nchunks, nblocks;
  const uint32_t* __restrict__ ftile;
  int band_rows;
  bool band0;
  uint16_t* __restrict__ orows;
  const uint32_t* __restrict__ frows;
  const uint16_t* carry_in;
  uint16_t* carry_out;
  int32_t rec, a_prev;
  uint32_t pf[32];

  __device__ RecBand(const FrameDesc& f, const TileGeo& g, int32_t step_, const uint32_t* ftile_,
                     RecWarpSmem& sm_, int lane_)
      : sm(sm_), lane(lane_), plane(f.dst[g.plane]), pitch(f.dst_pitch[g.plane]), W(g.w), H(g.h), x0(g.x),
        y0(g.y), maxs(f.max_sample), step(step_), nchunks((g.w + 31) >> 5), nblocks((g.w + 31 + 31) >> 5),
        ftile(ftile_) {}

  __device__ void load_chunk(int k) {
    const int col = k * 32 + lane;
    const uint32_t* __restrict__ p = frows + col;
    if (band_rows == 32 && col < W) {
#pragma unroll
      for (int r = 0; r < 32; ++r) pf[r] = ldf(p + static_cast<int64_t>(r) * W);
    } else {
#pragma unroll
      for (int r = 0; r < 32; ++r) pf[r] = (r < band_rows && col < W) ? ldf(p + static_cast<int64_t>(r) * W) : 0u;
    }
  }
  __device__ void store_chunk(int k) {
    const int pj = k * 32 + lane;
#pragma unroll
    for (int r = 0; r < 32; ++r) sm.fold[r * kFS + ((pj + r) & 63)] = pf[r];
  }
  __device__ void flush_chunk(int k) {
    const int col = k * 32 + lane;
    if (col < W) {
      uint16_t* __restrict__ q = orows + col;
      if (band_rows == 32) {
#pragma unroll
        for (int r = 0; r < 32; ++r) q[static_cast<int64_t>(r) * pitch] = sm.out[r * kSrcStride + ((col + r) & 63)];
      } else {
        for (int r = 0; r < band_rows; ++r) q[static_cast<int64_t>(r) * pitch] = sm.out[r * kSrcStride + ((col + r) & 63)];
      }
    }
  }
  __device__ void begin(int band, const uint16_t* cin, uint16_t* cout) {
    band_rows = min(32, H - band * 32);
    band0 = band == 0;
    orows = plane + static_cast<int64_t>(y0 + band * 32) * pitch + x0;
    frows = ftile + static_cast<int64_t>(band * 32) * W;
    carry_in = cin;
    carry_out = cout;
    load_chunk(0);
    store_chunk(0);
    if (nchunks > 1) load_chunk(1);
    __syncwarp();
    rec = 0;
    a_prev = 0;
  }
  __device__ void block(int blk) {
    if (blk > 0) {
      if (blk < nchunks) store_chunk(blk);
      __syncwarp();
      if (blk >= 2 && blk - 2 < nchunks) flush_chunk(blk - 2);
      if (blk + 1 < nchunks) load_chunk(blk + 1);
    }
    const int t0 = blk * 32;
    if (t0 < 31 || t0 + 31 >= W)
      rec_block<MED, STEP1, true, UNROLL, SPLIT>(sm, carry_in, carry_out, lane, t0, W, maxs, step, band0, rec, a_prev);
    else
      rec_block<MED, STEP1, false, UNROLL, SPLIT>(sm, carry_in, carry_out, lane, t0, W, maxs, step, band0, rec, a_prev);
  }
  __device__ void end() {
    __syncwarp();
    for (int j = max(0, nblocks - 2); j < nchunks; ++j) flush_chunk(j);
    __syncwarp();
  }
};

// The two warps of pair p meet at named barrier 1 + p (64 threads).
__device__ __forceinline__ void pair_sync(int pair) {
  asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory");
}

template <bool MED, bool STEP1, int UNROLL, bool PAIRS>
__device__ void rec_tile(const FrameDesc& f, const TileGeo& g, int32_t step, const uint32_t* __restrict__ ftile,
                         RecWarpSmem* smw, int warp, int lane) {
  if constexpr (PAIRS) {
    if (pair_splits(g.w, g.h)) {
      // warp pair: even bands on the first warp, odd bands on the second two
      // blocks behind, in lock-step at the pair barrier after every slot; each
      // warp writes its bands' last rows to its own carry row and reads the
      // other's.  Both warps take the same number of slots (a function of the
      // tile's size only).
      const int pw = warp & 1;
      RecWarpSmem& sm = smw[warp];
      RecBand<MED, STEP1, UNROLL, true> rb(f, g, step, ftile, sm, lane);
      const int n = rb.nblocks, nbands = (g.h + 31) >> 5;
      const int own = pw ? (nbands / 2) * n : ((nbands + 1) / 2) * n;
      const int slots = max(((nbands + 1) / 2) * n, (nbands / 2) * n + 2);
      for (int gs = 0; gs < slots; ++gs) {
        const int sl = gs - 2 * pw;
        if (sl >= 0 && sl < own) {
          const int q = sl / n, blk = sl - q * n;
          if (blk == 0) rb.begin(2 * q + pw, smw[warp ^ 1].carry, sm.carry);
          rb.block(blk);
          if (blk == n - 1) rb.end();
        }
        pair_sync(warp >> 1);
      }
      return;
    }
    if (warp & 1) return;  // too small to split: the pair's first warp alone
  }
  RecWarpSmem& sm = smw[warp];
  RecBand<MED, STEP1, UNROLL, false> rb(f, g, step, ftile, sm, lane);
  for (int band = 0; band * 32 < g.h; ++band) {
    rb.begin(band, sm.carry, sm.carry);
    for (int blk = 0; blk < rb.nblocks; ++blk) rb.block(blk);
    rb.end();
  }
}

// The frames' statuses, final once the entropy decoders are done, by the first
// CTA of the reconstruction.
__device__ __forceinline__ void write_results(const FrameDesc* frames, const FrameState* state, int nframes,
                                              int64_t* results) {
  if (blockIdx.x != 0) return;
  for (int i = threadIdx.x; i < nframes; i += blockDim.x) {
    const int slot = frames[i].slot;
    results[2 * slot] = state[i].status;
    results[2 * slot + 1] = 0;
  }
}

// Tiles come from a queue.  With warp pairs, the pair's first warp claims a
// tile and both read it after the pair barrier (two alternating slots, so a
// claim never overwrites a tile the other warp has yet to read); both then
// make the same decisions from the same tile, so they meet at every barrier.
template <int UNROLL, bool PAIRS>
__global__ void __launch_bounds__(kWarpsPerCta * 32, PAIRS ? 3 : 4)
dec_reconstruct_kernel(const FrameDesc* __restrict__ frames, const FrameState* __restrict__ state,
                       const BatchDims* __restrict__ dims, const uint32_t* __restrict__ folded,
                       int* __restrict__ queue, int64_t* __restrict__ results) {
  static_assert(kWarpsPerCta % 2 == 0, "warp pairs");
  constexpr bool pairs = PAIRS;
  const int nframes = dims->frames_p[0];
  write_results(frames, state, nframes, results);
  const int64_t total_tiles = dims->tiles_p[0];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int64_t claimed[kWarpsPerCta / 2][2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  RecWarpSmem* smw = reinterpret_cast<RecWarpSmem*>(smem_raw);
  for (int it = 0;; ++it) {
    int64_t t = 0;
    if (pairs) {
      if ((warp & 1) == 0 && lane == 0) claimed[warp >> 1][it & 1] = atomicAdd(queue, 1);
      pair_sync(warp >> 1);
      t = claimed[warp >> 1][it & 1];
    } else {
      if (lane == 0) t = atomicAdd(queue, 1);
      t = __shfl_sync(kFull, t, 0);
    }
    if (t >= total_tiles) break;
    const int fi = frame_of_tile(frames, nframes, t);
    const FrameDesc& f = frames[fi];
    if (state[fi].status != 0) continue;
    const TileGeo g = tile_geo(f, t - f.tile_base);
    if (g.w > kFastMaxW) continue;
    const uint32_t* ftile = folded + f.sample_base + g.sample_base;
    if (f.use_med0) {
      if (f.step0 == 1) rec_tile<true, true, UNROLL, PAIRS>(f, g, 1, ftile, smw, warp, lane);
      else rec_tile<true, false, UNROLL, PAIRS>(f, g, f.step0, ftile, smw, warp, lane);
    } else {
      if (f.step0 == 1) rec_tile<false, true, UNROLL, PAIRS>(f, g, 1, ftile, smw, warp, lane);
      else rec_tile<false, false, UNROLL, PAIRS>(f, g, f.step0, ftile, smw, warp, lane);
    }
  }
}

// ---------------------------------------------------------------------------
// dec_reconstruct on u16 symbols (every batch without a lossless 16-bit
// frame): the two-rows-per-lane wavefront of fvb_wave.cuh.  Up to depth 12
// the entropy decoders have already turned symbols into residuals times the
// step (fold_value), so a step is one packed add-clamp after the prediction;
// depth 16 unfolds and scales its symbols here, in 32 bits a row.
//
// Bound by shared-memory latency and issue, about 22 instructions for a step of
// 64 samples (28 for 32 before): 16 4K rgb10 frames 701 -> 414 us (4 bytes a
// sample, 245 us at the copy rate), a 1080p rgb10 frame 80 -> 35 us.

// Eight steps of a window block.
template <bool MED, bool O1>
__device__ __forceinline__ void rec_wave_steps(WavePacked& st, WaveBlock<O1>& blk, int g,
                                               const WaveWords<false>& x, const WaveWords<O1>& y, const WaveCarry& c,
                                               int32_t maxs, int32_t) {
  const uint32_t maxs2 = pair2(maxs);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t dq = wave_pack(x, y, j);
    const uint32_t a = st.neighbours(c.up[j >> 1], j & 1, blk.lane);
    const uint32_t rn = __viaddmin_s16x2_relu(st.template predict<MED>(a, maxs2), dq, maxs2);
    blk.put(g, j, st.rec, rn, st.rec, rn);
    st.above = a;
    st.rec = rn;
  }
}

template <bool MED, bool O1>
__device__ __forceinline__ void rec_wave_steps(WaveWide& st, WaveBlock<O1>& blk, int g,
                                               const WaveWords<false>& x, const WaveWords<O1>& y, const WaveCarry& c,
                                               int32_t maxs, int32_t step) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    int32_t a0, a1;
    st.neighbours(c.up[j >> 1], j & 1, blk.lane, a0, a1);
    const uint32_t was = st.packed();
    const int32_t p0 = st.template predict<MED>(st.rec0, a0, st.above0, maxs);
    const int32_t p1 = st.template predict<MED>(st.rec1, a1, st.above1, maxs);
    st.rec0 = __viaddmin_s32_relu(p0, unzigzag(x.sample(j)) * step, maxs);
    st.rec1 = __viaddmin_s32_relu(p1, unzigzag(y.sample(j)) * step, maxs);
    st.above0 = a0;
    st.above1 = a1;
    const uint32_t rn = st.packed();
    blk.put(g, j, was, rn, was, rn);
  }
}

// One window block: 32 steps in four groups of eight, the next group's words
// loaded before this group's results are stored over theirs.
template <bool MED, bool O1, typename St>
__device__ __forceinline__ void rec_wave_block(St& st, WaveBlock<O1> blk, int32_t maxs, int32_t step) {
  WaveWords<false> x, xn;
  WaveWords<O1> y, yn;
  WaveCarry c, cn;
  x.first(blk.p0);
  y.first(blk.p1);
  x.load(blk.p0, 0);
  y.load(blk.p1, 0);
  c.load(blk.crow, 0);
#pragma unroll 1
  for (int g = 0; g < 4; g += 2) {
    xn.after(x);
    yn.after(y);
    xn.load(blk.p0, g + 1);
    yn.load(blk.p1, g + 1);
    cn.load(blk.crow, g + 1);
    rec_wave_steps<MED>(st, blk, g, x, y, c, maxs, step);
    x.after(xn);
    y.after(yn);
    if (g == 0) {
      x.load(blk.p0, 2);
      y.load(blk.p1, 2);
      c.load(blk.crow, 2);
    }
    rec_wave_steps<MED>(st, blk, g + 1, xn, yn, cn, maxs, step);
  }
  blk.finish(st.packed(), st.packed());
}

// ODD_W: the tile's rows start on even and odd samples in turn
template <bool MED, bool WIDE, bool ODD_W, bool PAIR>
__device__ void rec_wave_tile(const FrameDesc& f, const TileGeo& g, const uint16_t* __restrict__ ftile, WaveSm* sms,
                              int warp, int lane) {
  WaveSm& sm = sms[warp];
  for (int i = lane; i < kCarryCols / 8; i += 32) reinterpret_cast<uint4*>(sm.carry)[i] = make_uint4(0, 0, 0, 0);
  if (PAIR) wave_pair_sync(warp);
  else __syncwarp();
  const uint16_t* above = sms[PAIR ? warp ^ 1 : warp].carry;
  WaveIo<false, !PAIR> io(sm, lane, g.w, ftile, g.w, f.dst[g.plane] + static_cast<int64_t>(g.y) * f.dst_pitch[g.plane] + g.x,
                       f.dst_pitch[g.plane], nullptr, nullptr);
  std::conditional_t<WIDE, WaveWide, WavePacked> st;
  auto begin = [&] {
    st = {};
    io.fetch(0);
  };
  auto block = [&](int b) {
    if (b) {
      io.flush(b - 1);
      io.move_head(b);
      __syncwarp();
    }
    if (b + 1 < io.nblk) io.fetch(b + 1);
    else cp_async_commit();
    io.wait();
    io.template fix_edge<false>(b);
    rec_wave_block<MED, !ODD_W>(st, WaveBlock<!ODD_W>(sm, above, b, lane, io.off0, io.off1), f.max_sample, f.step0);
    __syncwarp();
  };
  auto end = [&] {
    io.flush_last();
    __syncwarp();
  };
  wave_sweep<PAIR>(io, g.h, warp, begin, block, end);
}

template <bool PAIR>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4)
dec_reconstruct_wave_kernel(const FrameDesc* __restrict__ frames, const FrameState* __restrict__ state,
                            const BatchDims* __restrict__ dims, const uint16_t* __restrict__ folded,
                            int* __restrict__ queue, int64_t* __restrict__ results) {
  const int nframes = dims->frames_p[0];
  write_results(frames, state, nframes, results);
  const int64_t total_tiles = dims->tiles_p[0];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WaveSm* sms = reinterpret_cast<WaveSm*>(smem_raw);
  // a warp's (a pair's) first tile goes by its place -- the first warps of all
  // CTAs before the second ones, so few tiles spread over all SMs -- and the
  // rest come from the queue (for pairs there are none, or by place too)
  const int64_t takers = static_cast<int64_t>(gridDim.x) * (PAIR ? kWarpsPerCta / 2 : kWarpsPerCta);
  for (int64_t t = static_cast<int64_t>(PAIR ? warp >> 1 : warp) * gridDim.x + blockIdx.x; t < total_tiles;) {
    const int64_t mine = t;
    if (PAIR) {
      t += takers;
    } else {
      if (lane == 0) t = takers + atomicAdd(queue, 1);
      t = __shfl_sync(kFull, t, 0);
    }
    const int fi = frame_of_tile(frames, nframes, mine);
    const FrameDesc& f = frames[fi];
    if (state[fi].status != 0) continue;
    const TileGeo g = tile_geo(f, mine - f.tile_base);
    if (g.w > kFastMaxW) continue;
    const uint16_t* ftile = folded + f.sample_base + g.sample_base;
    const bool odd = g.w & 1, wide = f.bit_depth > 12;
    if (f.use_med0) {
      if (!wide) odd ? rec_wave_tile<true, false, true, PAIR>(f, g, ftile, sms, warp, lane)
                     : rec_wave_tile<true, false, false, PAIR>(f, g, ftile, sms, warp, lane);
      else odd ? rec_wave_tile<true, true, true, PAIR>(f, g, ftile, sms, warp, lane)
               : rec_wave_tile<true, true, false, PAIR>(f, g, ftile, sms, warp, lane);
    } else {
      if (!wide) odd ? rec_wave_tile<false, false, true, PAIR>(f, g, ftile, sms, warp, lane)
                     : rec_wave_tile<false, false, false, PAIR>(f, g, ftile, sms, warp, lane);
      else odd ? rec_wave_tile<false, true, true, PAIR>(f, g, ftile, sms, warp, lane)
               : rec_wave_tile<false, true, false, PAIR>(f, g, ftile, sms, warp, lane);
    }
  }
}

// The wavefront block of the u32 dec_reconstruct is a launch-time choice (4,
// 8, 16 or 32 steps unrolled; identical planes), as are its warps per tile.
cudaError_t dec_reconstruct_set_smem() {
  const int b32 = static_cast<int>(dec_reconstruct_smem(false)), b16 = static_cast<int>(dec_reconstruct_smem(true));
  for (auto k : {dec_reconstruct_kernel<4, false>, dec_reconstruct_kernel<8, false>,
                 dec_reconstruct_kernel<16, false>, dec_reconstruct_kernel<32, false>,
                 dec_reconstruct_kernel<8, true>}) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, b32);
    if (e != cudaSuccess) return e;
  }
  for (auto k : {dec_reconstruct_wave_kernel<false>, dec_reconstruct_wave_kernel<true>}) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, b16);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

void dec_reconstruct_launch(int unroll, int tile_warps, bool fold16, bool pairs, int grid, cudaStream_t stream,
                            const FrameDesc* frames, const FrameState* state, const BatchDims* dims,
                            const void* folded, int* queue, int64_t* results) {
  if (fold16) {
    auto k = pairs ? dec_reconstruct_wave_kernel<true> : dec_reconstruct_wave_kernel<false>;
    k<<<grid, kWarpsPerCta * 32, dec_reconstruct_smem(true), stream>>>(
        frames, state, dims, static_cast<const uint16_t*>(folded), queue, results);
    return;
  }
  // warp pairs run with the default wavefront block
  auto k = tile_warps == 2 ? dec_reconstruct_kernel<8, true>
           : unroll == 4   ? dec_reconstruct_kernel<4, false>
           : unroll == 16  ? dec_reconstruct_kernel<16, false>
           : unroll == 32  ? dec_reconstruct_kernel<32, false>
                           : dec_reconstruct_kernel<8, false>;
  k<<<grid, kWarpsPerCta * 32, dec_reconstruct_smem(false), stream>>>(
      frames, state, dims, static_cast<const uint32_t*>(folded), queue, results);
}

void dec_rans_launch(bool fold16, bool few, bool roomy, int grid, cudaStream_t stream, const FrameDesc* frames,
                     FrameState* state, const ShardInfo* shards, DecodeLists* lists, const int32_t* list_items,
                     const RansTable* tables, void* folded) {
  const int threads = few ? 32 : kWarpsPerCta * 32;
  const size_t smem = few ? dec_rans_slots_smem() : roomy ? dec_rans_smem<true>() : dec_rans_smem<false>();
  if (fold16) {
    auto k = few     ? dec_rans_slots_kernel<uint16_t>
             : roomy ? dec_rans_kernel<uint16_t, true>
                     : dec_rans_kernel<uint16_t, false>;
    k<<<grid, threads, smem, stream>>>(frames, state, shards, lists, list_items, tables,
                                       static_cast<uint16_t*>(folded));
  } else {
    auto k = few     ? dec_rans_slots_kernel<uint32_t>
             : roomy ? dec_rans_kernel<uint32_t, true>
                     : dec_rans_kernel<uint32_t, false>;
    k<<<grid, threads, smem, stream>>>(frames, state, shards, lists, list_items, tables,
                                       static_cast<uint32_t*>(folded));
  }
}

cudaError_t dec_rans_set_smem() {
  const int b = static_cast<int>(dec_rans_smem<false>()), br = static_cast<int>(dec_rans_smem<true>()),
            bs = static_cast<int>(dec_rans_slots_smem());
  auto set = [](auto k, int bytes) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e != cudaSuccess ? e
                            : cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                                   cudaSharedmemCarveoutMaxShared);
  };
  cudaError_t e = set(dec_rans_kernel<uint16_t, false>, b);
  if (e == cudaSuccess) e = set(dec_rans_kernel<uint32_t, false>, b);
  if (e == cudaSuccess) e = set(dec_rans_kernel<uint16_t, true>, br);
  if (e == cudaSuccess) e = set(dec_rans_kernel<uint32_t, true>, br);
  if (e == cudaSuccess) e = set(dec_rans_slots_kernel<uint16_t>, bs);
  if (e == cudaSuccess) e = set(dec_rans_slots_kernel<uint32_t>, bs);
  return e;
}

// Every kernel of the decode asks for the same split of the L1/shared array as
// dec_rans: an SM changes its split only when it is empty, so with another
// split dec_other could not join dec_rans on an SM (a 1080p rgb10 frame took
// 350 us instead of 307).
cudaError_t dec_other_set_smem() {
  cudaError_t e = cudaFuncSetAttribute(dec_other_kernel<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(dec_other_smem(true)));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(dec_other_kernel<uint32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(dec_other_smem(false)));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(dec_other_kernel<uint16_t>, cudaFuncAttributePreferredSharedMemoryCarveout,
                           cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(dec_other_kernel<uint32_t>, cudaFuncAttributePreferredSharedMemoryCarveout,
                              cudaSharedmemCarveoutMaxShared);
}

void dec_other_launch(bool fold16, int grid, cudaStream_t stream, const FrameDesc* frames, FrameState* state,
                      const ShardInfo* shards, const BatchDims* dims, DecodeLists* lists, const int32_t* list_items,
                      void* folded) {
  if (fold16)
    dec_other_kernel<uint16_t><<<grid, 32 * kOtherWarps, dec_other_smem(true), stream>>>(frames, state, shards, dims, lists, list_items,
                                                         static_cast<uint16_t*>(folded));
  else
    dec_other_kernel<uint32_t><<<grid, 32 * kOtherWarps, dec_other_smem(false), stream>>>(frames, state, shards, dims, lists, list_items,
                                                         static_cast<uint32_t*>(folded));
}

// Wide tiles: antidiagonal order with neighbours read back from the output
// plane (decode.cu:572-605).
__global__ void dec_reconstruct_wide_kernel(const FrameDesc* __restrict__ frames, const FrameState* __restrict__ state,
                                            const BatchDims* __restrict__ dims, const void* __restrict__ folded,
                                            int fold16) {
  const int nframes = dims->frames_p[0];
  const int64_t total_tiles = dims->tiles_p[0];
  for (int64_t t = blockIdx.x; t < total_tiles; t += gridDim.x) {
    const int fi = frame_of_tile(frames, nframes, t);
    const FrameDesc& f = frames[fi];
    if (state[fi].status != 0) continue;
    const TileGeo g = tile_geo(f, t - f.tile_base);
    if (g.w <= kFastMaxW) continue;
    uint16_t* plane = f.dst[g.plane];
    const int64_t pitch = f.dst_pitch[g.plane];
    const int64_t fbase = f.sample_base + g.sample_base;
    const int32_t maxs = f.max_sample;
    const bool med = f.use_med0 != 0;
    const Deltas deltas(f, folded, fold16);
    for (int d = 0; d < g.w + g.h - 1; ++d) {
      const int y0 = max(0, d - g.w + 1), y1 = min(d, g.h - 1);
      for (int y = y0 + threadIdx.x; y <= y1; y += blockDim.x) {
        const int x = d - y;
        uint16_t* o = plane + static_cast<int64_t>(g.y + y) * pitch + g.x + x;
        const int32_t dq = deltas[fbase + static_cast<int64_t>(y) * g.w + x];
        const int32_t l = x > 0 ? o[-1] : 0;
        const int32_t a = y > 0 ? o[-pitch] : 0;
        const int32_t ul = (x > 0 && y > 0) ? o[-pitch - 1] : 0;
        const int32_t pred = med ? predict_med(l, a, ul) : predict_grad(l, a, ul, maxs);
        *o = static_cast<uint16_t>(max(0, min(maxs, pred + dq)));
      }
      __syncthreads();
    }
  }
}

// predictor="serial": one thread per tile in raster order (decode.cu:608-656).
__global__ void dec_reconstruct_serial_kernel(const FrameDesc* __restrict__ frames, const FrameState* __restrict__ state,
                                              const BatchDims* __restrict__ dims, const void* __restrict__ folded,
                                              int fold16, int64_t* __restrict__ results) {
  const int nframes = dims->frames_p[0];
  write_results(frames, state, nframes, results);
  const int64_t total_tiles = dims->tiles_p[0];
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= total_tiles) return;
  const int fi = frame_of_tile(frames, nframes, t);
  const FrameDesc& f = frames[fi];
  if (state[fi].status != 0) return;
  const TileGeo g = tile_geo(f, t - f.tile_base);
  uint16_t* plane = f.dst[g.plane];
  const int64_t pitch = f.dst_pitch[g.plane];
  const int64_t fbase = f.sample_base + g.sample_base;
  const int32_t maxs = f.max_sample;
  const bool med = f.use_med0 != 0;
  const Deltas deltas(f, folded, fold16);
  for (int y = 0; y < g.h; ++y) {
    int32_t left = 0, ul = 0;
    uint16_t* orow = plane + static_cast<int64_t>(g.y + y) * pitch + g.x;
    const int64_t frow = fbase + static_cast<int64_t>(y) * g.w;
    for (int x = 0; x < g.w; ++x) {
      const int32_t a = y > 0 ? orow[x - pitch] : 0;
      const int32_t pred = med ? predict_med(left, a, ul) : predict_grad(left, a, ul, maxs);
      const int32_t r = max(0, min(maxs, pred + deltas[frow + x]));
      orow[x] = static_cast<uint16_t>(r);
      ul = a;
      left = r;
    }
  }
}

}  // namespace fvb
