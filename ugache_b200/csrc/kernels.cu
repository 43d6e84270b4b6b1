// sm_100a kernels of the extraction path.  Everything here is integer index arithmetic
// and raw byte copies; rows move as 16- or 32-byte vectors (4-byte words when a row size
// is not a multiple of 16).
#include "kernels.cuh"

#include <algorithm>
#include <cstring>
#include <type_traits>

namespace ugc {

namespace {

constexpr int kBlock = 256;          // threads per CTA everywhere
constexpr int kWarpsPerBlock = kBlock / 32;
constexpr unsigned kFull = 0xffffffffu;

// ------------------------------------------------------------------------------------
// memory access helpers
// ------------------------------------------------------------------------------------

template <int BYTES>
struct Vec;
template <>
struct Vec<4> {
  uint32_t v[1];
};
template <>
struct __align__(16) Vec<16> {
  uint32_t v[4];
};
template <>
struct __align__(32) Vec<32> {
  uint32_t v[8];
};

// Row payload loads: read-only path, allocating in L1.  Under a Zipf key distribution a few
// rows make up a large share of every batch (the hottest row alone is 18 % of the keys at
// alpha 1.2, 32 % at 1.4); without L1 allocation all of those reads queue at the few L2 slices
// that hold the row, which cost 20-25 % of the step (42 -> 31 us at alpha 1.4, measured).
#define UGC_LD_ROW "ld.global.nc"
__device__ __forceinline__ void ld_row(Vec<4>& r, const void* p) {
  asm volatile(UGC_LD_ROW ".b32 %0, [%1];" : "=r"(r.v[0]) : "l"(p));
}
__device__ __forceinline__ void ld_row(Vec<16>& r, const void* p) {
  asm volatile(UGC_LD_ROW ".v4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3])
               : "l"(p));
}
__device__ __forceinline__ void ld_row(Vec<32>& r, const void* p) {
  asm volatile(UGC_LD_ROW ".v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]),
                 "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
               : "l"(p));
}
// Output stores: streaming (evict-first) so the written rows do not push hot cache rows
// out of L2.
__device__ __forceinline__ void st_row(void* p, const Vec<4>& r) {
  asm volatile("st.global.cs.b32 [%0], %1;" ::"l"(p), "r"(r.v[0]) : "memory");
}
__device__ __forceinline__ void st_row(void* p, const Vec<16>& r) {
  asm volatile("st.global.cs.v4.b32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(r.v[0]), "r"(r.v[1]),
               "r"(r.v[2]), "r"(r.v[3])
               : "memory");
}
__device__ __forceinline__ void st_row(void* p, const Vec<32>& r) {
  asm volatile("st.global.cs.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r.v[0]),
               "r"(r.v[1]), "r"(r.v[2]), "r"(r.v[3]), "r"(r.v[4]), "r"(r.v[5]), "r"(r.v[6]),
               "r"(r.v[7])
               : "memory");
}
// Plain (write-back) store used when the destination is the cache slice itself.
__device__ __forceinline__ void st_keep(void* p, const Vec<4>& r) {
  *reinterpret_cast<uint32_t*>(p) = r.v[0];
}
__device__ __forceinline__ void st_keep(void* p, const Vec<16>& r) {
  *reinterpret_cast<uint4*>(p) = make_uint4(r.v[0], r.v[1], r.v[2], r.v[3]);
}
__device__ __forceinline__ void st_keep(void* p, const Vec<32>& r) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r.v[0]),
               "r"(r.v[1]), "r"(r.v[2]), "r"(r.v[3]), "r"(r.v[4]), "r"(r.v[5]), "r"(r.v[6]),
               "r"(r.v[7])
               : "memory");
}

// One 32-byte table line = 4 slots {key, word}.  Coherent load (a refresh may be
// inserting or evicting while lookups run), L2 only.
struct Line {
  uint32_t key[kSlotsPerLine];
  uint32_t word[kSlotsPerLine];
};
__device__ __forceinline__ Line ld_line(const uint2* slots, uint32_t line) {
  Line l;
  const uint2* p = slots + (size_t)line * kSlotsPerLine;
  asm volatile("ld.global.cg.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(l.key[0]), "=r"(l.word[0]), "=r"(l.key[1]), "=r"(l.word[1]),
                 "=r"(l.key[2]), "=r"(l.word[2]), "=r"(l.key[3]), "=r"(l.word[3])
               : "l"(p));
  return l;
}

// MurmurHash3_32 of one 32-bit key, seed 0: the hash of the reference's probing table
// (coll_cache_lib/cuda/cache_hashtable.cuh:56-135); here it picks the first line.
__host__ __device__ __forceinline__ uint32_t murmur3_32(uint32_t key) {
  uint32_t k1 = key * 0xcc9e2d51u;
  k1 = (k1 << 15) | (k1 >> 17);
  k1 *= 0x1b873593u;
  uint32_t h1 = k1;
  h1 = (h1 << 13) | (h1 >> 19);
  h1 = h1 * 5u + 0xe6546b64u;
  h1 ^= 4u;
  h1 ^= h1 >> 16;
  h1 *= 0x85ebca6bu;
  h1 ^= h1 >> 13;
  h1 *= 0xc2b2ae35u;
  h1 ^= h1 >> 16;
  return h1;
}

// Result of inspecting one line for `key`: the word if a live slot matches, else whether
// the search may stop (a never-used slot was seen).
__device__ __forceinline__ bool line_find(const Line& l, uint32_t key, uint32_t& word, bool& stop) {
  stop = false;
#pragma unroll
  for (int s = 0; s < kSlotsPerLine; s++) {
    if (l.key[s] == key) {  // live slots carry the key with the top bit clear
      word = l.word[s];
      return true;
    }
  }
#pragma unroll
  for (int s = 0; s < kSlotsPerLine; s++) stop |= (l.key[s] == kEmptyWord);
  return false;
}

// Probes after the first line (already loaded by the caller).  Bounded by the table size.
__device__ __forceinline__ uint32_t probe_rest(const uint2* slots, uint32_t line_mask, uint32_t key,
                                            uint32_t line) {
  for (uint32_t step = 0; step < line_mask; step++) {
    line = (line + 1) & line_mask;
    Line l = ld_line(slots, line);
    uint32_t w;
    bool stop;
    if (line_find(l, key, w, stop)) return w;
    if (stop) return kEmptyWord;
  }
  return kEmptyWord;
}

__device__ __forceinline__ uint32_t table_lookup(const TableView& t, uint32_t key) {
  if (t.kind == kTableFlat) {
    uint32_t w;
    asm volatile("ld.global.cg.b32 %0, [%1];" : "=r"(w) : "l"(t.flat + key));
    return w;
  }
  uint32_t line = murmur3_32(key) & t.line_mask;
  Line l = ld_line(t.slots, line);
  uint32_t w;
  bool stop;
  if (line_find(l, key, w, stop)) return w;
  if (stop) return kEmptyWord;
  return probe_rest(t.slots, t.line_mask, key, line);
}

// Keys: read once, and past the L1, which other launches of the stream overlap with.  Volatile, so that
// they stay on their side of the dependency wait.
__device__ __forceinline__ uint64_t ld_key(const uint32_t* p) {
  uint32_t k;
  asm volatile("ld.global.cg.b32 %0, [%1];" : "=r"(k) : "l"(p) : "memory");
  return k;
}
__device__ __forceinline__ uint64_t ld_key(const long long* p) {
  uint64_t k;
  asm volatile("ld.global.cg.b64 %0, [%1];" : "=l"(k) : "l"(p) : "memory");
  return k;
}

// Extractions that run, by stream: CTA i < kRunMarks puts the extraction's ordinal into mark i once it is
// past its dependency wait and takes it out when it ends (the grouped gather: mark 0, for the whole grid).
__device__ __align__(128) uint32_t g_running[kRunSlots][kRunMarks];

// Whether the extraction ahead still runs.  Only then may a launch read keys, table and rows ahead of its
// dependency wait: it has nothing but that extraction to wait for.  All that came before is complete, since
// the extraction was past its own wait; no ordinary kernel or copy stands in between, which would have
// waited for the extraction's end; and the library's other kernels let the next launch start no earlier
// than behind their wait.  What the extraction ahead writes itself, its rows, the host keeps apart
// (order_in_stream).  Without this proof a launch waits first.  Waiting first always costs 13,312 keys back
// to back 2.0 us of 6.5, and 212,992 keys with 7,277 host rows 15 of 102.  The marks are read once a CTA, and
// no more of them than in use: the same line read by every warp cost 500,009 keys 5 to 10 us of 164, 128 marks
// a CTA 3.  With 8 marks of a direct extraction instead of 128 its last CTAs, which wait for host rows, were
// missed (100 M x 512-byte rows, 3,217 host rows: 89.4 us, with 128 87.7).  All threads of the CTA take part.
__device__ __forceinline__ bool still_running(const StreamOrder& o) {
  if (o.ahead == 0) return false;
  uint32_t mark = 0;
  if (threadIdx.x < o.marks)
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(mark) : "l"(&g_running[o.slot][threadIdx.x]) : "memory");
  return __syncthreads_or(mark == o.ahead);
}
__device__ __forceinline__ void set_running(const StreamOrder& o, uint32_t mark) {
  if (o.seq) *const_cast<volatile uint32_t*>(&g_running[o.slot][mark]) = o.seq;
}
__device__ __forceinline__ void clear_running(const StreamOrder& o, uint32_t mark) {
  if (o.seq) asm volatile("red.relaxed.gpu.global.and.b32 [%0], %1;" ::"l"(&g_running[o.slot][mark]), "r"(0u) : "memory");
}

// Address range of a host row, for the ordering of the host list.
constexpr int kHostBuckets = 4096;
__device__ __forceinline__ uint32_t host_bucket(uint32_t off, uint32_t shift) {
  return min(off >> shift, (uint32_t)kHostBuckets - 1);
}

// ------------------------------------------------------------------------------------
// lookup + group by source
// ------------------------------------------------------------------------------------
// What bounds it is latency and, with one key per thread, the three list counters, which sit in one
// sector of the L2 and take one addition every 0.6 ns: 6,656 CTAs x 3 of them were half of the 38 us
// a batch of 1.7 M keys took.  Four keys a thread make a quarter of the CTAs.
template <typename KeyT, int kKeysPerThread>
__global__ void __launch_bounds__(kBlock)
    lookup_group_kernel(const KeyT* __restrict__ keys, uint32_t n, TableView t, uint32_t local_loc,
                        uint32_t host_loc, uint32_t host_mask, uint64_t* __restrict__ list_local,
                        uint64_t* __restrict__ list_remote, uint64_t* __restrict__ list_host,
                        Counters* counters, StreamOrder order, uint32_t* host_hist, uint32_t hist_shift) {
  __shared__ uint32_t s_cnt[kWarpsPerBlock][kKeysPerThread][kNumGroup];
  __shared__ uint32_t s_base[kNumGroup];

  const uint32_t tid = threadIdx.x;
  const uint32_t warp = tid >> 5, lane = tid & 31;
  const uint32_t tile_base = blockIdx.x * (kBlock * kKeysPerThread);
  unsigned long long t_begin = 0;
  if (blockIdx.x == 0 && tid == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_begin));

  if (!still_running(order)) asm volatile("griddepcontrol.wait;" ::: "memory");
  uint32_t key[kKeysPerThread];
  bool valid[kKeysPerThread];
  uint32_t bad = 0;
#pragma unroll
  for (int j = 0; j < kKeysPerThread; j++) {
    uint32_t idx = tile_base + j * kBlock + tid;
    valid[j] = idx < n;
    uint64_t k = valid[j] ? ld_key(keys + idx) : 0;
    if (k >= t.num_keys) {  // also catches negative int64 ids
      valid[j] = false;
      bad++;
      k = 0;
    }
    key[j] = (uint32_t)k;
  }
  // Let the gather that follows in the stream be scheduled as soon as SM resources allow
  // (it waits for this grid's completion before it reads the lists).
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // First probe of every key is issued before any is consumed.
  uint32_t word[kKeysPerThread];
  if (t.kind == kTableFlat) {
#pragma unroll
    for (int j = 0; j < kKeysPerThread; j++) {
      word[j] = kEmptyWord;
      if (valid[j]) asm volatile("ld.global.cg.b32 %0, [%1];" : "=r"(word[j]) : "l"(t.flat + key[j]));
    }
  } else {
    Line first[kKeysPerThread];
    uint32_t line[kKeysPerThread];
#pragma unroll
    for (int j = 0; j < kKeysPerThread; j++) {
      line[j] = murmur3_32(key[j]) & t.line_mask;
      first[j] = ld_line(t.slots, line[j]);
    }
#pragma unroll
    for (int j = 0; j < kKeysPerThread; j++) {
      uint32_t w;
      bool stop;
      if (line_find(first[j], key[j], w, stop)) {
        word[j] = w;
      } else if (stop) {
        word[j] = kEmptyWord;
      } else {
        word[j] = probe_rest(t.slots, t.line_mask, key[j], line[j]);
      }
    }
  }

  // Everything below touches the lists and counters that the previous lookup's gather may still
  // be using: wait for it (no-op unless this kernel was launched with programmatic stream
  // serialization, and if it has waited already).
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (bad) atomicAdd(&counters->err_key_range, (unsigned long long)bad);
  if (blockIdx.x == 0 && tid < kNumGroup) counters->t_end[tid] = 0;  // re-armed for the gather's timestamps
  if (blockIdx.x == 0 && tid == 0) counters->t_index = t_begin;

  // Group, count per warp with ballots.
  uint32_t group[kKeysPerThread], rank_in_warp[kKeysPerThread];
  uint64_t rec[kKeysPerThread];
#pragma unroll
  for (int j = 0; j < kKeysPerThread; j++) {
    uint32_t idx = tile_base + j * kBlock + tid;
    uint32_t loc, off;
    if (word[j] == kEmptyWord) {
      loc = host_loc;
      off = key[j] & host_mask;
      group[j] = kGroupHost;
    } else {
      loc = word_loc(word[j]);
      off = word_off(word[j]);
      group[j] = (loc == local_loc) ? kGroupLocal : kGroupRemote;
    }
    if (!valid[j]) group[j] = kNumGroup;
    // address range of a host row, counted for the ordering of the host list (below)
    if (host_hist != nullptr && group[j] == (uint32_t)kGroupHost)
      atomicAdd(&host_hist[host_bucket(off, hist_shift)], 1u);
    rec[j] = make_record(idx, loc, off);
    rank_in_warp[j] = 0;
#pragma unroll
    for (int g = 0; g < kNumGroup; g++) {
      unsigned m = __ballot_sync(kFull, group[j] == (uint32_t)g);
      if (group[j] == (uint32_t)g) rank_in_warp[j] = __popc(m & ((1u << lane) - 1));
      if (lane == 0) s_cnt[warp][j][g] = __popc(m);
    }
  }
  __syncthreads();
  // Exclusive scan of the 8x4 per-warp counts of each group (one thread per group), then
  // one global atomic per (CTA, group).
  if (tid < kNumGroup) {
    uint32_t run = 0;
    for (int j = 0; j < kKeysPerThread; j++)
      for (int w = 0; w < kWarpsPerBlock; w++) {
        uint32_t c = s_cnt[w][j][tid];
        s_cnt[w][j][tid] = run;
        run += c;
      }
    s_base[tid] = run ? atomicAdd(&counters->count[tid], run) : 0;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kKeysPerThread; j++) {
    if (group[j] == kNumGroup) continue;
    uint32_t pos = s_base[group[j]] + s_cnt[warp][j][group[j]] + rank_in_warp[j];
    uint64_t* dst = group[j] == kGroupLocal ? list_local
                                             : (group[j] == kGroupRemote ? list_remote : list_host);
    dst[pos] = rec[j];
  }
}

// ------------------------------------------------------------------------------------
// row copy core: a "worker" is a group of LPR lanes that copies one row at a time,
// UNROLL rows in flight per worker.
// ------------------------------------------------------------------------------------
struct RecordIndex {  // rows described by 64-bit records
  const uint64_t* list;
  const void* const* src_base;  // per location
  char* out;
  uint32_t row_bytes;
  __device__ __forceinline__ void get(uint32_t i, const char*& src, char*& dst) const {
    uint64_t r = list[i];
    src = static_cast<const char*>(src_base[rec_loc(r)]) + (size_t)rec_off(r) * row_bytes;
    dst = out + (size_t)rec_dst(r) * row_bytes;
  }
};
struct KeySlotIndex {  // fill: host row of a key -> cache slot
  const uint32_t* keys;
  SlotView slots;
  uint32_t host_mask;
  const char* host;
  char* slice;
  uint32_t row_bytes;
  __device__ __forceinline__ void get(uint32_t i, const char*& src, char*& dst) const {
    uint32_t k = keys[i] & host_mask;
    uint32_t s = slots.data ? slots.data[slot_pos(slots, i)] : slots.base + i;
    src = host + (size_t)k * row_bytes;
    dst = slice + (size_t)s * row_bytes;
  }
};

template <int VEC, int LPR, int UNROLL, bool STREAM_OUT, typename Index>
__device__ __forceinline__ void copy_rows(const Index& ix, uint32_t count, uint32_t worker,
                                          uint32_t n_workers, uint32_t sublane,
                                          uint32_t vecs_per_row) {
  for (uint32_t base = worker; base < count; base += n_workers * UNROLL) {
    const char* src[UNROLL];
    char* dst[UNROLL];
    bool ok[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      uint32_t i = base + u * n_workers;
      ok[u] = i < count;
      src[u] = nullptr;
      dst[u] = nullptr;
      if (ok[u]) ix.get(i, src[u], dst[u]);
    }
    for (uint32_t c = sublane; c < vecs_per_row; c += LPR) {
      Vec<VEC> v[UNROLL];
#pragma unroll
      for (int u = 0; u < UNROLL; u++)
        if (ok[u]) ld_row(v[u], src[u] + (size_t)c * VEC);
#pragma unroll
      for (int u = 0; u < UNROLL; u++)
        if (ok[u]) {
          if (STREAM_OUT) {
            st_row(dst[u] + (size_t)c * VEC, v[u]);
          } else {
            st_keep(dst[u] + (size_t)c * VEC, v[u]);
          }
        }
    }
  }
}

// ------------------------------------------------------------------------------------
// role-partitioned gather
// ------------------------------------------------------------------------------------
__device__ __forceinline__ int ceil_div_i(uint32_t a, uint32_t b) { return (int)((a + b - 1) / b); }

// Splits the grid (>= 3 CTAs) into host / remote / local groups from the device-resident
// counts.  CTAs [0, n_host) serve host rows, [n_host, n_host+n_remote) peer rows, the rest
// local rows: the long-latency sources get the lowest block indices, which start first.
// A group's share of the CTAs follows the time its bytes need on its link (bytes / bandwidth,
// the rule the reference's link tables encode as SM counts per link,
// coll_cache_lib/coll_cache/asymm_link_desc.cc:247-289), limited by what keeps that link full
// (the caps) and by the rows there are.  A non-empty group always gets at least one CTA.
__device__ __forceinline__ void split_roles(const GatherParams& p, const uint32_t cnt[kNumGroup],
                                            int grid, int& n_host, int& n_remote) {
  const uint32_t rmin = (uint32_t)p.rows_per_cta_min;
  const float t_loc = (float)cnt[kGroupLocal] * 2.0f * p.t_byte[kGroupLocal];
  const float t_rem = (float)cnt[kGroupRemote] * p.t_byte[kGroupRemote];
  const float t_host = (float)cnt[kGroupHost] * p.t_byte[kGroupHost];
  const float t_all = t_loc + t_rem + t_host;
  auto share = [&](float t, uint32_t c, int cap) -> int {
    if (c == 0) return 0;
    int n = t_all > 0.f ? (int)ceilf((float)grid * t / t_all) : cap;
    n = min(n, min(cap, ceil_div_i(c, rmin)));
    return max(n, 1);
  };
  n_host = share(t_host, cnt[kGroupHost], p.host_cta_cap);
  // an ordered host list is worked by a set number of CTAs: with more, the rows in flight spread
  // over more of the table than the order is worth (unless no row is local: then all CTAs work it)
  if (p.host_hist && cnt[kGroupHost]) n_host = max(1, min(p.host_cta_cap, ceil_div_i(cnt[kGroupHost], rmin)));
  n_remote = share(t_rem, cnt[kGroupRemote], p.remote_cta_cap);
  if (p.fixed_split) {
    n_host = cnt[kGroupHost] ? max(p.host_cta_cap, 1) : 0;
    n_remote = cnt[kGroupRemote] ? max(p.remote_cta_cap, 1) : 0;
  }
  const int avail = grid - (cnt[kGroupLocal] ? 1 : 0);
  while (n_host + n_remote > avail) {  // small grids only
    if (n_remote >= n_host && n_remote > 1) {
      n_remote--;
    } else if (n_host > 1) {
      n_host--;
    } else {
      n_remote--;
    }
  }
  if (cnt[kGroupLocal] == 0) {  // nothing local: the spare CTAs help the other groups
    if (cnt[kGroupRemote]) {
      n_remote = grid - n_host;
    } else if (cnt[kGroupHost]) {
      n_host = grid;
    }
  }
}

// ---- bulk-async (TMA engine) staging of rows whose source is far away -------------------
// One elected lane per warp moves whole rows: cp.async.bulk global -> shared with an mbarrier
// counting the bytes, then cp.async.bulk shared -> global.  The copy engine keeps many rows
// in flight without holding registers or load-queue slots of the SM.  No cluster, no
// multicast; source may be pinned host memory or a peer GPU's memory.
constexpr int kBulkSlots = 8;          // rows in flight per warp
constexpr uint32_t kBulkSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst_smem, const void* src, uint32_t bytes,
                                         uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst_smem),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void bulk_s2g(void* dst, uint32_t src_smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"(src_smem), "r"(bytes)
               : "memory");
}

// Rows [worker, worker + n_workers, ...) of the list, one warp per worker, lane 0 drives.
// Returns false if a wait ran out (the caller records it; the kernel still terminates).
__device__ __forceinline__ bool copy_rows_bulk(const RecordIndex& ix, uint32_t count,
                                               uint32_t worker, uint32_t n_workers,
                                               unsigned char* stage, uint64_t* bars) {
  const uint32_t lane = threadIdx.x & 31;
  bool ok_all = true;
  if (lane == 0) {
    uint32_t parity = 0;
    for (int u = 0; u < kBulkSlots; u++) mbar_init(smem_u32(&bars[u]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (uint32_t base = worker; base < count; base += n_workers * kBulkSlots) {
      char* dst[kBulkSlots];
      bool ok[kBulkSlots];
#pragma unroll
      for (int u = 0; u < kBulkSlots; u++) {
        uint32_t i = base + u * n_workers;
        ok[u] = i < count;
        dst[u] = nullptr;
        if (ok[u]) {
          const char* src;
          ix.get(i, src, dst[u]);
          uint32_t bar = smem_u32(&bars[u]);
          mbar_expect_tx(bar, ix.row_bytes);
          bulk_g2s(smem_u32(stage + (size_t)u * ix.row_bytes), src, ix.row_bytes, bar);
        }
      }
#pragma unroll
      for (int u = 0; u < kBulkSlots; u++) {
        if (!ok[u]) continue;
        uint32_t bar = smem_u32(&bars[u]);
        uint32_t spins = 0;
        while (!mbar_try_wait(bar, parity)) {
          if (++spins > kBulkSpinLimit) {
            ok_all = false;
            break;
          }
        }
        if (!ok_all) break;
        bulk_s2g(dst[u], smem_u32(stage + (size_t)u * ix.row_bytes), ix.row_bytes);
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      // the slots are reused by the next pass: wait until the stores have read them
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      if (!ok_all) break;
      parity ^= 1;
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  __syncwarp();
  return ok_all;
}

// Counts of the lookup that just finished, into the pinned host mirror: one 16-byte store, and only
// when they differ from what the mirror shows by more than a sixteenth (the host compares them with
// thresholds).  A store that crosses PCIe, or the fence that five single words needed between them,
// holds the end of the launch back: 2 us of the 6.6 that 208 keys took.
__device__ __forceinline__ void publish_feedback(Feedback* f, Counters* c, const uint32_t cnt[kNumGroup],
                                                 uint32_t seq) {
  if (f == nullptr) return;
  uint32_t* shown = c->shown;
  bool same = shown[kNumGroup] != 0;
#pragma unroll
  for (int g = 0; g < kNumGroup; g++) {
    const uint32_t was = shown[g];
    same = same && (cnt[g] > was ? cnt[g] - was : was - cnt[g]) <= (was >> 4);
  }
  if (same) return;
  const uint4 v = make_uint4(cnt[0], cnt[1], cnt[2], seq);
  *reinterpret_cast<uint4*>(shown) = v;
  asm volatile("st.volatile.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(f), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

template <int VEC, int LPR, int UNROLL>
__global__ void __launch_bounds__(1024) gather_roles_kernel(GatherParams p) {
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  const int grid = (int)gridDim.x;
  const int b = (int)blockIdx.x;
  // The lookup kernel ahead of this one in the stream must have finished writing the lists.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (b == 0 && threadIdx.x == 0) set_running(p.order, 0);
  // The next lookup's key loads and table probes may start while this grid drains.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  unsigned long long t0 = 0;
  if (threadIdx.x == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  uint32_t cnt[kNumGroup];
#pragma unroll
  for (int g = 0; g < kNumGroup; g++) cnt[g] = p.counters->count[g];

  int n_host, n_remote;
  split_roles(p, cnt, grid, n_host, n_remote);

  // the counts behind the host list's order are used up: zero again for the next lookup
  if (p.host_hist && b == grid - 1)
    for (uint32_t i = threadIdx.x; i < 2 * kHostBuckets / 4; i += blockDim.x)
      reinterpret_cast<uint4*>(p.host_hist)[i] = make_uint4(0, 0, 0, 0);

  const uint32_t vecs_per_row = p.row_bytes / VEC;
  const uint32_t workers_per_cta = blockDim.x / LPR;
  const uint32_t worker_in_cta = threadIdx.x / LPR;
  const uint32_t sublane = threadIdx.x % LPR;

  int g, first, num;
  if (b < n_host) {
    g = kGroupHost;
    first = 0;
    num = n_host;
  } else if (b < n_host + n_remote) {
    g = kGroupRemote;
    first = n_host;
    num = n_remote;
  } else {
    g = kGroupLocal;
    first = n_host + n_remote;
    num = grid - first;
  }
  RecordIndex ix;
  ix.src_base = p.src_base;
  ix.out = static_cast<char*>(p.out);
  ix.row_bytes = p.row_bytes;
  // rows [lo, lo + len) of list `gg`, shared among `n_ctas` CTAs of which this one is `cta`
  auto copy_span = [&](int gg, uint32_t lo, uint32_t len, uint32_t cta, uint32_t n_ctas) {
    ix.list = (gg == kGroupLocal ? p.list[kGroupLocal]
                                 : (gg == kGroupRemote ? p.list[kGroupRemote] : p.list[kGroupHost])) + lo;
    if (VEC == 32 && gg == kGroupHost) {
      // host rows always move as 16-byte vectors, 4 rows in flight per lane group: 32-byte
      // loads from pinned host memory were slower on every machine measured
      constexpr int kHostLpr = LPR * 2 > 32 ? 32 : LPR * 2;
      const uint32_t wpc = blockDim.x / kHostLpr;
      copy_rows<16, kHostLpr, 4, true>(ix, len, cta * wpc + threadIdx.x / kHostLpr, n_ctas * wpc,
                                       threadIdx.x % kHostLpr, p.row_bytes / 16);
    } else {
      copy_rows<VEC, LPR, UNROLL, true>(ix, len, cta * workers_per_cta + worker_in_cta,
                                        n_ctas * workers_per_cta, sublane, vecs_per_row);
    }
  };
  if (!p.dynamic || p.bulk_mask != 0) {
    // fixed striding: every CTA of a group takes rows b-first, b-first+num, ... of its list
    if (cnt[g] != 0) {
      const bool bulk = (g == kGroupHost && (p.bulk_mask & 1)) || (g == kGroupRemote && (p.bulk_mask & 2));
      if (bulk) {
        ix.list = p.list[g];
        const uint32_t warps_per_cta = blockDim.x >> 5;
        const uint32_t warp = threadIdx.x >> 5;
        uint64_t* bars = reinterpret_cast<uint64_t*>(dyn_smem) + (size_t)warp * kBulkSlots;
        unsigned char* stage = dyn_smem + (size_t)warps_per_cta * kBulkSlots * sizeof(uint64_t) +
                               (size_t)warp * kBulkSlots * p.row_bytes;
        bool ok = copy_rows_bulk(ix, cnt[g], (uint32_t)(b - first) * warps_per_cta + warp,
                                 (uint32_t)num * warps_per_cta, stage, bars);
        if (!ok && (threadIdx.x & 31) == 0) atomicAdd(&p.counters->err_table, 1ull);
      } else {
        copy_span(g, 0, cnt[g], (uint32_t)(b - first), (uint32_t)num);
      }
    }
  } else {
    // Chunked hand-out.  Chunk i < (CTAs of the group) of a list belongs to the group's i-th
    // CTA without any atomic; further chunks come from the list's cursor, fetched one chunk
    // ahead so that the atomic's latency overlaps the copy.  A CTA that finds its own list
    // drained moves on to the other lists (far sources first), so no CTA idles while rows
    // are left anywhere.
    __shared__ uint32_t s_next;
    const uint32_t chunk = workers_per_cta * UNROLL * 2;
    const int o1 = g == kGroupRemote ? kGroupHost : kGroupRemote;
    const int o2 = g == kGroupLocal ? kGroupHost : kGroupLocal;
#pragma unroll
    for (int k = 0; k < kNumGroup; k++) {
      const int gg = k == 0 ? g : (k == 1 ? o1 : o2);
      const uint32_t total =
          gg == kGroupLocal ? cnt[kGroupLocal] : (gg == kGroupRemote ? cnt[kGroupRemote] : cnt[kGroupHost]);
      if (total == 0) continue;
      if (k > 0 && gg == kGroupHost && p.host_hist) continue;  // ordered: see split_roles
      const int ctas_gg = gg == kGroupLocal ? grid - n_host - n_remote : (gg == kGroupRemote ? n_remote : n_host);
      const uint32_t owned = (uint32_t)ctas_gg * chunk;  // rows covered by the first chunks
      if (k > 0 && owned >= total) continue;             // nothing beyond them to take
      uint32_t* cursor = &p.counters->cursor[0] + gg;
      uint32_t base, fetched = 0;
      if (k == 0) {
        base = (uint32_t)(b - first) * chunk;
        if (threadIdx.x == 0 && owned < total) fetched = atomicAdd(cursor, chunk);
      } else {
        if (threadIdx.x == 0) s_next = atomicAdd(cursor, chunk);
        __syncthreads();
        base = owned + s_next;
        __syncthreads();
        if (threadIdx.x == 0 && base < total) fetched = atomicAdd(cursor, chunk);
      }
      bool did = false;
      while (base < total) {
        copy_span(gg, base, min(chunk, total - base), 0u, 1u);
        did = true;
        if (threadIdx.x == 0) s_next = fetched;
        __syncthreads();
        base = owned + s_next;
        __syncthreads();
        if (threadIdx.x == 0 && base < total) fetched = atomicAdd(cursor, chunk);
      }
      if (did && k > 0 && threadIdx.x == 0) {  // finish time of a group this CTA helped
        unsigned long long th;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(th));
        atomicMax(&p.counters->t_end[0] + gg, th);
      }
    }
  }

  // The last CTA to finish publishes the counts of this lookup and re-arms the counters.
  __syncthreads();
  if (threadIdx.x == 0) {
    // when each source group was done, for ugc_stats (one atomic per CTA)
    unsigned long long t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    if (b == 0) p.counters->t_start = t0;
    if (cnt[g] != 0) atomicMax(&p.counters->t_end[g], t1);
    __threadfence();
    uint32_t done = atomicAdd(&p.counters->done_ctas, 1u);
    if (done == (uint32_t)grid - 1) {
#pragma unroll
      for (int g2 = 0; g2 < kNumGroup; g2++) {
        p.counters->last_count[g2] = cnt[g2];
        p.counters->count[g2] = 0;
      }
      p.counters->last_keys = p.n_keys;
      p.counters->done_ctas = 0;
#pragma unroll
      for (int g2 = 0; g2 < kNumGroup; g2++) p.counters->cursor[g2] = 0;
      publish_feedback(p.feedback, p.counters, cnt, p.seq);
      clear_running(p.order, 0);
      __threadfence();
    }
  }
}

// ------------------------------------------------------------------------------------
// distinct keys of a batch
// ------------------------------------------------------------------------------------
// One 32-bit stamp per id of the key space: {epoch : 8 | index : 24}.  A key is new in this
// batch when its stamp carries another epoch; the thread that swings the stamp to the current
// epoch takes the next index and records the key.  The index of every key of the batch is read by
// the extraction that follows (the owner may not have stored it yet when another thread of the claim
// looks).  No sort: the key space is dense and its table already costs 4 bytes per id.
constexpr uint32_t kStampPending = 0x00ffffffu;

// What bounded the claim was the L2's rate of operations on ONE address (0.6 ns each): before the
// first of them lands, every occurrence of the hottest id (18 % of a Zipf-1.2 batch) sees the old
// stamp and tries to swing it, and each warp took its indices with an addition of its own.  So a
// CTA's 1024 keys first meet in a direct-mapped set of ids in shared memory, where one occurrence
// of an id goes on to the L2 (an id whose place is taken goes there itself), and a CTA takes its
// indices with one addition.  212,992 keys, 29,504 of them distinct, claim,
// extraction and index together: 45 -> 20.6 us.
constexpr int kClaimKpt = 4;
constexpr uint32_t kClaimSlots = 2048;

template <typename KeyT>
__global__ void __launch_bounds__(kBlock)
    unique_claim_kernel(const KeyT* __restrict__ keys, uint32_t n, uint64_t num_keys, uint32_t epoch,
                        uint32_t* stamp, KeyT* __restrict__ unique_keys, uint32_t* count,
                        Counters* counters) {
  __shared__ uint32_t s_key[kClaimSlots];
  __shared__ uint32_t s_warp[kWarpsPerBlock];
  __shared__ uint32_t s_base;
  for (uint32_t i = threadIdx.x; i < kClaimSlots; i += kBlock) s_key[i] = kEmptyWord;
  // everything is read and written behind the dependency wait: the stamps and the count are the
  // previous call's, and the keys may be what the launch ahead writes
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t base = blockIdx.x * (kBlock * kClaimKpt) + threadIdx.x;
  const uint32_t mine = (epoch << 24) | kStampPending;
  uint32_t key[kClaimKpt], cur[kClaimKpt], bad = 0;
#pragma unroll
  for (int j = 0; j < kClaimKpt; j++) {
    const uint32_t i = base + j * kBlock;
    const uint64_t k = i < n ? (uint64_t)keys[i] : num_keys;
    key[j] = k < num_keys ? (uint32_t)k : kEmptyWord;  // also drops negative int64 ids
    bad += i < n && k >= num_keys;
  }
  __syncthreads();  // s_key is clear
#pragma unroll
  for (int j = 0; j < kClaimKpt; j++) {
    cur[j] = mine;
    if (key[j] != kEmptyWord) cur[j] = *reinterpret_cast<volatile uint32_t*>(stamp + key[j]);
  }
  // one occurrence of an id in this CTA goes on
  bool go[kClaimKpt];
#pragma unroll
  for (int j = 0; j < kClaimKpt; j++) {
    go[j] = (cur[j] >> 24) != epoch;
    if (go[j]) {
      volatile uint32_t* slot = s_key + ((key[j] * 2654435761u) >> 21);
      uint32_t held = *slot;
      if (held == kEmptyWord) held = atomicCAS(const_cast<uint32_t*>(slot), kEmptyWord, key[j]);
      go[j] = held != key[j];  // kEmptyWord: this thread's; another id: goes on by itself
    }
  }
  uint32_t old[kClaimKpt];
#pragma unroll
  for (int j = 0; j < kClaimKpt; j++)
    if (go[j]) old[j] = atomicCAS(stamp + key[j], cur[j], mine);
  uint32_t before[kClaimKpt], total = 0;  // winners of this warp ahead of this thread's, per key
#pragma unroll
  for (int j = 0; j < kClaimKpt; j++) {
    if (go[j]) {
      while (old[j] != cur[j] && (old[j] >> 24) != epoch) {
        cur[j] = old[j];
        old[j] = atomicCAS(stamp + key[j], cur[j], mine);
      }
      go[j] = old[j] == cur[j];
    }
    const unsigned m = __ballot_sync(kFull, go[j]);
    before[j] = total + __popc(m & ((1u << lane) - 1));
    total += __popc(m);
  }
  if (lane == 0) s_warp[warp] = total;
  bad = __reduce_add_sync(kFull, bad);
  if (lane == 0 && bad) atomicAdd(&counters->err_key_range, (unsigned long long)bad);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kWarpsPerBlock; w++) {
      const uint32_t c = s_warp[w];
      s_warp[w] = run;
      run += c;
    }
    s_base = run ? atomicAdd(count, run) : 0;
  }
  __syncthreads();
  const uint32_t first = s_base + s_warp[warp];
#pragma unroll
  for (int j = 0; j < kClaimKpt; j++) {
    if (!go[j]) continue;
    unique_keys[first + before[j]] = (KeyT)key[j];
    stamp[key[j]] = (epoch << 24) | (first + before[j]);
  }
}
static_assert(kClaimSlots == 1u << 11, "the slot is the top 11 bits of the hash");

// ------------------------------------------------------------------------------------
// host list in address order
// ------------------------------------------------------------------------------------
// Rows of pinned host memory arrive faster when the reads in flight lie close together and move
// through the table in ascending order, which is what the reference gets from sorting its whole
// index (coll_cache_lib/cache_context.cu:702-761).  Measured with nothing else running, random
// against ordered (kHostBuckets ranges): 128-byte rows 37 -> 49 GB/s over a 1 GB table and 8.9 ->
// 14.2 over 32 GB, 256-byte rows 17.7 -> 23.4 over 32 GB, 512-byte rows 35.7 -> 38.0.  256 ranges
// gave a third of that over 32 GB: the window of rows in flight has to be narrower than a range.
// Only the host list is ordered, by a counting sort: the lookup counts the ranges while it emits the
// list, one small kernel scatters it, the gather clears the counts for the next lookup.
// `hist` holds kHostBuckets counts followed by kHostBuckets cursors, all zero on entry.
constexpr int kScatterBlock = 512;
constexpr int kBucketsPerThread = kHostBuckets / kScatterBlock;

__global__ void __launch_bounds__(kScatterBlock)
    host_scatter_kernel(const uint64_t* __restrict__ list, uint64_t* __restrict__ sorted,
                        const Counters* counters, uint32_t* hist, uint32_t shift) {
  __shared__ uint32_t s_start[kHostBuckets];
  __shared__ uint32_t s_warp[kScatterBlock / 32];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // exclusive prefix of the counts, the same in every CTA
  uint32_t cnt[kBucketsPerThread], sum = 0;
  const uint4* h4 = reinterpret_cast<const uint4*>(hist) + threadIdx.x * (kBucketsPerThread / 4);
#pragma unroll
  for (int i = 0; i < kBucketsPerThread / 4; i++) {
    const uint4 h = __ldcg(h4 + i);
    cnt[4 * i] = h.x, cnt[4 * i + 1] = h.y, cnt[4 * i + 2] = h.z, cnt[4 * i + 3] = h.w;
    sum += h.x + h.y + h.z + h.w;
  }
  uint32_t x = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, x, d);
    if (lane >= (uint32_t)d) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  uint32_t run = x - sum;
  for (uint32_t w = 0; w < warp; w++) run += s_warp[w];
#pragma unroll
  for (int i = 0; i < kBucketsPerThread; i++) {
    s_start[threadIdx.x * kBucketsPerThread + i] = run;
    run += cnt[i];
  }
  __syncthreads();
  uint32_t* cursor = hist + kHostBuckets;
  const uint32_t n = counters->count[kGroupHost];
  for (uint32_t i = blockIdx.x * kScatterBlock + threadIdx.x; i < n; i += gridDim.x * kScatterBlock) {
    const uint64_t rec = list[i];
    const uint32_t b = host_bucket(rec_off(rec), shift);
    sorted[s_start[b] + atomicAdd(&cursor[b], 1u)] = rec;
  }
}

// ------------------------------------------------------------------------------------
// direct extraction: table probe and row copy in ONE kernel, no index lists
// ------------------------------------------------------------------------------------
// A warp owns tiles of 32 consecutive keys or fewer, down to one (direct_tile_shift) -- the largest
// size that leaves every warp nearly the same number of tiles; with 32-key tiles a batch of
// 212,992 keys is 1.4 tiles per warp, so 40 % of the warps would carry twice the work of the
// rest.  Lane l probes the table for key l of the tile;
// the row addresses then travel by shuffle to the lane groups that copy the rows, so the
// destination of a tile is one contiguous piece of the output.  Rows of every source (local
// slice, peer slice over NVLink, pinned host memory) are copied where they come up, which
// spreads the few far rows of a batch evenly over the SMs and over the kernel's duration.
// Keys are loaded two tiles ahead and probed one tile ahead of the tile being copied.
// Tiles are dealt to warps so that consecutive tiles land on different CTAs: every SM gets
// the same number of rows to within one tile.
//
// This is the counterpart of the reference's ungrouped extraction (one extract_data over
// DataIterMixLoc, coll_cache_lib/cache_context.cu:1295-1329, :137-159) with the table
// lookup folded in; the grouped path above stays the better shape when many rows of a batch
// come from the host.
// A table read in flight: one 4-slot line (probing table) or one word (flat).  The kind is a template
// parameter so that a flat table's probe holds one register across the row copies instead of eight.
template <bool FLAT>
struct Probe {
  uint32_t k0, k1, k2, k3, w0, w1, w2, w3;
};
template <>
struct Probe<true> {
  uint32_t w0;
};

__device__ __forceinline__ void probe_issue(const TableView& t, uint32_t key, bool valid, Probe<true>& pr) {
  pr.w0 = kEmptyWord;
  if (valid) asm volatile("ld.global.cg.b32 %0, [%1];" : "=r"(pr.w0) : "l"(t.flat + key));
}
__device__ __forceinline__ void probe_issue(const TableView& t, uint32_t key, bool valid, Probe<false>& pr) {
  pr.k0 = pr.k1 = pr.k2 = pr.k3 = kEmptyWord;
  pr.w0 = pr.w1 = pr.w2 = pr.w3 = kEmptyWord;
  if (valid) {
    const uint2* a = t.slots + (size_t)(murmur3_32(key) & t.line_mask) * kSlotsPerLine;
    asm volatile("ld.global.cg.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(pr.k0), "=r"(pr.w0), "=r"(pr.k1), "=r"(pr.w1), "=r"(pr.k2), "=r"(pr.w2),
                   "=r"(pr.k3), "=r"(pr.w3)
                 : "l"(a));
  }
}

__device__ __forceinline__ uint32_t probe_resolve(const TableView&, const Probe<true>& pr, uint32_t, bool) {
  return pr.w0;
}
__device__ __forceinline__ uint32_t probe_resolve(const TableView& t, const Probe<false>& pr, uint32_t key,
                                                  bool valid) {
  if (!valid) return pr.w0;
  if (pr.k0 == key) return pr.w0;  // live slots carry the key with the top bit clear
  if (pr.k1 == key) return pr.w1;
  if (pr.k2 == key) return pr.w2;
  if (pr.k3 == key) return pr.w3;
  if (pr.k0 == kEmptyWord || pr.k1 == kEmptyWord || pr.k2 == kEmptyWord || pr.k3 == kEmptyWord)
    return kEmptyWord;  // a never-used slot ends the search
  return probe_rest(t.slots, t.line_mask, key, murmur3_32(key) & t.line_mask);
}

// Key `lane` of tile `tl` (tiles of 1 << shift keys; lanes beyond the tile hold no key); ids
// outside [0, num_keys) are counted and dropped.
template <typename KeyT>
__device__ __forceinline__ void fetch_key(const KeyT* __restrict__ keys, uint32_t tl, uint32_t n_tiles,
                                          uint32_t shift, uint32_t n_keys, uint64_t num_keys,
                                          uint32_t lane, uint32_t& key, bool& valid, uint32_t& bad) {
  const uint32_t idx = (tl << shift) + lane;
  valid = tl < n_tiles && (lane >> shift) == 0 && idx < n_keys;
  uint64_t k = valid ? ld_key(keys + idx) : 0;
  if (k >= num_keys) {  // also catches negative int64 ids
    valid = false;
    bad++;
    k = 0;
  }
  key = (uint32_t)k;
}

// Keys per tile (log2): 32 at first.  A batch that leaves warps without a tile is bound by the chain
// key - probe - rows of one warp: halve the tile while all tiles still run at once, down to the rows
// one pass copies (208 keys of 512-byte rows back to back: one pass of 4 rows a warp instead of
// eight, 6.6 -> 4.3 us).  Then halve it to 8 at least while the warps' tile counts differ by a tenth.
__host__ __device__ inline uint32_t direct_tile_shift(uint32_t n_keys, uint32_t n_warps, uint32_t rows_per_pass) {
  uint32_t shift = 5;
  auto tiles = [&](uint32_t sh) { return (uint32_t)(((uint64_t)n_keys + (1u << sh) - 1) >> sh); };
  while (shift > 0 && (1u << (shift - 1)) >= rows_per_pass && tiles(shift - 1) <= n_warps) shift--;
  while (shift > 3 && (1u << (shift - 1)) >= rows_per_pass) {
    const uint32_t t = tiles(shift);
    const uint32_t rounds = (t + n_warps - 1) / n_warps;
    if (t <= n_warps || 10ull * t >= 9ull * rounds * n_warps) break;
    shift--;
  }
  return shift;
}

// UNIQUE: the extraction of a deduplicated lookup.  Its keys, their number and the stamps come from
// the claim just ahead in the stream, so it waits first; the tile size follows the number found; and
// it writes the index of every key of the batch, whose loads go out with the first probes instead of
// in a launch of their own.  It lets nothing start early: what it writes besides rows (the index, the
// number) may be the next launch's keys.
template <typename KeyT, int VEC, bool FLAT, bool DEEP, bool EARLY, bool UNIQUE>
__global__ void __launch_bounds__(kBlock, DEEP ? 3 : 4)
    extract_direct_kernel(const KeyT* __restrict__ keys, DirectParams p) {
  // rows in flight per lane group: 4 (2 with 32-byte vectors) at 4 CTAs per SM, or twice that
  // at 3 CTAs per SM
  constexpr int UNROLL = (VEC == 32 ? 2 : 4) * (DEEP ? 2 : 1);
  __shared__ uint32_t s_cnt[kNumGroup];
  __shared__ const char* s_src[kMaxLocation];
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < kMaxLocation; i++) s_src[i] = static_cast<const char*>(p.src_base[i]);
  }
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n_warps = gridDim.x * (blockDim.x >> 5);
  uint32_t n_keys = p.n_keys, tshift = p.tile_shift;
  uint32_t inv_at = 0, inv_step = 0;
  uint64_t inv_key[2] = {0, 0};
  if (UNIQUE) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    n_keys = min(__ldcg(&p.counters->unique_count[p.unique_slot]), p.n_keys);
    if (tshift > 5) tshift = direct_tile_shift(n_keys, n_warps, min(32u, UNROLL * (32u >> p.lpr_shift)));
    inv_at = blockIdx.x * blockDim.x + threadIdx.x;
    inv_step = gridDim.x * blockDim.x;
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (inv_at + j * inv_step < p.n_keys)
        inv_key[j] = (uint64_t)static_cast<const KeyT*>(p.batch_keys)[inv_at + j * inv_step];
  }
  const uint32_t tile_keys = 1u << tshift;
  const uint32_t n_tiles = (n_keys + tile_keys - 1) >> tshift;
  uint32_t tile = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  if (threadIdx.x < kNumGroup) s_cnt[threadIdx.x] = 0;

  uint32_t bad = 0;

  // The dependency wait comes first, unless the extraction ahead still runs (still_running): then the
  // first two key loads and the first probe go out ahead of it.
  bool waited = false;
  Vec<VEC> early;
  uint32_t early_row = 32;  // lane whose key the row in `early` belongs to; 32 = none
  const uint32_t early_tile = tile;
  auto wait_for_launch_ahead = [&]() {
    waited = true;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!UNIQUE) {
      // The next launch may start: behind the wait, so that whatever it finds running or waits for,
      // nothing older than this extraction is still under way.
      if (blockIdx.x < kRunMarks && lane == 0) set_running(p.order, blockIdx.x);
      asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    if (EARLY && early_row < 32) {
      if (lane < p.row_bytes / VEC)
        st_row(static_cast<char*>(p.out) + (((size_t)early_tile << tshift) + early_row) * p.row_bytes +
                   (size_t)lane * VEC,
               early);
    }
    // The extraction ahead of this one is complete now.  One thread hands ITS counts on (they
    // sit in the other slot, final) -- to the pinned host mirror the library reads to choose
    // the mode of later lookups -- and clears that slot for the launch after this one.
    // (the thread chosen for this belongs to the warp that is dealt the fewest tiles -- the last
    // warp of the last CTA -- so that the writes across PCIe delay no warp the launch waits for)
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 32) {
      uint32_t* other = p.counters->dcount[p.slot ^ 1u];
      uint32_t prev[kNumGroup];
#pragma unroll
      for (int g = 0; g < kNumGroup; g++) prev[g] = other[g];
      if (p.publish_prev) publish_feedback(p.feedback, p.counters, prev, p.prev_seq);
#pragma unroll
      for (int g = 0; g < kNumGroup; g++) other[g] = 0;
      unsigned long long t0;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
      p.counters->t_start = t0;
      p.counters->t_index = 0;
      p.counters->last_keys = p.n_keys;
      if (UNIQUE) {
        *p.n_unique = n_keys;
        if (p.unique_clear != kNoSlot) p.counters->unique_count[p.unique_clear] = 0;  // for the next one
      }
    }
  };
  const bool ahead_runs = !UNIQUE && still_running(p.order);
  if (!UNIQUE && !ahead_runs) asm volatile("griddepcontrol.wait;" ::: "memory");
  uint32_t key_cur, key_nxt;
  bool ok_cur, ok_nxt;
  fetch_key(keys, tile, n_tiles, tshift, n_keys, p.table.num_keys, lane, key_cur, ok_cur, bad);
  fetch_key(keys, tile + n_warps, n_tiles, tshift, n_keys, p.table.num_keys, lane, key_nxt, ok_nxt, bad);
  Probe<FLAT> pr;
  probe_issue(p.table, key_cur, ok_cur, pr);
  auto batch_index = [&](uint64_t k) {  // index of an id of the batch among the distinct ones
    return k < p.table.num_keys ? (int32_t)(__ldcg(p.stamp + k) & kStampPending) : -1;
  };
  int32_t inv_idx[2];
  if (UNIQUE) {
#pragma unroll
    for (int j = 0; j < 2; j++) inv_idx[j] = batch_index(inv_key[j]);
  }
  uint32_t word = probe_resolve(p.table, pr, key_cur, ok_cur);
  // EARLY: the first host row of this warp's first tile is fetched before the dependency wait
  // and held in registers, one piece per lane.
  // CTAs of this launch become resident while the launch ahead is still waiting for ITS last
  // host rows; their requests keep the host link's queue filled across the boundary between
  // two launches, where it would otherwise run empty and fill up again.
  uint32_t early_lane = 32;
  if (EARLY && ahead_runs) {
    const bool is_host = ok_cur && word == kEmptyWord;
    const unsigned hmask = __ballot_sync(kFull, is_host);
    if (hmask && p.row_bytes / VEC <= 32) {
      early_lane = __ffs(hmask) - 1;
      const uint32_t k = __shfl_sync(kFull, key_cur, early_lane);
      if (lane < p.row_bytes / VEC)
        ld_row(early, static_cast<const char*>(p.host_base) + (size_t)(k & p.host_mask) * p.row_bytes +
                          (size_t)lane * VEC);
    }
    early_row = early_lane;
  }
  // With the extraction ahead still running the dependency wait comes as late as it can: behind the
  // loads of this warp's first rows, and ahead of its first store (the batch ahead may have had the
  // same output buffer).  A batch of one pass per warp then has all its loads behind it when the
  // launch ahead ends.
  if (UNIQUE) {
    wait_for_launch_ahead();
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (inv_at + j * inv_step < p.n_keys) p.inverse[inv_at + j * inv_step] = inv_idx[j];
  }

  const uint32_t lpr = 1u << p.lpr_shift;
  const uint32_t rpi = 32u >> p.lpr_shift;       // rows per warp-wide load
  const uint32_t sub = lane & (lpr - 1);
  const uint32_t rsel = lane >> p.lpr_shift;
  const uint32_t vecs_per_row = p.row_bytes / VEC;
  __syncthreads();  // s_src, s_cnt

  while (tile < n_tiles) {
    // next tile's probe and the key load two tiles ahead go out before this tile's rows
    probe_issue(p.table, key_nxt, ok_nxt, pr);
    uint32_t key_nn;
    bool ok_nn;
    fetch_key(keys, tile + 2 * n_warps, n_tiles, tshift, n_keys, p.table.num_keys, lane, key_nn, ok_nn, bad);

    // this lane's key: source address and group
    const char* src = nullptr;
    uint32_t group = kNumGroup;
    if (ok_cur) {
      uint32_t loc, off;
      if (word == kEmptyWord) {
        loc = p.host_loc;
        off = key_cur & p.host_mask;
        group = kGroupHost;
      } else {
        loc = word_loc(word);
        off = word_off(word);
        group = loc == p.local_loc ? kGroupLocal : kGroupRemote;
      }
      src = s_src[loc] + (size_t)off * p.row_bytes;
    }
    if (EARLY && lane == early_lane) src = nullptr;  // copied already (still counted below)
    early_lane = 32;
#pragma unroll
    for (int g = 0; g < kNumGroup; g++) {
      const uint32_t n = __popc(__ballot_sync(kFull, group == (uint32_t)g));
      if (lane == 0 && n) atomicAdd(&s_cnt[g], n);
    }

    char* out_tile = static_cast<char*>(p.out) + ((size_t)tile << tshift) * p.row_bytes;
    const unsigned long long src_bits = reinterpret_cast<unsigned long long>(src);
    const size_t row_step = (size_t)rpi * p.row_bytes;  // between the rows of one lane group
    for (uint32_t rb = 0; rb < tile_keys; rb += UNROLL * rpi) {
      const char* s[UNROLL];
#pragma unroll
      for (int u = 0; u < UNROLL; u++) {
        const uint32_t r = rb + u * rpi + rsel;
        const unsigned long long a = __shfl_sync(kFull, src_bits, r & 31);
        s[u] = r < tile_keys ? reinterpret_cast<const char*>(a) : nullptr;
      }
      char* d0 = out_tile + (size_t)(rb + rsel) * p.row_bytes;
      for (uint32_t c = sub; c < vecs_per_row; c += lpr) {
        Vec<VEC> v[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++)
          if (s[u]) ld_row(v[u], s[u] + (size_t)c * VEC);
        if (!waited) wait_for_launch_ahead();
#pragma unroll
        for (int u = 0; u < UNROLL; u++)
          if (s[u]) st_row(d0 + u * row_step + (size_t)c * VEC, v[u]);
      }
    }

    word = probe_resolve(p.table, pr, key_nxt, ok_nxt);
    key_cur = key_nxt;
    ok_cur = ok_nxt;
    key_nxt = key_nn;
    ok_nxt = ok_nn;
    tile += n_warps;
  }

  if (!waited) wait_for_launch_ahead();  // a warp without rows
  if (UNIQUE)
    for (uint32_t i = inv_at + 2 * inv_step; i < p.n_keys; i += inv_step)
      p.inverse[i] = batch_index((uint64_t)static_cast<const KeyT*>(p.batch_keys)[i]);
  // Per-source counts of this lookup: fire-and-forget adds into the slot this launch owns.
  // Nothing here waits on memory, so the kernel ends with its last row store: no count of
  // finished CTAs, no fence, no single CTA that tidies up after the others.
  if (bad) atomicAdd(&p.counters->err_key_range, (unsigned long long)bad);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t* mine = p.counters->dcount[p.slot];
#pragma unroll
    for (int g = 0; g < kNumGroup; g++)
      if (s_cnt[g]) atomicAdd(mine + g, s_cnt[g]);
    unsigned long long t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    atomicMax(&p.counters->t_end[kGroupLocal], t1);  // one span for the whole kernel
    if (!UNIQUE && blockIdx.x < kRunMarks) clear_running(p.order, blockIdx.x);
  }
}

// ------------------------------------------------------------------------------------
// pooled lookup: table probe, row fetch and per-bag sum in ONE kernel
// ------------------------------------------------------------------------------------
// A bag is a run of consecutive keys; its result is the sum (or mean) of its rows, one fp32
// vector of `dim` elements.  The looked-up rows never reach memory.  The additions of one output
// element happen in key order, in fp32, starting from +0, one rounding each (no fused multiply-add
// is involved), so the result is bit-for-bit what a sequential fp32 loop over the bag gives on any
// machine.  Keys outside [0, num_keys) are counted and contribute nothing.  The reference leaves
// pooling to the model that consumes the rows; this is the fused form of lookup + segment sum.
//
// What bounds it is latency: offsets - keys - table - rows is a chain of reads, and the order of the
// additions leaves a bag to the lanes that own its columns.  So
//  * a CTA is as many warps as a row has columns of 32 pieces; it takes a tile of consecutive bags,
//    and its threads probe all of the tile's keys at once (two a thread, addresses through shared
//    memory) instead of each lane group its own bag's;
//  * 4-byte pieces put four times the warps on a bag and hold 64 rows of it in flight per lane, at four
//    times the instructions; with 16-byte pieces it is 8 rows;
//  * the loads run on over the ends of bags, and a bag's end is rare code outside the row loop.
// Before (a lane group probed and summed bag by bag) and now: 8192 ragged bags of 26 rows of 512 bytes
// 55.7 -> 26.0 us (22 with one cache whose rows the L2 holds), 65,536 bags of 5 fp16 rows of 128 bytes 23.6 -> 15.7, 73 bags of 400 rows of 1 KiB
// 167 -> 32, 145 bags of 877 rows of 256 bytes 108 -> 20, 186 bags of 23 rows of 128 bytes 15 -> 6.4.
// With 16-byte pieces and many bags the rows' way through the L1 and the instructions bound it.
template <bool F16, int VEC>
__device__ __forceinline__ void pool_add(float* acc, const Vec<VEC>& v) {
  if (F16) {
#pragma unroll
    for (int i = 0; i < VEC / 4; i++) {
      // volatile: the widened values of many rows in flight would not fit the registers, and moving
      // the conversion out of a loop over the bags that share those rows is what the compiler does
      float x, y;
      asm volatile("{\n\t.reg .f16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.f32.f16 %0, a;\n\tcvt.f32.f16 %1, b;\n\t}"
                   : "=f"(x), "=f"(y)
                   : "r"(v.v[i]));
      acc[2 * i] = __fadd_rn(acc[2 * i], x);
      acc[2 * i + 1] = __fadd_rn(acc[2 * i + 1], y);
    }
  } else {
    const float* f = reinterpret_cast<const float*>(&v);
#pragma unroll
    for (int i = 0; i < VEC / 4; i++) acc[i] = __fadd_rn(acc[i], f[i]);
  }
}

// Position in `keys` where bag b starts (b == n_bags: where the last one ends), inside [0, n_keys].
__device__ __forceinline__ uint32_t pool_bag_start(const PoolParams& p, uint32_t b) {
  const long long o = p.offsets ? p.offsets[b] : (long long)b * p.bag_size;
  return (uint32_t)min(max(o, 0ll), (long long)p.n_keys);
}

constexpr int kPoolMaxBlock = 256;  // eight columns; wider rows take several CTAs a tile
constexpr uint32_t kPoolMaxBags = 128;  // bags a tile

template <typename KeyT, bool F16, int VEC>
__global__ void __launch_bounds__(kPoolMaxBlock, VEC == 16 ? 3 : 2) lookup_pool_kernel(const KeyT* __restrict__ keys, PoolParams p) {
  constexpr int NF = VEC / (F16 ? 2 : 4);  // elements per piece of a row (VEC bytes)
  constexpr uint32_t UNROLL = VEC == 16 ? 8 : 64;  // rows in flight per lane
  constexpr int KPT = 2;                   // keys a thread probes at a time
  __shared__ const char* s_src[kMaxLocation];
  __shared__ const char* s_row[KPT * kPoolMaxBlock];  // rows of the chunk of keys at hand; nullptr: none
  __shared__ uint32_t s_end[kPoolMaxBags + 1];        // where the tile's bags start, and the last one ends
  __shared__ uint32_t s_cnt[kNumGroup + 1];
  const uint32_t tid = threadIdx.x;
  if (tid < kMaxLocation) s_src[tid] = static_cast<const char*>(p.src_base[tid]);
  if (tid <= kNumGroup) s_cnt[tid] = 0;
  // nothing is read ahead of the dependency wait: keys and offsets may be what the launch ahead writes
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  const uint32_t tile = blockIdx.x / p.col_blocks, col_block = blockIdx.x - tile * p.col_blocks;
  const uint32_t bag_lo = tile * p.bags_per_tile;
  const uint32_t n_bags = min(p.bags_per_tile, p.n_bags - bag_lo);
  for (uint32_t i = tid; i <= n_bags; i += blockDim.x) s_end[i] = pool_bag_start(p, bag_lo + i);
  __syncthreads();
  const uint32_t k_lo = s_end[0];
  const uint32_t k_hi = max(k_lo, s_end[n_bags]);

  // a lane group (as many lanes as a column has pieces) adds up one column of the bags
  // [bag, bag_hi) of the tile; rows of less than 32 pieces leave a warp several groups, which
  // share out the tile's bags
  const uint32_t lpr = 1u << p.lpr_shift;
  const uint32_t groups = 32u >> p.lpr_shift;
  const uint32_t group = (tid & 31) >> p.lpr_shift;
  const uint32_t c = ((col_block * (blockDim.x >> 5) + (tid >> 5)) << p.lpr_shift) + (tid & (lpr - 1));
  const bool has = c < p.row_bytes / VEC;
  uint32_t bag = n_bags * group / groups;
  const uint32_t bag_hi = n_bags * (group + 1) / groups;
  uint32_t bag_begin = min(max(s_end[bag], k_lo), k_hi);
  uint32_t bag_end = bag < bag_hi ? max(bag_begin, min(s_end[bag + 1], k_hi)) : bag_begin;
  uint32_t k = bag_begin;                                               // the group's next key
  const uint32_t k_end = max(k, min(s_end[bag_hi], k_hi));              // and the end of its keys
  float acc[NF];
#pragma unroll
  for (int i = 0; i < NF; i++) acc[i] = 0.f;
  // writes bag `bag` out and moves on to the next one
  auto flush = [&]() {
    if (has) {
      const uint32_t len = bag_end - bag_begin;
      if (p.mean && len > 0) {
        const float d = (float)len;
#pragma unroll
        for (int i = 0; i < NF; i++) acc[i] = __fdiv_rn(acc[i], d);
      }
      float* dst = p.out + (size_t)(bag_lo + bag) * p.dim + (size_t)c * NF;
      if (NF >= 4) {
#pragma unroll
        for (int i = 0; i + 3 < NF; i += 4)
          reinterpret_cast<float4*>(dst)[i / 4] = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
      } else if (NF == 2) {
        *reinterpret_cast<float2*>(dst) = make_float2(acc[0], acc[NF - 1]);
      } else {
        dst[0] = acc[0];
      }
    }
#pragma unroll
    for (int i = 0; i < NF; i++) acc[i] = 0.f;
    bag++;
    bag_begin = bag_end;
    if (bag < bag_hi) bag_end = max(bag_begin, min(s_end[bag + 1], k_hi));
  };

  uint32_t bad = 0, n_local = 0, n_remote = 0, n_host = 0;
  const uint32_t chunk = KPT * blockDim.x;
  for (uint32_t c0 = k_lo; c0 < k_hi; c0 += chunk) {
    uint64_t key[KPT];
#pragma unroll
    for (int j = 0; j < KPT; j++) {
      const uint32_t i = c0 + j * blockDim.x + tid;
      key[j] = i < k_hi ? (uint64_t)keys[i] : 0;
    }
    uint32_t word[KPT];
#pragma unroll
    for (int j = 0; j < KPT; j++) {
      word[j] = kEmptyWord;
      if (c0 + j * blockDim.x + tid < k_hi && key[j] < p.table.num_keys) word[j] = table_lookup(p.table, (uint32_t)key[j]);
    }
    if (c0 != k_lo) __syncthreads();  // every group is done with the chunk before
#pragma unroll
    for (int j = 0; j < KPT; j++) {
      const char* src = nullptr;
      if (c0 + j * blockDim.x + tid < k_hi) {
        if (key[j] >= p.table.num_keys) {  // also catches negative int64 ids
          bad++;
        } else if (word[j] == kEmptyWord) {
          src = s_src[p.host_loc] + (size_t)((uint32_t)key[j] & p.host_mask) * p.row_bytes;
          n_host++;
        } else {
          const uint32_t loc = word_loc(word[j]);
          src = s_src[loc] + (size_t)word_off(word[j]) * p.row_bytes;
          if (loc == p.local_loc) {
            n_local++;
          } else {
            n_remote++;
          }
        }
      }
      s_row[j * blockDim.x + tid] = src;
    }
    __syncthreads();
    const uint32_t stop = min(k_end, c0 + chunk);
    for (; k < stop; k += min(UNROLL, stop - k)) {
      Vec<VEC> v[UNROLL];
#pragma unroll
      for (uint32_t u = 0; u < UNROLL; u++) {
        // a row that is not there adds +0, which leaves a sum that started from +0 as it is
#pragma unroll
        for (int i = 0; i < VEC / 4; i++) v[u].v[i] = 0;
        const char* src = k + u < stop ? s_row[k + u - c0] : nullptr;
        if (has && src) ld_row(v[u], src + (size_t)c * VEC);
      }
      // the part of these rows that lies in the bag at hand, then the bag's end, and on: the end of
      // a bag stands here once, not behind every row (it is long, and instructions are what small
      // pieces spend their time on)
      const uint32_t n = min(UNROLL, stop - k);
      if (bag_end - k >= n) {
#pragma unroll
        for (uint32_t u = 0; u < UNROLL; u++) pool_add<F16, VEC>(acc, v[u]);
      } else {
        for (uint32_t lo = 0;;) {
          const uint32_t hi = min(n, bag_end - k);
#pragma unroll
          for (uint32_t u = 0; u < UNROLL; u++)
            if (u >= lo && u < hi) pool_add<F16, VEC>(acc, v[u]);
          lo = hi;
          if (hi >= n || bag >= bag_hi) break;
          flush();  // also passes empty bags
        }
      }
    }
  }
  while (bag < bag_hi) flush();  // the last bag, and empty ones after it

  // counts: one global atomic per CTA and counter (an atomic per thread on one address would
  // take longer than the kernel's memory traffic)
  if (col_block != 0) return;
  n_local = __reduce_add_sync(kFull, n_local);
  n_remote = __reduce_add_sync(kFull, n_remote);
  n_host = __reduce_add_sync(kFull, n_host);
  bad = __reduce_add_sync(kFull, bad);
  if ((tid & 31) == 0) {
    if (n_local) atomicAdd(&s_cnt[kGroupLocal], n_local);
    if (n_remote) atomicAdd(&s_cnt[kGroupRemote], n_remote);
    if (n_host) atomicAdd(&s_cnt[kGroupHost], n_host);
    if (bad) atomicAdd(&s_cnt[kNumGroup], bad);
  }
  __syncthreads();
  if (tid < kNumGroup && s_cnt[tid]) atomicAdd(&p.counters->pool_rows[tid], (unsigned long long)s_cnt[tid]);
  if (tid == kNumGroup && s_cnt[kNumGroup])
    atomicAdd(&p.counters->err_key_range, (unsigned long long)s_cnt[kNumGroup]);
}

template <int VEC, int LPR, int UNROLL>
__global__ void __launch_bounds__(kBlock) fill_scatter_kernel(KeySlotIndex ix, uint32_t n) {
  const uint32_t vecs_per_row = ix.row_bytes / VEC;
  constexpr uint32_t kWorkersPerCta = kBlock / LPR;
  const uint32_t worker = blockIdx.x * kWorkersPerCta + threadIdx.x / LPR;
  copy_rows<VEC, LPR, UNROLL, false>(ix, n, worker, gridDim.x * kWorkersPerCta, threadIdx.x % LPR,
                                     vecs_per_row);
}

// ------------------------------------------------------------------------------------
// table maintenance
// ------------------------------------------------------------------------------------
__global__ void table_clear_kernel(uint4* p, size_t n16) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (; i < n16; i += stride) p[i] = make_uint4(kEmptyWord, kEmptyWord, kEmptyWord, kEmptyWord);
}

// Inserts a key that is not live in the table.  A slot is free when its key has the top
// bit set (never used, or evicted).  Key and word are published by one 64-bit
// compare-and-swap, so a concurrent lookup sees the slot either free or complete.
__device__ __forceinline__ bool insert_hashed(const TableView& t, uint32_t key, uint32_t word) {
  uint32_t line = murmur3_32(key) & t.line_mask;
  for (uint32_t step = 0; step <= t.line_mask; step++) {
    Line l = ld_line(t.slots, line);
#pragma unroll
    for (int s = 0; s < kSlotsPerLine; s++) {
      if (l.key[s] == key) return false;  // already live: caller counts it as an error
      if (l.key[s] & kTombstone) {
        unsigned long long* slot =
            reinterpret_cast<unsigned long long*>(t.slots + (size_t)line * kSlotsPerLine + s);
        unsigned long long expect = ((unsigned long long)l.word[s] << 32) | l.key[s];
        unsigned long long want = ((unsigned long long)word << 32) | key;
        if (atomicCAS(slot, expect, want) == expect) return true;
        // lost the race for this slot: keep scanning (the winner holds a different key)
      }
    }
    line = (line + 1) & t.line_mask;
  }
  return false;
}

__global__ void __launch_bounds__(kBlock)
    table_insert_kernel(TableView t, const uint32_t* __restrict__ keys, SlotView offs, uint32_t loc,
                        uint32_t n, Counters* counters, bool allow_same) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t key = keys[i];
  uint32_t word = pack_word(loc, offs.data ? offs.data[slot_pos(offs, i)] : offs.base + i);
  bool ok;
  if (key >= t.num_keys) {
    ok = false;
  } else if (t.kind == kTableFlat) {
    const uint32_t old = atomicExch(t.flat + key, word);
    ok = old == kEmptyWord || (allow_same && old == word);
  } else if (allow_same) {
    // The key may be live further along its probe sequence than the first free slot: look
    // for it before a slot is claimed, or it would end up in the table twice.
    const uint32_t w = table_lookup(t, key);
    ok = w == word || (w == kEmptyWord && insert_hashed(t, key, word));
  } else {
    ok = insert_hashed(t, key, word);
  }
  if (!ok) atomicAdd(&counters->err_table, 1ull);
}

// Refresh: every key of the list leaves its present source.  If its new source is a peer whose
// table shows the row there already, the entry's word is replaced in place by (peer, slot) --
// one 32-bit store, so a concurrent lookup sees the old or the new source, both valid until the
// grace period ends; otherwise the entry is removed (the key is served by the host until a later
// phase of the refresh inserts it again).
__global__ void __launch_bounds__(kBlock)
    table_repoint_kernel(RepointParams p, const uint32_t* __restrict__ keys, uint32_t n, Counters* counters) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t key = keys[i];
  const TableView& t = p.own;
  bool ok = false;
  if (key < t.num_keys) {
    uint32_t word_new = kEmptyWord;
    const uint32_t src_new = p.src_new[key];
    if (src_new < p.num_device && src_new != p.me && p.peer[src_new].num_keys) {
      const uint32_t w = table_lookup(p.peer[src_new], key);
      if (w != kEmptyWord && word_loc(w) == src_new) word_new = w;
    }
    if (t.kind == kTableFlat) {
      ok = atomicExch(t.flat + key, word_new) != kEmptyWord;
    } else {
      uint32_t line = murmur3_32(key) & t.line_mask;
      for (uint32_t step = 0; step <= t.line_mask && !ok; step++) {
        Line l = ld_line(t.slots, line);
        bool stop = false;
#pragma unroll
        for (int s = 0; s < kSlotsPerLine; s++) {
          if (l.key[s] == key && !ok) {
            uint2* slot = &t.slots[(size_t)line * kSlotsPerLine + s];
            if (word_new == kEmptyWord) {
              atomicOr(&slot->x, kTombstone);
            } else {
              atomicExch(&slot->y, word_new);
            }
            ok = true;
          }
          stop |= (l.key[s] == kEmptyWord);
        }
        if (stop) break;
        line = (line + 1) & t.line_mask;
      }
    }
  }
  if (!ok) atomicAdd(&counters->err_table, 1ull);
}

__global__ void __launch_bounds__(kBlock)
    table_evict_kernel(TableView t, const uint32_t* __restrict__ keys, uint32_t n,
                       Counters* counters) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t key = keys[i];
  bool ok = false;
  if (key < t.num_keys) {
    if (t.kind == kTableFlat) {
      ok = atomicExch(t.flat + key, kEmptyWord) != kEmptyWord;
    } else {
      uint32_t line = murmur3_32(key) & t.line_mask;
      for (uint32_t step = 0; step <= t.line_mask && !ok; step++) {
        Line l = ld_line(t.slots, line);
        bool stop = false;
#pragma unroll
        for (int s = 0; s < kSlotsPerLine; s++) {
          if (l.key[s] == key && !ok) {
            atomicOr(&t.slots[(size_t)line * kSlotsPerLine + s].x, kTombstone);
            ok = true;
          }
          stop |= (l.key[s] == kEmptyWord);
        }
        if (stop) break;
        line = (line + 1) & t.line_mask;
      }
    }
  }
  if (!ok) atomicAdd(&counters->err_table, 1ull);
}

__global__ void __launch_bounds__(kBlock)
    table_words_kernel(TableView t, const uint32_t* __restrict__ keys, uint32_t n,
                       uint32_t* __restrict__ words) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t key = keys[i];
  words[i] = key < t.num_keys ? table_lookup(t, key) : kEmptyWord;
}

__global__ void __launch_bounds__(kBlock)
    table_resolve_kernel(TableView peer, const uint32_t* __restrict__ keys, uint32_t n,
                         uint32_t expect_loc, SlotView offs, Counters* counters) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t key = keys[i];
  uint32_t w = key < peer.num_keys ? table_lookup(peer, key) : kEmptyWord;
  uint32_t* dst = offs.data + slot_pos(offs, i);
  if (w == kEmptyWord || word_loc(w) != expect_loc) {
    atomicAdd(&counters->err_table, 1ull);
    *dst = 0;
  } else {
    *dst = word_off(w);
  }
}

__global__ void iota_kernel(uint32_t* dst, uint32_t start, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (; i < n; i += stride) dst[i] = start + i;
}

// ------------------------------------------------------------------------------------
// key classification over the whole id space (build and refresh), ordered compaction
// ------------------------------------------------------------------------------------
// For every key the placement gives the source that serves this reader.  Build wants one
// ascending key list per GPU source; a refresh wants the ascending lists of keys whose
// source changed (evict here, bring in here, drop a peer entry, point to a peer).  Three
// passes over tiles of kClassTile keys: per-tile counts, a scan over tiles, a stable scatter.
constexpr int kClassTile = 2048;
constexpr int kClassRounds = kClassTile / kBlock;

// Bit mask of the lists key k belongs to (see ClassifyParams in device_types.h).
__device__ __forceinline__ uint32_t class_mask(const ClassifyParams& p, uint64_t k) {
  const uint32_t src_new = p.src_new[k];
  if (p.src_old == nullptr) return src_new < p.num_device ? (1u << src_new) : 0u;  // build
  const uint32_t src_old = p.src_old[k];
  if (src_old == src_new) return 0u;
  uint32_t m = 0;
  if (src_old == p.me) m |= 1u << kListEvict;
  if (src_new == p.me) m |= 1u << kListInsert;
  if (src_old < p.num_device && src_old != p.me) m |= 1u << kListDropRemote;
  if (src_new < p.num_device && src_new != p.me) m |= 1u << (kListAttach0 + src_new);
  return m;
}

__global__ void __launch_bounds__(kBlock) classify_count_kernel(ClassifyParams p, uint32_t* tile_counts) {
  __shared__ uint32_t s_cnt[kMaxClassLists];
  if (threadIdx.x < kMaxClassLists) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t base = (uint64_t)blockIdx.x * kClassTile;
  uint32_t masks[kClassRounds];
#pragma unroll
  for (int j = 0; j < kClassRounds; j++) {
    uint64_t k = base + (uint64_t)j * kBlock + threadIdx.x;
    masks[j] = k < p.num_keys ? class_mask(p, k) : 0u;
  }
  for (int l = 0; l < p.num_lists; l++) {
    uint32_t c = 0;
#pragma unroll
    for (int j = 0; j < kClassRounds; j++) c += (masks[j] >> l) & 1u;
    c = __reduce_add_sync(kFull, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_cnt[l], c);
  }
  __syncthreads();
  if (threadIdx.x < kMaxClassLists)
    tile_counts[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = s_cnt[threadIdx.x];
}

// One CTA per list: exclusive scan of that list's per-tile counts, total to totals[list].
__global__ void __launch_bounds__(1024) classify_scan_kernel(uint32_t* tile_counts, uint32_t n_tiles,
                                                             unsigned long long* totals) {
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_carry;
  uint32_t* row = tile_counts + (size_t)blockIdx.x * n_tiles;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  unsigned long long total = 0;
  for (uint32_t start = 0; start < n_tiles; start += 1024) {
    const uint32_t i = start + threadIdx.x;
    const uint32_t v = i < n_tiles ? row[i] : 0;
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t y = __shfl_up_sync(kFull, x, d);
      if (lane >= (uint32_t)d) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = s_warp[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        uint32_t y = __shfl_up_sync(kFull, w, d);
        if (lane >= (uint32_t)d) w += y;
      }
      s_warp[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    const uint32_t carry = s_carry;
    const uint32_t before = carry + (warp ? s_warp[warp - 1] : 0) + x - v;  // exclusive prefix
    if (i < n_tiles) row[i] = before;
    __syncthreads();
    if (threadIdx.x == 1023) {
      s_carry = carry + s_warp[31];
    }
    __syncthreads();
    total = s_carry;
  }
  // per-tile offsets are 32-bit: a list holds fewer than 2^32 keys (the id space is < 2^31)
  if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kBlock)
    classify_scatter_kernel(ClassifyParams p, const uint32_t* __restrict__ tile_offsets,
                            uint32_t* __restrict__ out) {
  __shared__ uint32_t s_warp_cnt[kWarpsPerBlock][kMaxClassLists];
  __shared__ uint32_t s_running[kMaxClassLists];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kMaxClassLists)
    s_running[threadIdx.x] = tile_offsets[(size_t)threadIdx.x * gridDim.x + blockIdx.x];
  __syncthreads();
  const uint64_t base = (uint64_t)blockIdx.x * kClassTile;
  for (int j = 0; j < kClassRounds; j++) {
    const uint64_t k = base + (uint64_t)j * kBlock + threadIdx.x;
    const uint32_t m = k < p.num_keys ? class_mask(p, k) : 0u;
    uint32_t rank[kMaxClassLists];
    for (int l = 0; l < p.num_lists; l++) {
      const unsigned b = __ballot_sync(kFull, (m >> l) & 1u);
      rank[l] = __popc(b & ((1u << lane) - 1));
      if (lane == 0) s_warp_cnt[warp][l] = __popc(b);
    }
    __syncthreads();
    for (int l = 0; l < p.num_lists; l++) {
      if ((m >> l) & 1u) {
        uint32_t pos = s_running[l] + rank[l];
        for (uint32_t w = 0; w < warp; w++) pos += s_warp_cnt[w][l];
        out[p.list_base[l] + pos] = (uint32_t)k;
      }
    }
    __syncthreads();
    if (threadIdx.x < (uint32_t)p.num_lists) {
      uint32_t add = 0;
      for (int w = 0; w < kWarpsPerBlock; w++) add += s_warp_cnt[w][threadIdx.x];
      s_running[threadIdx.x] += add;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------
// hotness recording: per-key access counts of a batch, kept on the device
// ------------------------------------------------------------------------------------
// What bounds it is the L2's rate of additions to ONE address (0.6 ns each): the hottest id is 18 %
// of a Zipf-1.2 batch, 38,000 additions of 212,992, which took 22 us one by one.  So the hot ids are
// added up before they leave the SM: lanes of a warp that hold the same id find each other (match)
// and count once, and a direct-mapped set of kRecordSlots counters in shared memory, one per id
// that comes first, takes the warps' counts; an id whose slot is taken goes straight to the L2.
// 1024 keys a CTA: enough for the hot ids to meet, few enough to fill the SMs from 150 k keys on.
constexpr int kRecordKpt = 4;
constexpr uint32_t kRecordSlots = 1024;

template <typename KeyT>
__global__ void __launch_bounds__(kBlock)
    record_kernel(const KeyT* __restrict__ keys, uint32_t n, uint32_t* __restrict__ counts,
                  uint64_t num_keys) {
  __shared__ uint32_t s_key[kRecordSlots], s_cnt[kRecordSlots];
  for (uint32_t i = threadIdx.x; i < kRecordSlots; i += kBlock) {
    s_key[i] = kEmptyWord;
    s_cnt[i] = 0;
  }
  // the keys are read behind the dependency wait: they may be what the launch ahead writes
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t base = blockIdx.x * (kBlock * kRecordKpt) + threadIdx.x;
  uint32_t key[kRecordKpt];
#pragma unroll
  for (int j = 0; j < kRecordKpt; j++) {
    const uint64_t i = (uint64_t)base + j * kBlock;
    const uint64_t k = i < n ? (uint64_t)keys[i] : num_keys;
    key[j] = k < num_keys ? (uint32_t)k : kEmptyWord;  // also drops negative int64 ids
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRecordKpt; j++) {
    const unsigned same = __match_any_sync(kFull, key[j]);
    if (key[j] == kEmptyWord || (threadIdx.x & 31) != (uint32_t)(__ffs(same) - 1)) continue;
    const uint32_t slot = (key[j] * 2654435761u) >> 22;
    const uint32_t held = atomicCAS(&s_key[slot], kEmptyWord, key[j]);
    if (held == kEmptyWord || held == key[j]) {
      atomicAdd(&s_cnt[slot], (uint32_t)__popc(same));
    } else {
      atomicAdd(counts + key[j], (uint32_t)__popc(same));  // fire-and-forget reduction in L2
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kRecordSlots; i += kBlock)
    if (s_cnt[i]) atomicAdd(counts + s_key[i], s_cnt[i]);
}
static_assert(kRecordSlots == 1u << 10, "the slot is the top 10 bits of the hash");

// ------------------------------------------------------------------------------------
// synthetic table rows
// ------------------------------------------------------------------------------------
__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
__device__ __forceinline__ uint32_t gen_f32_bits(uint64_t seed, uint64_t e) {
  uint64_t x = splitmix64(seed ^ splitmix64(e));
  return __float_as_uint((float)(x >> 40) * (1.0f / 8388608.0f) - 1.0f);
}
__device__ __forceinline__ uint32_t gen_f16_bits(uint64_t seed, uint64_t e) {
  uint64_t x = splitmix64(seed ^ splitmix64(e));
  int v = (int)(x >> 53) - 1024;  // value = v * 2^-10
  if (v == 0) return 0;
  uint32_t sign = 0;
  if (v < 0) {
    sign = 0x8000u;
    v = -v;
  }
  int msb = 31 - __clz(v);
  uint32_t exp = (uint32_t)(msb - 10 + 15);
  uint32_t man = ((uint32_t)v << (10 - msb)) & 0x3ffu;
  return sign | (exp << 10) | man;
}

// One thread writes 4 bytes: one fp32 element or two fp16 elements.
__global__ void gen_table_kernel(uint32_t* dst, uint64_t seed, uint64_t elem_begin, uint64_t n_words,
                                 int elem_bytes) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (; i < n_words; i += stride) {
    uint32_t w;
    if (elem_bytes == 4) {
      w = gen_f32_bits(seed, elem_begin + i);
    } else {
      uint64_t e = elem_begin + 2 * i;
      w = gen_f16_bits(seed, e) | (gen_f16_bits(seed, e + 1) << 16);
    }
    dst[i] = w;
  }
}

// ------------------------------------------------------------------------------------
// dispatch helpers
// ------------------------------------------------------------------------------------
inline int grid_for(uint32_t n) { return (int)((n + kBlock - 1) / kBlock); }

// Lanes per row: the smallest power of two >= vectors per row, at most a warp.
inline int lanes_per_row(uint32_t row_bytes, int vec) {
  uint32_t vecs = row_bytes / (uint32_t)vec;
  int l = 1;
  while ((uint32_t)l < vecs && l < 32) l <<= 1;
  return l;
}

// Launch with programmatic stream serialization: the kernel may be scheduled while its
// predecessor in the stream is still running and orders itself with griddepcontrol.wait.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kern)(KArgs...), int grid, int block, size_t smem, cudaStream_t s,
                       bool pdl, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

template <int VEC, int LPR, int UNROLL>
cudaError_t gather_launch(const GatherParams& p, int grid, int block, size_t smem, cudaStream_t s) {
  auto kern = gather_roles_kernel<VEC, LPR, UNROLL>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  return launch_pdl(kern, grid, block, smem, s, p.pdl != 0, p);
}

template <int VEC, int UNROLL>
cudaError_t gather_dispatch_lpr(const GatherParams& p, int grid, int block, size_t smem, cudaStream_t s) {
  switch (lanes_per_row(p.row_bytes, VEC)) {
    case 1: return gather_launch<VEC, 1, UNROLL>(p, grid, block, smem, s);
    case 2: return gather_launch<VEC, 2, UNROLL>(p, grid, block, smem, s);
    case 4: return gather_launch<VEC, 4, UNROLL>(p, grid, block, smem, s);
    case 8: return gather_launch<VEC, 8, UNROLL>(p, grid, block, smem, s);
    case 16: return gather_launch<VEC, 16, UNROLL>(p, grid, block, smem, s);
    default: return gather_launch<VEC, 32, UNROLL>(p, grid, block, smem, s);
  }
}

template <int VEC, int UNROLL>
cudaError_t fill_dispatch_lpr(const KeySlotIndex& ix, uint32_t n, int grid, cudaStream_t s) {
  switch (lanes_per_row(ix.row_bytes, VEC)) {
    case 1: fill_scatter_kernel<VEC, 1, UNROLL><<<grid, kBlock, 0, s>>>(ix, n); break;
    case 2: fill_scatter_kernel<VEC, 2, UNROLL><<<grid, kBlock, 0, s>>>(ix, n); break;
    case 4: fill_scatter_kernel<VEC, 4, UNROLL><<<grid, kBlock, 0, s>>>(ix, n); break;
    case 8: fill_scatter_kernel<VEC, 8, UNROLL><<<grid, kBlock, 0, s>>>(ix, n); break;
    case 16: fill_scatter_kernel<VEC, 16, UNROLL><<<grid, kBlock, 0, s>>>(ix, n); break;
    default: fill_scatter_kernel<VEC, 32, UNROLL><<<grid, kBlock, 0, s>>>(ix, n); break;
  }
  return cudaGetLastError();
}

inline uint32_t host_mask_of(int empty_feat) {
  return empty_feat > 0 && empty_feat < 32 ? ((1u << empty_feat) - 1u) : 0xffffffffu;
}

// bucket = row offset >> shift: kHostBuckets ranges over the host table
inline uint32_t host_order_shift(uint64_t host_rows) {
  uint32_t shift = 0;
  while (shift < 31 && (host_rows >> shift) > (uint64_t)kHostBuckets) shift++;
  return shift;
}

}  // namespace

// ------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------
cudaError_t launch_lookup_group(const void* keys, int key_bytes, uint32_t n, const TableView& table,
                                uint32_t local_loc, uint32_t host_loc, int empty_feat,
                                uint64_t* list_local, uint64_t* list_remote, uint64_t* list_host,
                                Counters* counters, const StreamOrder& order, int keys_per_thread, int sm_count,
                                uint32_t* host_hist, uint64_t host_rows, bool pdl, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const uint32_t mask = host_mask_of(empty_feat);
  const uint32_t shift = host_order_shift(host_rows);
  // 0: four keys a thread once that still leaves every SM four CTAs, one below
  if (keys_per_thread == 0) keys_per_thread = n >= (uint64_t)sm_count * 4 * kBlock * 4 ? 4 : 1;
#define UGC_LAUNCH_LOOKUP(KEYT, KPT)                                                             \
  return launch_pdl(lookup_group_kernel<KEYT, KPT>, (int)((n + kBlock * KPT - 1) / (kBlock * KPT)), \
                    kBlock, 0, stream, pdl, static_cast<const KEYT*>(keys), n, table, local_loc,   \
                    host_loc, mask, list_local, list_remote, list_host, counters, order, host_hist, shift)
  if (key_bytes == 8) {
    if (keys_per_thread == 1) UGC_LAUNCH_LOOKUP(long long, 1);
    if (keys_per_thread == 2) UGC_LAUNCH_LOOKUP(long long, 2);
    UGC_LAUNCH_LOOKUP(long long, 4);
  } else {
    if (keys_per_thread == 1) UGC_LAUNCH_LOOKUP(uint32_t, 1);
    if (keys_per_thread == 2) UGC_LAUNCH_LOOKUP(uint32_t, 2);
    UGC_LAUNCH_LOOKUP(uint32_t, 4);
  }
#undef UGC_LAUNCH_LOOKUP
}

int usable_vec_bytes(uint32_t row_bytes, int want, const void* out, const void* const* src_base,
                     int n_src) {
  uintptr_t bits = reinterpret_cast<uintptr_t>(out) | row_bytes;
  for (int i = 0; i < n_src; i++) bits |= reinterpret_cast<uintptr_t>(src_base[i]);
  if (want >= 32 && (bits & 31) == 0) return 32;
  if (want >= 16 && (bits & 15) == 0) return 16;
  return 4;
}

cudaError_t launch_extract_direct(const void* keys, int key_bytes, const DirectParams& p_in, int grid,
                                  int block, int vec_bytes, bool deep, bool early_host, bool pdl,
                                  cudaStream_t stream) {
  if (block != 128 && block != 256) block = kBlock;
  const int warps_per_block = block / 32;
  if (p_in.n_keys == 0) return cudaSuccess;
  DirectParams p = p_in;
  const int vec = usable_vec_bytes(p.row_bytes, vec_bytes, p.out, p.src_base, kMaxLocation);
  const int lpr = lanes_per_row(p.row_bytes, vec);
  p.lpr_shift = 0;
  while ((1 << p.lpr_shift) < lpr) p.lpr_shift++;
  // p.tile_shift 3..5 forces the tile
  const int unroll = (vec == 32 ? 2 : 4) * (deep && !p.stamp ? 2 : 1);
  uint32_t shift = p_in.tile_shift;
  p.tile_shift = shift;
  if (shift < 3 || shift > 5) {
    shift = direct_tile_shift(p.n_keys, (uint32_t)(grid * warps_per_block), (uint32_t)std::min(32, unroll * (32 / lpr)));
    p.tile_shift = p.stamp ? 32u : shift;  // of a deduplicated lookup the kernel knows the number of keys
  }
  const int tiles = (int)(((long long)p.n_keys + (1ll << shift) - 1) >> shift);
  grid = std::max(1, std::min(grid, (tiles + warps_per_block - 1) / warps_per_block));
  auto launch = [&](auto key, auto vec_c, auto flat_c) {
    using KeyT = decltype(key);
    constexpr int V = decltype(vec_c)::value;
    constexpr bool F = decltype(flat_c)::value;
    const KeyT* k = static_cast<const KeyT*>(keys);
    if (p.stamp)
      return launch_pdl(extract_direct_kernel<KeyT, V, F, false, false, true>, grid, block, 0, stream, pdl, k, p);
    if (deep) return launch_pdl(extract_direct_kernel<KeyT, V, F, true, false, false>, grid, block, 0, stream, pdl, k, p);
    if (early_host)
      return launch_pdl(extract_direct_kernel<KeyT, V, F, false, true, false>, grid, block, 0, stream, pdl, k, p);
    return launch_pdl(extract_direct_kernel<KeyT, V, F, false, false, false>, grid, block, 0, stream, pdl, k, p);
  };
  auto by_table = [&](auto key, auto vec_c) {
    return p.table.kind == kTableFlat ? launch(key, vec_c, std::true_type{}) : launch(key, vec_c, std::false_type{});
  };
  auto by_vec = [&](auto key) {
    if (vec == 32) return by_table(key, std::integral_constant<int, 32>{});
    if (vec == 16) return by_table(key, std::integral_constant<int, 16>{});
    return by_table(key, std::integral_constant<int, 4>{});
  };
  return key_bytes == 8 ? by_vec((long long)0) : by_vec((uint32_t)0);
}

cudaError_t launch_lookup_pool(const void* keys, int key_bytes, const PoolParams& p_in, bool f16,
                               int sm_count, int vec_bytes, bool pdl, cudaStream_t stream) {
  if (p_in.n_bags == 0) return cudaSuccess;
  PoolParams p = p_in;
  // 4-byte pieces while 16-byte ones would keep fewer than five warps an SM busy.  Few bags are bound
  // by how many rows of one bag are in flight, many by instructions.  Measured, 4- against 16-byte:
  // 512-byte rows, 212,992 keys in 256 bags 27.5 / 52.6 us, 512 bags 22.1 / 31.0, 1024 bags 22.0 / 19.0,
  // 8192 bags 35.0 / 15.8; 128-byte fp16 rows, 80,000 keys in 2048 bags 8.2 / 11.2, 8192 bags 11.8 / 8.3.
  const uint64_t lanes16 = (uint64_t)p.n_bags * (p.row_bytes / 16);
  const int vec = vec_bytes == 4 || vec_bytes == 16 ? vec_bytes : lanes16 < (uint64_t)sm_count * 5 * 32 ? 4 : 16;
  const int lpr = lanes_per_row(p.row_bytes, vec);
  p.lpr_shift = 0;
  while ((1 << p.lpr_shift) < lpr) p.lpr_shift++;
  const uint32_t columns = (p.row_bytes / (uint32_t)vec + lpr - 1) / lpr;
  p.col_blocks = (columns + kPoolMaxBlock / 32 - 1) / (kPoolMaxBlock / 32);
  const uint32_t warps = (columns + p.col_blocks - 1) / p.col_blocks;
  // bags a tile: twice the keys of a resident warp's share of the batch, and no more than the CTA's
  // threads probe at once (104,982 keys of 32-byte rows: half of that 11.7 us, this 8.3)
  const uint64_t avg_bag = std::max<uint64_t>(1, p.offsets ? (uint64_t)p.n_keys / p.n_bags : p.bag_size);
  const uint64_t share = 2 * (uint64_t)p.n_keys * columns / ((uint64_t)sm_count * 32);
  const uint64_t want = std::min<uint64_t>(std::max<uint64_t>(share, 32 / lpr), 2 * 32 * warps);
  p.bags_per_tile = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(1, want / avg_bag), kPoolMaxBags);
  const uint64_t grid = ((uint64_t)p.n_bags + p.bags_per_tile - 1) / p.bags_per_tile * p.col_blocks;
  auto launch = [&](auto key, auto half, auto vec_c) {
    using KeyT = decltype(key);
    return launch_pdl(lookup_pool_kernel<KeyT, decltype(half)::value, decltype(vec_c)::value>, (int)grid,
                      (int)warps * 32, 0, stream, pdl, static_cast<const KeyT*>(keys), p);
  };
  auto by_vec = [&](auto key, auto half) {
    return vec == 16 ? launch(key, half, std::integral_constant<int, 16>{})
                     : launch(key, half, std::integral_constant<int, 4>{});
  };
  auto by_elem = [&](auto key) { return f16 ? by_vec(key, std::true_type{}) : by_vec(key, std::false_type{}); };
  return key_bytes == 8 ? by_elem((long long)0) : by_elem((uint32_t)0);
}

cudaError_t launch_unique_claim(const void* keys, int key_bytes, uint32_t n, uint64_t num_keys, uint32_t epoch,
                                uint32_t* stamp, void* unique_keys, uint32_t* count, Counters* counters, bool pdl,
                                cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const int grid = (int)(((uint64_t)n + kBlock * kClaimKpt - 1) / (kBlock * kClaimKpt));
  if (key_bytes == 8)
    return launch_pdl(unique_claim_kernel<long long>, grid, kBlock, 0, stream, pdl, static_cast<const long long*>(keys),
                      n, num_keys, epoch, stamp, static_cast<long long*>(unique_keys), count, counters);
  return launch_pdl(unique_claim_kernel<uint32_t>, grid, kBlock, 0, stream, pdl, static_cast<const uint32_t*>(keys), n,
                    num_keys, epoch, stamp, static_cast<uint32_t*>(unique_keys), count, counters);
}

size_t host_order_scratch_bytes() { return 2 * kHostBuckets * sizeof(uint32_t); }

cudaError_t launch_host_order(const uint64_t* list_host, uint64_t* sorted, const Counters* counters,
                              uint32_t* hist, uint64_t host_rows, int sm_count, bool pdl, cudaStream_t stream) {
  return launch_pdl(host_scatter_kernel, sm_count, kScatterBlock, 0, stream, pdl, list_host, sorted, counters, hist,
                    host_order_shift(host_rows));
}

// Host rows a CTA of the gather has in flight: four per lane group, in pieces of 16 bytes at most.
int gather_rows_in_flight(const GatherParams& p, int block, int vec_bytes) {
  const int vec = std::min(16, usable_vec_bytes(p.row_bytes, vec_bytes, p.out, p.src_base, kMaxLocation));
  return block / lanes_per_row(p.row_bytes, vec) * 4;
}

cudaError_t launch_gather_roles(const GatherParams& p_in, int grid, int block, int vec_bytes,
                                cudaStream_t stream) {
  GatherParams p = p_in;
  vec_bytes = usable_vec_bytes(p.row_bytes, vec_bytes, p.out, p.src_base, kMaxLocation);
  if (grid < 3) grid = 3;  // one CTA per source group at least
  if (block != 256 && block != 512 && block != 1024) block = 256;
  // bulk staging needs 16-byte aligned rows on both sides
  if (p.row_bytes % 16 != 0 || (reinterpret_cast<uintptr_t>(p.out) & 15)) p.bulk_mask = 0;
  size_t smem = 0;
  if (p.bulk_mask) {
    smem = (size_t)(block / 32) * kBulkSlots * (sizeof(uint64_t) + p.row_bytes);
    if (smem > 200 * 1024) {
      p.bulk_mask = 0;
      smem = 0;
    }
  }
  if (vec_bytes == 32) return gather_dispatch_lpr<32, 2>(p, grid, block, smem, stream);
  if (vec_bytes == 16) return gather_dispatch_lpr<16, 4>(p, grid, block, smem, stream);
  return gather_dispatch_lpr<4, 4>(p, grid, block, smem, stream);
}

cudaError_t launch_fill_scatter(const void* host_table, void* slice, const uint32_t* keys,
                                const SlotView& slots, uint32_t n, uint32_t row_bytes,
                                int empty_feat, int grid, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  KeySlotIndex ix;
  ix.keys = keys;
  ix.slots = slots;
  ix.host_mask = host_mask_of(empty_feat);
  ix.host = static_cast<const char*>(host_table);
  ix.slice = static_cast<char*>(slice);
  ix.row_bytes = row_bytes;
  if (grid < 1) grid = 1;
  const void* bases[1] = {host_table};
  if (usable_vec_bytes(row_bytes, 16, slice, bases, 1) == 16) return fill_dispatch_lpr<16, 8>(ix, n, grid, stream);
  return fill_dispatch_lpr<4, 8>(ix, n, grid, stream);
}

cudaError_t launch_table_clear(const TableView& t, cudaStream_t stream) {
  size_t bytes = t.kind == kTableFlat ? (size_t)t.num_keys * 4
                                      : ((size_t)t.line_mask + 1) * kSlotsPerLine * sizeof(uint2);
  // flat tables are allocated rounded up to 16 bytes by the runtime
  size_t n16 = (bytes + 15) / 16;
  void* base = t.kind == kTableFlat ? static_cast<void*>(t.flat) : static_cast<void*>(t.slots);
  table_clear_kernel<<<1184, kBlock, 0, stream>>>(static_cast<uint4*>(base), n16);
  return cudaGetLastError();
}

cudaError_t launch_table_insert(const TableView& t, const uint32_t* keys, const SlotView& offs,
                                uint32_t loc, uint32_t n, Counters* counters, cudaStream_t stream,
                                bool allow_same) {
  if (n == 0) return cudaSuccess;
  table_insert_kernel<<<grid_for(n), kBlock, 0, stream>>>(t, keys, offs, loc, n, counters, allow_same);
  return cudaGetLastError();
}

cudaError_t launch_table_repoint(const RepointParams& p, const uint32_t* keys, uint32_t n,
                                 Counters* counters, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  table_repoint_kernel<<<grid_for(n), kBlock, 0, stream>>>(p, keys, n, counters);
  return cudaGetLastError();
}

cudaError_t launch_iota(uint32_t* dst, uint32_t start, uint32_t n, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  iota_kernel<<<std::min(grid_for(n), 148 * 8), kBlock, 0, stream>>>(dst, start, n);
  return cudaGetLastError();
}

cudaError_t launch_table_evict(const TableView& t, const uint32_t* keys, uint32_t n,
                               Counters* counters, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  table_evict_kernel<<<grid_for(n), kBlock, 0, stream>>>(t, keys, n, counters);
  return cudaGetLastError();
}

cudaError_t launch_table_words(const TableView& t, const uint32_t* keys, uint32_t n,
                               uint32_t* words, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  table_words_kernel<<<grid_for(n), kBlock, 0, stream>>>(t, keys, n, words);
  return cudaGetLastError();
}

cudaError_t launch_table_resolve(const TableView& peer, const uint32_t* keys, uint32_t n,
                                 uint32_t expect_loc, const SlotView& offs, Counters* counters,
                                 cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  table_resolve_kernel<<<grid_for(n), kBlock, 0, stream>>>(peer, keys, n, expect_loc, offs, counters);
  return cudaGetLastError();
}

size_t classify_scratch_bytes(uint64_t num_keys) {
  const size_t n_tiles = (size_t)((num_keys + kClassTile - 1) / kClassTile);
  return n_tiles * kMaxClassLists * sizeof(uint32_t) + kMaxClassLists * sizeof(unsigned long long) + 256;
}

// scratch layout: tile counts [kMaxClassLists][n_tiles] u32, then totals [kMaxClassLists] u64
cudaError_t launch_classify_count(const ClassifyParams& p, void* scratch, cudaStream_t stream) {
  const uint32_t n_tiles = (uint32_t)((p.num_keys + kClassTile - 1) / kClassTile);
  uint32_t* tile_counts = static_cast<uint32_t*>(scratch);
  size_t off = ((size_t)n_tiles * kMaxClassLists * sizeof(uint32_t) + 255) / 256 * 256;
  unsigned long long* totals = reinterpret_cast<unsigned long long*>(static_cast<char*>(scratch) + off);
  classify_count_kernel<<<n_tiles, kBlock, 0, stream>>>(p, tile_counts);
  classify_scan_kernel<<<kMaxClassLists, 1024, 0, stream>>>(tile_counts, n_tiles, totals);
  return cudaGetLastError();
}

const unsigned long long* classify_totals(void* scratch, uint64_t num_keys) {
  const size_t n_tiles = (size_t)((num_keys + kClassTile - 1) / kClassTile);
  size_t off = (n_tiles * kMaxClassLists * sizeof(uint32_t) + 255) / 256 * 256;
  return reinterpret_cast<const unsigned long long*>(static_cast<char*>(scratch) + off);
}

cudaError_t launch_classify_scatter(const ClassifyParams& p, const void* scratch, uint32_t* out,
                                    cudaStream_t stream) {
  const uint32_t n_tiles = (uint32_t)((p.num_keys + kClassTile - 1) / kClassTile);
  classify_scatter_kernel<<<n_tiles, kBlock, 0, stream>>>(p, static_cast<const uint32_t*>(scratch), out);
  return cudaGetLastError();
}

cudaError_t launch_record(const void* keys, int key_bytes, uint32_t n, uint32_t* counts,
                          uint64_t num_keys, bool pdl, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const int grid = (int)(((uint64_t)n + kBlock * kRecordKpt - 1) / (kBlock * kRecordKpt));
  if (key_bytes == 8)
    return launch_pdl(record_kernel<long long>, grid, kBlock, 0, stream, pdl,
                      static_cast<const long long*>(keys), n, counts, num_keys);
  return launch_pdl(record_kernel<uint32_t>, grid, kBlock, 0, stream, pdl,
                    static_cast<const uint32_t*>(keys), n, counts, num_keys);
}

cudaError_t launch_gen_table(void* dst, uint64_t seed, uint64_t row_begin, uint64_t n_rows,
                             uint64_t dim, int elem_bytes, cudaStream_t stream) {
  uint64_t n_words = n_rows * dim * (uint64_t)elem_bytes / 4;
  if (n_words == 0) return cudaSuccess;
  uint64_t blocks = (n_words + kBlock - 1) / kBlock;
  int grid = (int)(blocks < 148ull * 16 ? blocks : 148ull * 16);
  gen_table_kernel<<<grid, kBlock, 0, stream>>>(static_cast<uint32_t*>(dst), seed, row_begin * dim,
                                                n_words, elem_bytes);
  return cudaGetLastError();
}

}  // namespace ugc
