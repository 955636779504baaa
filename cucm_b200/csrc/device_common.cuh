// device_common.cuh -- device helpers shared by the coder kernels.
//
// Included inside an anonymous namespace by every translation unit that
// instantiates the kernels (engine_kernels.cu, noalloc.cu), so each module
// carries its own copies and its own constant tables.
#pragma once

constexpr int kStageMin = 4096;
constexpr uint32_t kFlushBlock = 512;

__host__ __device__ constexpr int next_pow2(int v) {
  int p = 1;
  while (p < v) p <<= 1;
  return p;
}
__host__ __device__ constexpr int ilog2(int v) {
  int l = 0;
  while ((1 << l) < v) l++;
  return l;
}

// Overlay bucket of a key: Fibonacci hashing, logNB bits.
__device__ __forceinline__ uint32_t bucket_of(uint32_t key, int logNB) {
  return (key * 0x9E3779B1u) >> (32 - logNB);
}

__device__ inline void copy_tables(const Tables *from, Tables *dst) {
  const uint4 *src = reinterpret_cast<const uint4 *>(from);
  uint4 *d = reinterpret_cast<uint4 *>(dst);
  for (int i = threadIdx.x; i < (int)(sizeof(Tables) / 16); i += blockDim.x) d[i] = src[i];
}

// Restore a slot to its initial contents (zero, or the prelearned model).
__device__ inline void reset_slot(uint8_t *slot, const uint8_t *init_tables) {
  uint4 *d = reinterpret_cast<uint4 *>(slot);
  const size_t n = kSlotTableBytes / 16;
  if (init_tables) {
    const uint4 *src = reinterpret_cast<const uint4 *>(init_tables);
    for (size_t i = threadIdx.x; i < n; i += blockDim.x) d[i] = src[i];
  } else {
    const uint4 z = make_uint4(0, 0, 0, 0);
    for (size_t i = threadIdx.x; i < n; i += blockDim.x) d[i] = z;
  }
}

// Mixer output for one bit (Mixer::p, cucm_compress_v2.cu:636-644, then
// `if (pr < 2048) pr++`), given stretched inputs.
__device__ __forceinline__ int mix_pr(const int32_t *w, int cxt, const int smp[kOrders], const Tables *t) {
  long long sum = 0;
#pragma unroll
  for (int o = 0; o < kOrders; o++) sum += (long long)w[cxt * kOrders + o] * smp[o];
  sum >>= 16;
  int idx = sum < -2047 ? -2047 : (sum > 2048 ? 2048 : (int)sum);
  int pr = t->squash[idx + 2047];
  return pr < 2048 ? pr + 1 : pr;
}

// Coder state of a compress CTA (held by one warp; lane 0 codes).
struct Coder {
  uint32_t x1, x2;
  uint64_t head;     // bytes produced
  uint64_t flushed;  // bytes written to global
};

// One coder input in the form the coder consumes: the probability as a
// multiplier (pr << 20) and the coded bit as a mask (all ones for a 0).
__device__ __forceinline__ uint2 coder_entry(uint32_t e) {  // e = pr << 1 | y
  return make_uint2((e << 19) & 0xfff00000u, (e & 1u) - 1u);
}
__device__ __forceinline__ uint32_t coder_entry_u16(const uint2 &q) { return (q.x >> 19) | (q.y + 1u); }

// One bit: narrows [x1, x2] to the coded bit's part.  The split point
// x1 + floor((x2 - x1) * pr / 4096) is taken as the high word of
// (x2 - x1) * (pr << 20); it equals the reference's
// (r >> 12) * pr + ((r & 0xfff) * pr >> 12) (cucm_compress_v2.cu:855-856)
// because (r >> 12) * pr is exact.
__device__ __forceinline__ void coder_narrow(uint32_t f, uint32_t n, uint32_t &x1, uint32_t &x2) {
  const uint32_t t = __umulhi(x2 - x1, f);
  const uint32_t xm = x1 + t, xn = x1 + t + 1;
  x2 = (x2 & n) | (xm & ~n);
  x1 = (xn & n) | (x1 & ~n);
}
// The reference's form of one bit: any number of bytes.
__device__ __forceinline__ void coder_step(const uint2 &q, uint32_t &x1, uint32_t &x2, uint32_t &head, uint8_t *ring,
                                           uint32_t mask) {
  coder_narrow(q.x, q.y, x1, x2);
  while ((x1 ^ x2) < 0x1000000u) {
    ring[head & mask] = (uint8_t)(x2 >> 24);
    head++;
    x1 <<= 8;
    x2 = (x2 << 8) | 255u;
  }
}

// A coder is one serial chain, so it is bound by the latency of a step.  A
// branch, taken or not, costs ~25 cycles on it, more than the arithmetic of a
// bit, so a group of 16 bits runs without one: a bit shifts by 0 or 8, and its
// byte goes to the ring's head whether or not the head then advances past it.
// A bit that has to shift out two bytes or more (coded against odds of 2^8
// and up) is seen in `least`, and its group is done again in the reference's
// form.  48 cycles a bit for a warp alone (a probe; 50 in the compressor's coder
// warp, 53 in the fixed-model coder's; 62 in the tail pass, whose one thread a
// chunk votes and writes its bytes too) against 80-90 with the test after every
// bit, whatever the data; 8 bits a group measured 50, 4 bits 62, groups
// tested as a whole and resumed after the first shift 42-56, a next product
// for either outcome of the test 46-52, shifts of two bytes in the group as
// well 17 % more.  get(k) is the group's entry k in
// unrolled code, again(k) the same in a loop.
constexpr int kCoderGroup = 16;

template <class Get, class Again>
__device__ __forceinline__ void coder_group(Get get, Again again, uint32_t &x1, uint32_t &x2, uint32_t &head, uint8_t *ring,
                                            uint32_t mask) {
  const uint32_t a1 = x1, a2 = x2, ahead = head;
  uint32_t least = 0xffffffffu;
CUCM_UNROLL
  for (int i = 0; i < kCoderGroup; i++) {
    const uint2 q = get(i);
    coder_narrow(q.x, q.y, x1, x2);
    const uint32_t c = x1 ^ x2;
    least = min(least, c);
    ring[head & mask] = (uint8_t)(x2 >> 24);
    const uint32_t s = c < 0x1000000u ? 8u : 0u;
    head += s >> 3;
    x1 <<= s;
    x2 = __funnelshift_l(0xffffffffu, x2, s);
  }
  if (least < 0x10000u) {
    x1 = a1;
    x2 = a2;
    head = ahead;
#pragma unroll 1
    for (int i = 0; i < kCoderGroup; i++) coder_step(again(i), x1, x2, head, ring, mask);
  }
}

// The same for entries that lie one after the other, 16-byte aligned.
__device__ __forceinline__ void coder_group_at(const uint2 *e, uint32_t &x1, uint32_t &x2, uint32_t &head,
                                               uint8_t *ring, uint32_t mask) {
  coder_group(
      [&](int k) {
        const uint4 v = reinterpret_cast<const uint4 *>(e)[k >> 1];
        return k & 1 ? make_uint2(v.z, v.w) : make_uint2(v.x, v.y);
      },
      [&](int k) { return e[k]; }, x1, x2, head, ring, mask);
}

// Codes n entries into the shared-memory ring: group(j) takes entries
// j .. j + 15, entry(j) one.  All 32 lanes of the calling warp run the same
// arithmetic on the same data (and store the same bytes), so the control flow
// stays warp-uniform.  The ring never overruns: at most 4 bytes per bit are
// produced and at least stage - 4U bytes are free.
template <class Group, class Entry>
__device__ __forceinline__ void coder_run(Coder &c, uint8_t *stage, int stage_size, int n, Group group, Entry entry) {
  const uint32_t mask = (uint32_t)stage_size - 1;
  uint32_t x1 = c.x1, x2 = c.x2;
  uint32_t head = (uint32_t)c.head;
  const uint32_t head0 = head;
  int j = 0;
#pragma unroll 1
  for (; j + kCoderGroup <= n; j += kCoderGroup) group(j, x1, x2, head, mask);
#pragma unroll 1
  for (; j < n; j++) coder_step(entry(j), x1, x2, head, stage, mask);
  c.x1 = x1;
  c.x2 = x2;
  c.head += (uint32_t)(head - head0);
  __syncwarp();
}

// Entries as the mixing warps leave them (16-byte aligned).
__device__ __forceinline__ void coder_run_p(Coder &c, const uint2 *prm, uint8_t *stage, int stage_size, int n) {
  coder_run(
      c, stage, stage_size, n,
      [&](int j, uint32_t &x1, uint32_t &x2, uint32_t &head, uint32_t mask) {
        coder_group_at(prm + j, x1, x2, head, stage, mask);
      },
      [&](int j) { return prm[j]; });
}

// Warp-wide copy of complete 512-byte blocks from the ring to global.
__device__ inline void coder_flush_p(Coder &c, const uint8_t *stage, int stage_size, uint8_t *out, uint64_t cap) {
  const int lane = threadIdx.x & 31;
  const uint32_t mask = (uint32_t)stage_size - 1;
  while (c.head - c.flushed >= kFlushBlock) {
    if (c.flushed + kFlushBlock <= cap) {
      const uint32_t src = ((uint32_t)c.flushed & mask) + lane * 16;
      const uint4 v = *reinterpret_cast<const uint4 *>(stage + src);
      *reinterpret_cast<uint4 *>(out + c.flushed + lane * 16) = v;
    }
    c.flushed += kFlushBlock;
  }
  __syncwarp();
}

__device__ inline void coder_finish_p(Coder &c, uint8_t *stage, int stage_size, uint8_t *out, uint64_t cap,
                                      uint64_t *result) {
  const int lane = threadIdx.x & 31;
  const uint32_t mask = (uint32_t)stage_size - 1;
  if (lane == 0) stage[(uint32_t)c.head & mask] = (uint8_t)(c.x1 >> 24);  // flush byte, cucm_compress_v2.cu:902
  __syncwarp();
  c.head += 1;
  coder_flush_p(c, stage, stage_size, out, cap);
  for (uint64_t i = c.flushed + lane; i < c.head; i += 32)
    if (i < cap) out[i] = stage[(uint32_t)i & mask];
  if (lane == 0) *result = c.head;
  __syncwarp();
}

// Kernels with one thread per chunk's coder.  Its bytes go through a small
// ring of its own in shared memory (rows 4 bytes apart in the banks) and out in
// bursts, for all of a warp's lanes together.
constexpr int kLaneRing = 256;

__device__ __forceinline__ uint8_t *lane_ring(uint8_t *rings, int lane) { return rings + lane * (kLaneRing + 4); }

// Writes ring bytes [from, head) to out + base and starts the next burst;
// base moves on in steps of the ring, so head and from stay small.
__device__ __forceinline__ void lane_flush(const uint8_t *ring, uint64_t &base, uint32_t &from, uint32_t &head,
                                           uint8_t *out, uint64_t cap) {
#pragma unroll 4
  for (; from != head; from++)
    if (base + from < cap) out[base + from] = ring[from & (kLaneRing - 1)];
  base += head & ~(uint32_t)(kLaneRing - 1);
  head = from = head & (kLaneRing - 1);
}
__device__ __forceinline__ bool lane_flush_due(uint32_t from, uint32_t head) {
  return __any_sync(__activemask(), head - from >= 64);
}
