// fixed_model.cuh -- the fixed-model variant (the paper's section 4.5).
//
// Included by engine_kernels.cu (shares its tables).
//
// The paper discusses, and measures, keeping CuCM's model fixed after the
// prelearn pass: no StateMap or Mixer update while the data is coded.  The
// reference ships no code for it; this build defines its stream (container
// flag bit 1): every data bit of a chunk is predicted by the prelearned
// model as the prelearn pass predicts (keys over the chunk's own history,
// StateMaps, Mixer -- cucm_compress_v2.cu:930-955) and coded with the
// reference's binary coder; only the data bits are coded (no stale tail),
// then the flush byte.
//
// Nothing is written during coding, so one copy of the model serves every
// chunk: the slot image (192 MiB, read through the read-only cache and L2),
// and per CTA in shared memory the stretched probabilities of the 256
// states of each order and the 640 mixer weights.  That makes the variant
// two kernels instead of a pipeline:
//
//   fixed_prob_kernel   one thread per input byte computes its 8 bits'
//                       coder inputs (pr << 1 | y) -- every bit of every
//                       chunk in parallel -- into a u16 array;
//   fixed_coder_kernel  one thread per chunk runs the arithmetic coder over
//                       its chunk's array, or, while every chunk can have a
//                       warp scheduler of its own, a warp
//                       (fixed_coder_warp_kernel);
//
// and the decoder gives each chunk a warp, a nibble per round, or in calls with
// no more chunks than SMs a CTA, a byte per round.

constexpr int kFixedThreads = 256;

struct FixedSmem {
  int16_t spf[256 * kOrders];  // stretched statep of the model, [state][order]
  int32_t w[kMixCtx * kOrders];
  uint16_t squash[4096];
};

__device__ inline void fixed_load_model(FixedSmem *f, const ModelInit *init) {
  for (int i = threadIdx.x; i < 256 * kOrders; i += blockDim.x)
    f->spf[i] = g_tables.stretch[init->statep[i & 7][i >> 3] >> 20];
  for (int i = threadIdx.x; i < kMixCtx * kOrders; i += blockDim.x) f->w[i] = init->w[i];
  for (int i = threadIdx.x; i < 4096; i += blockDim.x) f->squash[i] = g_tables.squash[i];
}

// The state of one order's key in the read-only slot image.
__device__ __forceinline__ uint32_t fixed_state(const uint8_t *image, int o, uint32_t key) {
  return __ldg(image + table_offset(o) + key);
}

// Mixer output (Mixer::p, cucm_compress_v2.cu:636-644, then pr++ below 2048)
// for the stretched inputs of one bit.
__device__ __forceinline__ int fixed_mix(const FixedSmem *f, const int smp[kOrders], int c1) {
  int olen = 0;
CUCM_UNROLL
  for (int o = 0; o < kOrders; o++) olen += smp[o] != 1;
  const int cxt = olen + (c1 >> 5) * 10;
  long long sum = 0;
CUCM_UNROLL
  for (int o = 0; o < kOrders; o++) sum += (long long)f->w[cxt * kOrders + o] * smp[o];
  sum >>= 16;
  const int idx = sum < -2047 ? -2047 : (sum > 2048 ? 2048 : (int)sum);
  const int pr = f->squash[idx + 2047];
  return pr < 2048 ? pr + 1 : pr;
}

// Thread = (task, byte): each CTA pass covers 256 consecutive bytes of all
// the tasks' bytes laid end to end.  `first` holds each task's first index in
// that sequence (prefix sums of the chunk lengths), `total` its length.
__global__ void __launch_bounds__(kFixedThreads)
    fixed_prob_kernel(const FixedTask *tasks, const uint64_t *first, uint32_t ntasks, uint64_t total,
                      const uint8_t *image, const ModelInit *init) {
  __shared__ FixedSmem f;
  __shared__ uint32_t s_task;
  fixed_load_model(&f, init);
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < total; base += (uint64_t)gridDim.x * blockDim.x) {
    __syncthreads();
    if (threadIdx.x == 0) {  // the task holding byte `base`
      uint32_t lo = 0, hi = ntasks - 1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (first[mid] <= base) lo = mid; else hi = mid - 1;
      }
      s_task = lo;
    }
    __syncthreads();
    const uint64_t gi = base + threadIdx.x;
    if (gi >= total) continue;
    uint32_t ti = s_task;
    while (ti + 1 < ntasks && first[ti + 1] <= gi) ti++;
    const FixedTask &t = tasks[ti];
    const uint64_t q = gi - first[ti];
    const uint8_t *in = t.in;
    uint32_t hist[7];
CUCM_UNROLL
    for (int i = 0; i < 7; i++) hist[i] = q > (uint64_t)i ? __ldg(in + q - 1 - i) : 0u;
    const uint32_t cur = __ldg(in + q);
    uint16_t e[8];
CUCM_UNROLL
    for (int r = 0; r < 8; r++) {
      const uint32_t h0 = (1u << r) | (cur >> (8 - r));
      BitKeys kk;
      bit_keys(h0, hist, kk);
      int smp[kOrders];
CUCM_UNROLL
      for (int o = 0; o < kOrders; o++) smp[o] = f.spf[fixed_state(image, o, kk.k[o]) * kOrders + o];
      const int pr = fixed_mix(&f, smp, (int)hist[0]);
      e[r] = (uint16_t)((pr << 1) | ((cur >> (7 - r)) & 1u));
    }
    uint4 v;
    v.x = e[0] | ((uint32_t)e[1] << 16);
    v.y = e[2] | ((uint32_t)e[3] << 16);
    v.z = e[4] | ((uint32_t)e[5] << 16);
    v.w = e[6] | ((uint32_t)e[7] << 16);
    *reinterpret_cast<uint4 *>(t.prm + 8 * q) = v;
  }
}

// Warp = task: the coder as in the adaptive compressor, all lanes alike.  The
// lanes turn 32 bytes' inputs into the coder's entries side by side and write
// the bytes out together; a thread that does both beside its chain of bits is
// bound by the instructions it issues and takes 78 cycles a bit against 53, more
// than the 71 of a test after every bit.  Text, both kernels of the variant, ms
// with a test after every bit / a thread / a warp: one chunk of 64 KiB 19.1 /
// 20.9 / 13.9, 128 chunks of 16 KiB 9.1 / 6.4 / 4.6.
constexpr int kFixedStage = 2048;  // 32 bytes code at most 1 KiB; flushes go out in 512-byte blocks

__global__ void __launch_bounds__(32)
    fixed_coder_warp_kernel(const FixedTask *tasks, uint32_t *status) {
  __shared__ uint4 ent[32 * 4];
  __shared__ __align__(16) uint8_t stage[kFixedStage];
  const int lane = threadIdx.x;
  const FixedTask t = tasks[blockIdx.x];
  const uint4 *src = reinterpret_cast<const uint4 *>(t.prm);
  const uint64_t n = t.in_len;
  Coder c{0u, 0xffffffffu, 0, 0};
  auto load = [&](uint64_t p) { return p + lane < n ? __ldg(src + p + lane) : make_uint4(0, 0, 0, 0); };
  uint4 next = load(0);
  for (uint64_t p = 0; p < n; p += 32) {
    const uint32_t w[4] = {next.x, next.y, next.z, next.w};
CUCM_UNROLL
    for (int i = 0; i < 4; i++) {
      const uint2 a = coder_entry(w[i] & 0xffffu), b = coder_entry(w[i] >> 16);
      ent[4 * lane + i] = make_uint4(a.x, a.y, b.x, b.y);
    }
    next = load(p + 32);
    __syncwarp();
    const int bytes = n - p < 32 ? (int)(n - p) : 32;
    coder_run_p(c, reinterpret_cast<const uint2 *>(ent), stage, kFixedStage, 8 * bytes);
    coder_flush_p(c, stage, kFixedStage, t.out, t.out_cap);
  }
  coder_finish_p(c, stage, kFixedStage, t.out, t.out_cap, t.result);
  if (lane == 0 && c.head > t.out_cap) atomicOr(status, (uint32_t)kDevOverflow);
}

// Thread = task: the binary coder over the chunk's coder inputs, two bytes'
// (16 bits, one coder_group) at a time, then the flush byte
// (cucm_compress_v2.cu:902) and the payload length.  The next two bytes'
// inputs are in flight while two are coded.  For more chunks than warp
// schedulers: 600 of 16 KiB of text, both kernels, 13.0 -> 10.4 ms against a
// test after every bit.
__global__ void __launch_bounds__(32) fixed_coder_kernel(const FixedTask *tasks, uint32_t ntasks, uint32_t *status,
                                                         int lanes) {
  __shared__ uint8_t rings[32 * (kLaneRing + 4)];
  const int lane = threadIdx.x;
  const uint32_t i = blockIdx.x * (uint32_t)lanes + lane;
  if (lane >= lanes || i >= ntasks) return;
  const FixedTask t = tasks[i];
  uint8_t *ring = lane_ring(rings, lane);
  uint32_t x1 = 0, x2 = 0xffffffffu;
  uint32_t head = 0, from = 0;
  uint64_t base = 0;  // payload offset of ring position 0
  const uint4 *src = reinterpret_cast<const uint4 *>(t.prm);
  const uint64_t n = t.in_len;
  uint4 nxt[4];
CUCM_UNROLL
  for (int b = 0; b < 4; b++) nxt[b] = (uint64_t)b < n ? __ldg(src + b) : make_uint4(0, 0, 0, 0);
  for (uint64_t p = 0; p < n; p += 2) {
    const uint4 cur[2] = {nxt[0], nxt[1]};
    nxt[0] = nxt[2];
    nxt[1] = nxt[3];
    nxt[2] = p + 4 < n ? __ldg(src + p + 4) : make_uint4(0, 0, 0, 0);
    nxt[3] = p + 5 < n ? __ldg(src + p + 5) : make_uint4(0, 0, 0, 0);
    const uint32_t w[8] = {cur[0].x, cur[0].y, cur[0].z, cur[0].w, cur[1].x, cur[1].y, cur[1].z, cur[1].w};
    const uint16_t *e = t.prm + 8 * p;
    auto again = [&](int k) { return coder_entry(e[k]); };
    if (p + 2 <= n)
      coder_group([&](int k) { return coder_entry((w[k >> 1] >> (16 * (k & 1))) & 0xffffu); }, again, x1, x2, head, ring,
                  kLaneRing - 1);
    else
      for (int k = 0; k < 8; k++) coder_step(again(k), x1, x2, head, ring, kLaneRing - 1);
    if (lane_flush_due(from, head)) lane_flush(ring, base, from, head, t.out, t.out_cap);
  }
  ring[head & (kLaneRing - 1)] = (uint8_t)(x1 >> 24);
  head++;
  lane_flush(ring, base, from, head, t.out, t.out_cap);
  base += head;
  *t.result = base;
  if (base > t.out_cap) atomicOr(status, (uint32_t)kDevOverflow);
}

// The decoders.  They use the adaptive decoder's lanes (DecLane) and coder
// (dec_nibble), so the model's stretched probabilities and weights sit in its
// layout in shared memory, once per CTA.
constexpr int kFixedDecWarps = 8;

// The model but its slot tables, in shared memory behind `kept`.
constexpr size_t kFixedDecSpf = sizeof(int16_t) * kOrders * kDecSpfRow, kFixedDecW = sizeof(int32_t) * kMixCtx * kOrders;
__device__ __forceinline__ void fixed_dec_model(uint8_t *kept, const ModelInit *init, DecSmem &s) {
  s.spf = reinterpret_cast<int16_t *>(kept);
  s.w = reinterpret_cast<int32_t *>(kept + kFixedDecSpf);
  for (int i = threadIdx.x; i < 256 * kOrders; i += blockDim.x)
    s.spf[(i >> 8) * kDecSpfRow + (i & 255)] = g_tables.stretch[init->statep[dec_order(i >> 8)][i & 255] >> 20];
  for (int i = threadIdx.x; i < kMixCtx * kOrders; i += blockDim.x) s.w[i] = init->w[(i & ~7) + dec_order(i & 7)];
}

// Warp = chunk (tasks handed out by a queue): a nibble per round, the next
// round's gathers issued as soon as one is decoded.  All chunks read the same
// tables, so the gathers go through L1 and everything else is kept small: 31 KB
// a CTA, four CTAs an SM, 100 KB of L1 beside them.  Text in chunks of 2 KiB,
// ms against order 0/1 tables in shared memory, gathers past L1 and two CTAs an
// SM: 149 chunks 4.5 and 4.5, 500 4.6 and 5.2, 1,184 5.5 and 10.1, 2,368 9.0 and
// 20.1, 4,736 18.8 and 40.1.
constexpr size_t kFixedDecSquash = kFixedDecSpf + kFixedDecW, kFixedDecWin = kFixedDecSquash + sizeof(uint16_t) * 4096;
inline size_t fixed_dec_smem_bytes(int warps) { return kFixedDecWin + (size_t)warps * kDecWin; }

__global__ void __launch_bounds__(kFixedDecWarps * 32, 4)
    fixed_decode_kernel(const FixedTask *tasks, uint32_t ntasks, const uint8_t *image, const ModelInit *init,
                        uint32_t *queue) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  DecSmem s;
  fixed_dec_model(smem_raw, init, s);
  uint16_t *squash = reinterpret_cast<uint16_t *>(smem_raw + kFixedDecSquash);
  for (int i = threadIdx.x; i < 4096; i += blockDim.x)  // see dec_mix
    squash[i] = g_tables.squash[i] + (g_tables.squash[i] < 2048);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint8_t *win = smem_raw + kFixedDecWin + warp * kDecWin;
  const DecLane<false, true> ln(s, image, lane);
  for (;;) {
    uint32_t ti = 0;
    if (lane == 0) ti = atomicAdd(queue, 1u);
    ti = __shfl_sync(0xffffffffu, ti, 0);
    if (ti >= ntasks) break;
    const FixedTask t = tasks[ti];
    DecCoder c;
    dec_open(c, win, t.in, t.in_len, lane);
    uint32_t hist[7] = {0, 0, 0, 0, 0, 0, 0};
    uint32_t cur = 0, kk[4], st[4];
    int r = 0;
    const uint64_t rounds = 2 * t.out_cap;
    if (rounds) ln.gather(cur, r, hist, kk, st);
    uint32_t next = dec_ahead(c, win, t.in, t.in_len, lane);
    for (uint64_t rd = 0; rd < rounds; rd++) {
      int smp[4], cxt;
      const uint32_t pr = ln.predict(s, squash, st, hist[0], smp, cxt);
      DecPath path;
      const uint32_t nib = dec_nibble(c, path, pr << 20, next, win, lane);
      cur = (cur << 4) | nib;
      r += 4;
      if (r == 8) {
        if (lane == 0) t.out[rd >> 1] = (uint8_t)cur;
        dec_push(hist, cur);
        cur = 0;
        r = 0;
      }
      if (rd + 1 < rounds) ln.gather(cur, r, hist, kk, st);
      dec_settle(c, path, win);
      next = dec_ahead(c, win, t.in, t.in_len, lane);
    }
    __syncwarp();
  }
}

// CTA = chunk: a byte per round, the second nibble's nodes gathered with the
// first one's by a warp for each likely first nibble (decompress_wide.cuh, with
// nothing to update or record).
constexpr int kFixedWideThreads = 32 * (1 + kWideGuess);
constexpr size_t kFixedWideTab = kHashedOff, kFixedWideKept = kFixedWideTab + sizeof(Tables),
                 kFixedWideWin = kFixedWideKept + kFixedDecSpf + kFixedDecW, kFixedWideSmem = kFixedWideWin + kDecWin;

__global__ void __launch_bounds__(kFixedWideThreads, 1)
    fixed_decode_wide_kernel(const FixedTask *tasks, uint32_t ntasks, const uint8_t *image, const ModelInit *init,
                             uint32_t *queue) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ WideSmem ws;
  __shared__ uint32_t s_task;
  DecSmem s;
  s.t01 = smem_raw;
  Tables *tab = reinterpret_cast<Tables *>(smem_raw + kFixedWideTab);
  copy_tables(&g_tables, tab);
  const uint4 *src = reinterpret_cast<const uint4 *>(image);
  for (int i = threadIdx.x; i < (int)(kHashedOff / 16); i += blockDim.x) reinterpret_cast<uint4 *>(s.t01)[i] = src[i];
  fixed_dec_model(smem_raw + kFixedWideKept, init, s);
  __syncthreads();
  for (int i = threadIdx.x; i < 4096; i += blockDim.x) tab->squash[i] += tab->squash[i] < 2048;  // see dec_mix
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint8_t *win = smem_raw + kFixedWideWin;
  const DecLane<true> ln(s, image, lane);
  volatile uint32_t *ready = ws.ready;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_task = atomicAdd(queue, 1u);
    if (tid < kWideGuess) ws.ready[tid] = 0;
    __syncthreads();
    const uint32_t ti = s_task;
    if (ti >= ntasks) break;
    const FixedTask t = tasks[ti];
    uint32_t hist[7] = {0, 0, 0, 0, 0, 0, 0};
    uint32_t kk[4], st[4];
    int smp[4], cxt;
    if (warp == 0) {
      DecCoder c;
      dec_open(c, win, t.in, t.in_len, lane);
      if (t.out_cap) ln.gather(0, 0, hist, kk, st);
      uint32_t next = dec_ahead(c, win, t.in, t.in_len, lane);
      for (uint64_t b = 0; b < t.out_cap; b++) {
        const uint32_t seq = 2 * (uint32_t)b;
        uint32_t pr = ln.predict(s, tab->squash, st, hist[0], smp, cxt);
        DecPath path;
        const uint32_t hi = dec_nibble(c, path, pr << 20, next, win, lane);
        dec_settle(c, path, win);
        next = dec_ahead(c, win, t.in, t.in_len, lane);
        // ends with its warp's gathers, long before the bound; past it the nibble
        // is predicted here, with the same result, so there is nothing to report.
        // (No vote on the outcome, as warp_wait takes where a caller can set the
        // bound: 2 % of this kernel, 16.2 -> 16.6 ms for 8 KiB of random bytes.)
        uint32_t spins = 0, have;
        while ((have = ready[hi]) != seq + 1 && have != seq + 2)
          if (++spins >= kDecSpinLimit) break;
        __threadfence_block();
        uint32_t f_node = ws.f[hi][lane & 15];
        if (have != seq + 1) {
          ln.gather(hi, 4, hist, kk, st);
          pr = ln.predict(s, tab->squash, st, hist[0], smp, cxt);
          f_node = pr << 20;
        }
        const uint32_t lo = dec_nibble(c, path, f_node, next, win, lane);
        const uint32_t byte = (hi << 4) | lo;
        if (lane == 0) ws.byte[b % kWidePlaces] = byte;
        __syncwarp();
        if (spins < kDecSpinLimit)
          wide_byte_arrive((uint32_t)b);
        else
          wide_byte_wait((uint32_t)b);
        dec_push(hist, byte);
        if (b + 1 < t.out_cap) ln.gather(0, 0, hist, kk, st);
        dec_settle(c, path, win);
        next = dec_ahead(c, win, t.in, t.in_len, lane);
        if (lane == 0) t.out[b] = (uint8_t)byte;
      }
    } else {
      const uint32_t guess = (uint32_t)(warp - 1);
      for (uint64_t b = 0; b < t.out_cap; b++) {
        const bool follow = wide_follow(s, tab, guess, hist[0], lane);
        if (follow) {
          ln.gather(guess, 4, hist, kk, st);
          const uint32_t pr = ln.predict(s, tab->squash, st, hist[0], smp, cxt);
          if (lane < kDecNodes) ws.f[guess][lane] = pr << 20;
        }
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          ready[guess] = 2 * (uint32_t)b + (follow ? 1 : 2);
        }
        wide_byte_wait((uint32_t)b);
        dec_push(hist, ws.byte[b % kWidePlaces]);
      }
    }
  }
}
