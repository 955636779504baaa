// decompress_wide.cuh -- chunk decoder for calls with few chunks: an SM per
// chunk, a byte per memory round trip.  Units of 32..256 bits.
//
// Included by engine_kernels.cu after decompress_fast.cuh (same records, model
// update and unit end).
//
// The pair decoder waits for one round of gathers per nibble, ~1,450 of its
// ~2,290 cycles, and a chunk has no other work to fill the wait with.  Where
// the call has fewer chunks than the device has SMs, the second nibble's tree
// is gathered with the first one's: a warp for each of the 16 first nibbles
// takes the 15 nodes below it, if the chunk's order-1 model, which is in shared
// memory, thinks it likely enough.  When the decoding warp knows the first
// nibble, that nibble's warp has its predictions, and the byte costs one round
// trip instead of two.
//
//   warp 0 (decoding): the pair decoder's, a byte at a time: first nibble as
//     there, second from the predictions of that nibble's warp; a first nibble
//     that was not followed has its second gathered and predicted here;
//   warps 1..16 (one per first nibble): keys, gathers and predictions of the
//     second nibble's nodes; the one that was right records the decoded path;
//   warp 17 (updating): the pair decoder's.
//
// A byte costs up to 1,530 random lines against the pair's 180, of which the
// device serves ~25 a cycle, so this is for few chunks only: see
// kWideMaxChunks.

constexpr int kWideWarps = 18, kWideThreads = kWideWarps * 32;
constexpr int kWideGuess = kDecNodes + 1;  // first nibbles

// Chunks in flight up to which a call's chunks get an SM each.  Text in chunks
// of 16 KiB, against the pair decoder: 1.22 times as fast with one chunk, 1.24
// with 16, 1.17 with 64, 1.04 with 96, 0.92 with 148 (random bytes 0.96, 0.97,
// 0.94 with 1, 16, 64).
constexpr uint32_t kWideMaxChunks = 64;

// Least probability, by the order-1 model, of a first nibble that is followed:
// a little above 1 in 16, so that nothing is followed where all look alike.  16
// chunks of 16 KiB, ms with 0.03 / 0.065 / 0.1 / 0.15: text 30.9 / 31.1 / 32.0 /
// 36.9 (the pair decoder 39.0), random bytes 39.7 / 40.1 / 44.1 / 44.3 (39.0),
// int32 walk 33.6 / 33.4 / 33.9 / 34.1 (38.6), runs 22.5 / 22.3 / 22.1 / 22.1
// (24.2); of 64 chunks, random bytes 49.3 / 42.9 / 45.1 / 45.1 (40.1).
constexpr float kWideLeast = 0.065f;

struct WideSmem {
  uint32_t f[kWideGuess][kDecNodes + 1];  // predictions << 20 of the nodes below each first nibble
  uint32_t ready[kWideGuess];             // 2 * byte + 1 when they are there, 2 * byte + 2 when not followed
  uint32_t byte[kWidePlaces];             // the last bytes decoded, byte n in place n % kWidePlaces
};

// Byte nth is known (wide_crossing.h): the decoding warp arrives and goes on, or
// waits too where its wait for a `ready` has run out.
__device__ __forceinline__ void wide_byte_arrive(uint32_t nth) {
  asm volatile("bar.arrive %0, %1;" ::"r"(1 + nth % kWideBarriers), "n"(32 * (1 + kWideGuess)) : "memory");
}
__device__ __forceinline__ void wide_byte_wait(uint32_t nth) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + nth % kWideBarriers), "n"(32 * (1 + kWideGuess)) : "memory");
}

// Whether first nibble `guess` after byte c1 is likely enough, by the order-1
// model alone (lane & 3 = bit).
__device__ __forceinline__ bool wide_follow(const DecSmem &s, const Tables *tab, uint32_t guess, uint32_t c1,
                                            int lane) {
  const int i = lane & 3;
  const uint32_t h0 = (1u << i) | (guess >> (4 - i));
  const uint32_t state = s.t01[kOrder1Off + ((c1 << 8) | h0)];
  const int x = s.spf[4 * kDecSpfRow + state];  // column 4 is order 1
  const int p1 = tab->squash[x + 2047];
  float p = (float)(((guess >> (3 - i)) & 1u) ? p1 : 4096 - p1) * (1.0f / 4096.0f);
  p *= __shfl_xor_sync(0xffffffffu, p, 1);
  p *= __shfl_xor_sync(0xffffffffu, p, 2);
  return p > kWideLeast;
}

__device__ void decompress_wide_one(const ChunkTask &t, uint8_t *slot, const DecSmem &s, WideSmem &ws,
                                    const Tables *tab, const DecLayout &L, const ModelInit *init, uint32_t *status,
                                    uint32_t spin_limit) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int U = L.U;
  const uint64_t len = t.out_cap < t.cs ? t.out_cap : t.cs;  // bytes to decode
  const uint64_t nbits = 8ull * len;
  const uint8_t *pay = t.in;
  const uint64_t plen = t.in_len;

  dec_start<true, kWideThreads>(s, L, tab, init, slot, tid);
  if (tid < kWideGuess) ws.ready[tid] = 0;
  if (tid == 0) {
    s.prog[0] = 0;  // bytes whose first nibble is recorded
    s.prog[2] = 0;  // bytes whose second nibble is
  }
  __syncthreads();

  const bool decodes = warp == 0, updates = warp == kWideWarps - 1;
  DecCoder c;
  if (decodes) dec_open(c, s.win, pay, plen, lane);
  const DecLane<true> ln(s, slot, lane);
  const uint32_t guess = (uint32_t)(warp - 1);  // of a guessing warp
  volatile uint32_t *ready = ws.ready;
  uint32_t hist[7] = {0, 0, 0, 0, 0, 0, 0};
  uint32_t kk[4], st[4];
  uint32_t bytes = 0;  // bytes before this unit (wraps; only compared for equality or order within the chunk)
  bool ok = true;

  for (uint64_t base = 0; base < nbits; base += (uint64_t)U) {
    const int nunit = (int)(nbits - base < (uint64_t)U ? nbits - base : (uint64_t)U);
    const int nb = nunit >> 3;
    if (decodes) {
      ln.gather(0, 0, hist, kk, st);
      uint32_t next = dec_ahead(c, s.win, pay, plen, lane);
      for (int b = 0; b < nb; b++) {
        const uint32_t nth = bytes + (uint32_t)b, seq = 2 * nth;
        int smp[4], cxt;
        uint32_t pr = ln.predict(s, tab->squash, st, hist[0], smp, cxt);
        DecPath path;
        const uint32_t hi = dec_nibble(c, path, pr << 20, next, s.win, lane);
        const DecRecord first = dec_record(ln, kk, st, smp, pr, cxt, hi);
        dec_settle(c, path, s.win);
        next = dec_ahead(c, s.win, pay, plen, lane);
        // the predictions below it
        uint32_t have, f_node;
        const bool seen = dec_wait([&] { return (have = ready[hi]) == seq + 1 || have == seq + 2; },
                                   ok ? spin_limit : 1, [&] { f_node = ws.f[hi][lane & 15]; });
        ok = ok && seen;
        const bool followed = seen && have == seq + 1;
        if (!followed) {  // not followed, and there it is
          ln.gather(hi, 4, hist, kk, st);
          pr = ln.predict(s, tab->squash, st, hist[0], smp, cxt);
          f_node = pr << 20;
        }
        const uint32_t lo = dec_nibble(c, path, f_node, next, s.win, lane);
        if (!followed) dec_write_record(s, ln, dec_record(ln, kk, st, smp, pr, cxt, lo), 2 * b + 1);
        const uint32_t byte = (hi << 4) | lo;
        if (lane == 0) ws.byte[nth % kWidePlaces] = byte;
        __syncwarp();
        if (ok)
          wide_byte_arrive(nth);
        else
          wide_byte_wait(nth);
        dec_push(hist, byte);
        if (b + 1 < nb) ln.gather(0, 0, hist, kk, st);
        dec_settle(c, path, s.win);
        next = dec_ahead(c, s.win, pay, plen, lane);
        dec_write_record(s, ln, first, 2 * b);
        if (lane == 0) s.outb[b] = (uint8_t)byte;
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          s.prog[0] = nth + 1;
        }
      }
    } else if (!updates) {
      for (int b = 0; b < nb; b++) {
        const uint32_t nth = bytes + (uint32_t)b, seq = 2 * nth;
        const bool follow = wide_follow(s, tab, guess, hist[0], lane);
        int smp[4], cxt = 0;
        uint32_t pr = 0;
        if (follow) {
          ln.gather(guess, 4, hist, kk, st);
          pr = ln.predict(s, tab->squash, st, hist[0], smp, cxt);
          if (lane < kDecNodes) ws.f[guess][lane] = pr << 20;
        }
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          ready[guess] = seq + (follow ? 1 : 2);
        }
        wide_byte_wait(nth);
        const uint32_t byte = ws.byte[nth % kWidePlaces];
        if ((byte >> 4) == guess) {
          // the warp of the nibble that came records its path (the decoding warp
          // has, where it was not followed) and says so: the word only grows, since
          // the last byte's warp wrote it before it came to this crossing
          if (follow) dec_write_record(s, ln, dec_record(ln, kk, st, smp, pr, cxt, byte & 15u), 2 * b + 1);
          __syncwarp();
          if (lane == 0) {
            __threadfence_block();
            s.prog[2] = nth + 1;
          }
        }
        dec_push(hist, byte);
      }
    } else {
      for (int rd = 0; rd < (nunit >> 2); rd++) {
        const uint32_t done = bytes + (uint32_t)(rd >> 1);
        volatile uint32_t *prog = s.prog + (rd & 1 ? 2 : 0);
        ok = ok && dec_wait([&] { return (int32_t)(*prog - done) > 0; }, spin_limit);
        if (!ok) break;
        dec_update_round(s, tab, L, lane, rd);
      }
    }
    if (!ok && lane == 0) atomicOr(status, (uint32_t)kDevTimeout);
    __syncthreads();
    dec_unit_end<kWideThreads>(s, L, tab, slot, t.out + (base >> 3), nunit, tid);
    __syncthreads();
    bytes += (uint32_t)nb;
  }
}

// One chunk per CTA at a time, from the work queue.
__global__ void __launch_bounds__(kWideThreads, 1)
    decompress_wide_kernel(const ChunkTask *tasks, uint32_t ntasks, uint8_t *slots, const uint8_t *init_tables,
                           const ModelInit *init, uint32_t *queue, uint32_t *status, int unit, uint32_t spin_limit) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ WideSmem ws;
  __shared__ uint32_t s_task;
  const DecLayout L = make_dec_layout(unit, 1, true);
  Tables *tab = reinterpret_cast<Tables *>(smem_raw + L.off_tab);
  copy_tables(&g_tables, tab);
  __syncthreads();
  for (int i = threadIdx.x; i < 4096; i += blockDim.x) tab->squash[i] += tab->squash[i] < 2048;  // see dec_mix
  const DecSmem s = carve_dec(smem_raw, L, 0);
  uint8_t *slot = slots + (size_t)blockIdx.x * kSlotTableBytes;
  bool fresh = true;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_task = atomicAdd(queue, 1u);
    __syncthreads();
    const uint32_t ti = s_task;
    if (ti >= ntasks) break;
    const ChunkTask t = tasks[ti];
    if (t.unit != (uint32_t)unit || t.cs == 0) {
      if (threadIdx.x == 0) atomicOr(status, (uint32_t)kDevBadTask);
      continue;
    }
    if (!fresh) {
      reset_slot(slot, init_tables);
      __syncthreads();
    }
    fresh = false;
    decompress_wide_one(t, slot, s, ws, tab, L, init, status, spin_limit);
  }
}
