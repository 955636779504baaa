// decompress_fast.cuh -- chunk decoder, two warps per chunk, units of 32..256 bits.
//
// Included by engine_kernels.cu (shares its tables and helpers).
//
// The reference decodes a unit in speculation steps of L+1 bits, each step
// three launches and a host round trip (cucm_decompress_v2.cu:977-1032).
// Here a pair of warps owns a chunk and decodes it a nibble ("round") at a
// time.
//
// The decoding warp:
//   * gives the 15 nodes of the nibble's speculation tree (every prefix of
//     0..3 bits) their 8 context keys and frozen slot states -- two lanes per
//     node, the even and the odd orders, the 6 hashed orders' gathers in
//     flight together (orders 0 and 1 come from shared memory for a chunk alone
//     in its CTA), so a round costs one memory round trip;
//   * mixes and squashes each node's prediction against the frozen model
//     (probabilities kept stretched) and decodes the 4 bits, a lane per leaf of
//     the tree (dec_nibble);
//   * issues the next round's gathers, then has the lanes on the decoded path
//     record keys, states and mixer inputs of their bit in a per-unit ring,
//     and publishes the round.
// The updating warp follows, polling for published rounds, all four bits and
// eight orders of a round at once (dec_update_round): live states through a
// hash of the unit's keys, the StateMap probabilities and the mixer deltas.
// Nothing the decoding warp reads changes before the unit ends, so the two
// only meet there: the unit's last state of every slot goes to the slot
// tables, the live probabilities become the frozen ones and the summed mixer
// deltas join the weights (updateStateMap / updateMixer,
// cucm_decompress_v2.cu:870-896).  Rounds never straddle a unit or byte
// boundary: units are multiples of 32 bits.
//
// A round of one of 16 chunks takes 2,290 cycles: ~1,450 from the first gather
// to the last byte back (a single random gather from HBM takes 900, the
// slowest of 90 about 1,450; with 256 chunks ~1,800), ~360 to decode, ~250 for
// the next keys and gathers, ~160 to mix; recording and the coder state's
// broadcast run under the gathers.
//
// Several warp pairs of a CTA decode independent chunks and share the
// read-only tables.

constexpr int kDecMaxUnit = 256;
constexpr int kDecMaxPairs = 8;          // chunks per CTA (5 for units above 64 bits: 740 chunks' tables are 142 GB)
constexpr int kDecWin = 2048;            // payload window per chunk (bytes)
constexpr int kDecNodes = 15;            // nodes of a 4-bit speculation tree
constexpr size_t kDecSmemLimit = 227 * 1024;  // dynamic shared memory of one CTA
constexpr uint32_t kDecSpinLimit = 1u << 27;  // default bound on the updater's polls for a round (seconds)

// Everything a chunk keeps per order -- probabilities, weights, records -- is
// in columns: even orders in columns 0..3, odd ones in 4..7, the halves that
// the decoding warp's half warps take.
__host__ __device__ constexpr int dec_order(int col) { return 2 * (col & 3) + (col >> 2); }

// Row lengths of the [column][state] arrays: the columns' rows start in
// different banks.
constexpr int kDecSplRow = 260, kDecSpfRow = 264;
constexpr uint32_t kDecNone = 0xffu;  // no position (positions that are looked up end at 251)

struct DecLayout {
  int U, NT, logNT, warps, rounds;
  bool low;  // order 0/1 tables held in shared memory
  size_t off_spf, off_spl, off_w, off_dw, off_ovt, off_och, off_ons, off_prog, off_rk, off_rs, off_rsmp, off_rpc,
      off_win, off_outb, off_t01, per_warp, off_tab, total;
};

// Shared memory of `warps` chunks (warp pairs) and the shared tables.
// With `low`, each chunk also holds its order 0 and 1 tables (the first
// kHashedOff bytes of its slot, 64.25 KiB) in shared memory.
__host__ __device__ inline DecLayout make_dec_layout(int U, int warps, bool low = false) {
  DecLayout L;
  L.U = U;
  L.low = low;
  L.rounds = U / 4;
  L.NT = next_pow2(2 * U);
  L.logNT = ilog2(L.NT);
  L.warps = warps;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    size_t at = o;
    o = (o + bytes + 15) & ~(size_t)15;
    return at;
  };
  L.off_spf = take(sizeof(int16_t) * kOrders * kDecSpfRow);    // frozen probability, stretched [column][state]
  L.off_spl = take(sizeof(uint32_t) * kOrders * kDecSplRow);   // live statep [column][state]
  L.off_w = take(sizeof(int32_t) * kMixCtx * kOrders);         // frozen weights
  L.off_dw = take(sizeof(int32_t) * kMixCtx * kOrders);        // summed deltas of the unit
  L.off_ovt = take((size_t)kOrders * L.NT);                    // last position with a key hash [column][hash]
  L.off_och = take((size_t)U * kOrders);                       // position before it with that hash [bit][column]
  L.off_ons = take((size_t)U * kOrders);                       // state the bit left in its slot [bit][column]
  L.off_prog = take(sizeof(uint32_t) * 4);                     // rounds published; task index
  L.off_rk = take(sizeof(uint32_t) * L.rounds * 4 * kOrders);  // records [round][bit][column]
  L.off_rs = take((size_t)L.rounds * 4 * kOrders);
  L.off_rsmp = take(sizeof(int16_t) * L.rounds * 4 * kOrders);
  L.off_rpc = take(sizeof(uint32_t) * L.rounds * 4);           // pr | cxt << 16 | y << 24
  L.off_win = take((size_t)kDecWin);
  L.off_outb = take((size_t)kDecMaxUnit / 8);
  L.off_t01 = low ? take((size_t)kHashedOff) : 0;
  L.per_warp = o;
  L.off_tab = (size_t)warps * L.per_warp;
  L.total = L.off_tab + ((sizeof(Tables) + 15) & ~(size_t)15);
  return L;
}

struct DecSmem {
  int16_t *spf;
  uint32_t *spl;
  int32_t *w, *dw;
  uint8_t *ovt, *och, *ons;
  volatile uint32_t *prog;
  uint32_t *rk;
  uint8_t *rs;
  int16_t *rsmp;
  uint32_t *rpc;
  uint8_t *win, *outb;
  uint8_t *t01;  // order 0/1 tables, or null
};

__device__ inline DecSmem carve_dec(uint8_t *base, const DecLayout &L, int warp) {
  uint8_t *b = base + (size_t)warp * L.per_warp;
  DecSmem s;
  s.spf = reinterpret_cast<int16_t *>(b + L.off_spf);
  s.spl = reinterpret_cast<uint32_t *>(b + L.off_spl);
  s.w = reinterpret_cast<int32_t *>(b + L.off_w);
  s.dw = reinterpret_cast<int32_t *>(b + L.off_dw);
  s.ovt = b + L.off_ovt;
  s.och = b + L.off_och;
  s.ons = b + L.off_ons;
  s.prog = reinterpret_cast<volatile uint32_t *>(b + L.off_prog);
  s.rk = reinterpret_cast<uint32_t *>(b + L.off_rk);
  s.rs = b + L.off_rs;
  s.rsmp = reinterpret_cast<int16_t *>(b + L.off_rsmp);
  s.rpc = reinterpret_cast<uint32_t *>(b + L.off_rpc);
  s.win = b + L.off_win;
  s.outb = b + L.off_outb;
  s.t01 = L.low ? b + L.off_t01 : nullptr;
  return s;
}

// One slot state from the tables in HBM (L2-cached load).  The memory
// clobber keeps the load where it is written: a round's gathers go out
// before the previous round's record is stored to shared memory.
__device__ __forceinline__ uint32_t ld_slot_state(const uint8_t *p) {
  uint32_t v;
  asm volatile("ld.global.cg.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// One from tables that are never written: through L1, where chunks that read
// the same tables find each other's lines.
__device__ __forceinline__ uint32_t ld_kept_state(const uint8_t *p) {
  uint32_t v;
  asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Warp-wide refill of the payload window so that it starts at or just below
// payload byte `at`, on a 16-byte boundary of the payload's address (so the
// window base may lie up to 15 bytes before the payload).  Only 16-byte
// blocks that hold payload bytes are read; bytes past the payload are 255, as
// the reference's decoder shifts them in.  Returns the payload offset of window
// byte 0.
__device__ inline long long dec_refill(uint8_t *win, const uint8_t *pay, uint64_t plen, uint64_t at, int lane) {
  const uint8_t *a = reinterpret_cast<const uint8_t *>((reinterpret_cast<uintptr_t>(pay) + at) & ~(uintptr_t)15);
  const uint8_t *end = pay + plen;
  __syncwarp();  // (every lane has read what it needs of the old window)
  for (int j = lane; j < kDecWin / 16; j += 32) {
    const uint8_t *blk = a + 16 * j;
    uint4 v = make_uint4(~0u, ~0u, ~0u, ~0u);
    if (blk < end) {
      v = *reinterpret_cast<const uint4 *>(blk);
      const int have = end - blk < 16 ? (int)(end - blk) : 16;
      auto past = [&](int w) -> uint32_t {  // mask of word w's bytes past the payload
        const int n = have - 4 * w;
        return n >= 4 ? 0u : n <= 0 ? ~0u : ~0u << (8 * n);
      };
      v.x |= past(0);
      v.y |= past(1);
      v.z |= past(2);
      v.w |= past(3);
    }
    *reinterpret_cast<uint4 *>(win + 16 * j) = v;
  }
  __syncwarp();
  return (long long)(a - pay);
}

// The window's next four bytes from offset `at`, first byte highest.
__device__ __forceinline__ uint32_t dec_next4(const uint8_t *win, uint32_t at) {
  const uint32_t *w = reinterpret_cast<const uint32_t *>(win) + (at >> 2);
  return __byte_perm(__funnelshift_r(w[0], w[1], 8 * (at & 3)), 0, 0x0123);
}

// Coder state of a decoding warp, identical in every lane.
struct DecCoder {
  uint32_t x1, x2, x;
  uint64_t ioff;   // payload bytes taken
  long long wbase; // payload offset of the window's first byte
};

// Decodes 4 bits along the speculation tree (cucm_decompress_v2.cu:813-868)
// and returns them, first bit highest.  f_node: lane n (n < 15) holds node n's
// probability << 20; next: the payload's next four bytes.
//
// Lanes 0..15 (16..31 the same again) each run the coder down one leaf's path,
// taking its bits for granted and checking them against x on the side; one
// lane's check holds.  No step waits for a comparison, a shuffle or a branch: a
// bit shifts by 0 or 8, and where one of the first three has to shift further
// (seen in `least`) the nibble is decoded bit by bit instead.  The nibble is
// known before the path's state is: `settle` brings that to all lanes, once
// the next round's gathers are out.  Bit by bit the nibble took 340 cycles.
struct DecPath {
  uint32_t x1, x2, x, taken;  // of this lane's path, before the last bit's shift
  int leaf;                   // the path decoded, -1: the coder state is final already
};

__device__ __forceinline__ uint32_t dec_nibble(DecCoder &c, DecPath &w, uint32_t f_node, uint32_t next,
                                               const uint8_t *win, int lane) {
  const int p = lane & 15;
  uint32_t f[4];
  f[0] = __shfl_sync(0xffffffffu, f_node, 0);
  f[1] = __shfl_sync(0xffffffffu, f_node, 1 + (p >> 3));
  f[2] = __shfl_sync(0xffffffffu, f_node, 3 + (p >> 2));
  f[3] = __shfl_sync(0xffffffffu, f_node, 7 + (p >> 1));
  uint32_t x1 = c.x1, x2 = c.x2, x = c.x, nb = next, least = 0xffffffffu, taken = 0;
  bool ok = true;
CUCM_UNROLL
  for (int i = 0; i < 4; i++) {
    const uint32_t n = ((p >> (3 - i)) & 1) - 1u;  // all ones for a 0
    const uint32_t t = __umulhi(x2 - x1, f[i]);
    const uint32_t xm = x1 + t, xn = x1 + t + 1;
    ok = ok && ((x <= xm) == (n == 0u));
    x2 = (x2 & n) | (xm & ~n);
    x1 = (xn & n) | (x1 & ~n);
    if (i == 3) break;
    const uint32_t d = x1 ^ x2;
    least = min(least, d);
    const uint32_t s = d < 0x1000000u ? 8u : 0u;
    x1 <<= s;
    x2 = __funnelshift_l(0xffffffffu, x2, s);
    x = __funnelshift_l(nb, x, s);
    nb <<= s;
    taken += s;
  }
  const uint32_t hit = __ballot_sync(0xffffffffu, ok);
  const uint32_t far = __ballot_sync(0xffffffffu, ok && least < 0x10000u);
  // the lane with the check, in tests side by side (a find-first is ~20 cycles)
  const uint32_t leaf = ((hit & 0xff00u) ? 8u : 0u) | ((hit & 0xf0f0u) ? 4u : 0u) | ((hit & 0xccccu) ? 2u : 0u) |
                        ((hit & 0xaaaau) ? 1u : 0u);
  w.x1 = x1;
  w.x2 = x2;
  w.x = x;
  w.taken = taken;
  w.leaf = (int)leaf;
  if (!far) return leaf;
  uint32_t nib = 0;
  int n = 0;
#pragma unroll 1
  for (int i = 0; i < 4; i++) {
    const uint32_t xm = c.x1 + __umulhi(c.x2 - c.x1, __shfl_sync(0xffffffffu, f_node, n));
    const int y = c.x <= xm;
    if (y) c.x2 = xm; else c.x1 = xm + 1;
    while ((c.x1 ^ c.x2) < 0x1000000u) {
      c.x1 <<= 8;
      c.x2 = (c.x2 << 8) | 255u;
      c.x = (c.x << 8) | (uint32_t)win[(long long)c.ioff - c.wbase];
      c.ioff++;
    }
    nib = (nib << 1) | (uint32_t)y;
    n = 2 * n + 1 + y;
  }
  w.leaf = -1;
  return nib;
}

__device__ __forceinline__ void dec_settle(DecCoder &c, const DecPath &w, const uint8_t *win) {
  if (w.leaf < 0) return;
  c.x1 = __shfl_sync(0xffffffffu, w.x1, w.leaf);
  c.x2 = __shfl_sync(0xffffffffu, w.x2, w.leaf);
  c.x = __shfl_sync(0xffffffffu, w.x, w.leaf);
  c.ioff += __shfl_sync(0xffffffffu, w.taken, w.leaf) >> 3;
  while ((c.x1 ^ c.x2) < 0x1000000u) {  // the last bit's shift
    c.x1 <<= 8;
    c.x2 = (c.x2 << 8) | 255u;
    c.x = (c.x << 8) | (uint32_t)win[(long long)c.ioff - c.wbase];
    c.ioff++;
  }
}

// Model update of one round's 4 bits (lane = column lane & 7, bit lane >> 3):
// the live state of each slot (what an earlier bit of the unit left there, else
// the frozen state the prediction saw), its next state, the StateMap
// probability of the live state in bit order (cucm_decompress_v2.cu:870-883)
// and the mixer deltas (:885-896).
//
// A bit's key is looked up among the unit's earlier ones through a small hash
// of the last position per key hash, positions with the same hash chained
// backwards through och.  Nothing is cleared between units: a position at or
// past this round's is left from the unit before and ends a search, one before
// it holds a key of this unit, which is compared.  The four keys of a round
// and an order differ (they share the previous bytes; the hash is one-to-one
// in the partial byte), so the lookups do not depend on one another; only bits
// that meet the same state of the same order wait for each other.  A slot's
// earlier record is marked (bit 31 of its key): the unit end writes the
// unmarked ones.
//
// All shared-memory reads stand before the writes (the compiler keeps their
// order).  One lane per order, its four bits after one another, took 2,000
// cycles a round, more than the decoding warp's 120 gathers.
__device__ __forceinline__ void dec_update_round(const DecSmem &s, const Tables *tab, const DecLayout &L, int lane,
                                                 int rd) {
  const int o = lane & 7, i = lane >> 3;
  const uint32_t base = 4u * (uint32_t)rd, j = base + (uint32_t)i;
  const int r = 32 * rd + lane;
  const uint32_t k = s.rk[r];
  const uint32_t fz = s.rs[r];
  const int sm = s.rsmp[r];
  const uint32_t pc = s.rpc[4 * rd + i];
  const int y = (int)(pc >> 24) & 1, pr = (int)(pc & 0xffffu);
  const uint32_t cx = (pc >> 16) & 0xffu;
  const int delta = (int)(((long long)(((y << 12) - pr) * 7) * sm) >> 16);
  const uint32_t h = bucket_of(k, L.logNT);
  uint8_t *last = s.ovt + o * L.NT + h;
  const uint32_t p = *last;
  // the search: most end at the first position
  bool more = p < base;
  uint32_t q = more ? p : 0u, found = kDecNone;
  {
    const uint32_t kk = s.rk[q * kOrders + o], c = s.och[q * kOrders + o];
    if (more && kk == k) found = q;
    more = more && kk != k && c < q;
    q = more ? c : 0u;
  }
  while (__any_sync(0xffffffffu, more)) {
    const uint32_t kk = s.rk[q * kOrders + o], c = s.och[q * kOrders + o];
    if (more && kk == k) found = q;
    more = more && kk != k && c < q;
    q = more ? c : 0u;
  }
  const bool again = found != kDecNone;
  const uint32_t left = s.ons[(again ? found : 0u) * kOrders + o];
  const uint32_t live = again ? left : fz;
  const uint32_t next = tab->nex[live][y];
  uint32_t v = s.spl[o * kDecSplRow + live];
  // positions of this round with the same hash
  const uint32_t h0 = __shfl_sync(0xffffffffu, h, o), h1 = __shfl_sync(0xffffffffu, h, o + 8),
                 h2 = __shfl_sync(0xffffffffu, h, o + 16), h3 = __shfl_sync(0xffffffffu, h, o + 24);
  uint32_t before = p < base ? p : kDecNone;
  if (i > 0 && h0 == h) before = base;
  if (i > 1 && h1 == h) before = base + 1;
  if (i > 2 && h2 == h) before = base + 2;
  const bool last_of_hash = !((i < 1 && h1 == h) || (i < 2 && h2 == h) || (i < 3 && h3 == h));
  // a state met m times earlier in the round has count min(count + m, 1023)
  const uint32_t l0 = __shfl_sync(0xffffffffu, live, o), l1 = __shfl_sync(0xffffffffu, live, o + 8),
                 l2 = __shfl_sync(0xffffffffu, live, o + 16), l3 = __shfl_sync(0xffffffffu, live, o + 24);
  const bool e0 = i > 0 && l0 == live, e1 = i > 1 && l1 == live, e2 = i > 2 && l2 == live;
  const uint32_t m = (uint32_t)e0 + (uint32_t)e1 + (uint32_t)e2;
  const bool last_of_state = !((i < 1 && l1 == live) || (i < 2 && l2 == live) || (i < 3 && l3 == live));
  const uint32_t rate = tab->dt[min((v & 1023u) + m, 1023u)];
  uint32_t nv = statep_next(v, y, rate);
  if (__any_sync(0xffffffffu, m != 0)) {
    const uint32_t n0 = __shfl_sync(0xffffffffu, nv, o);
    v = e0 ? n0 : v;
    nv = statep_next(v, y, rate);
    const uint32_t n1 = __shfl_sync(0xffffffffu, nv, o + 8);
    v = e1 ? n1 : v;
    nv = statep_next(v, y, rate);
    const uint32_t n2 = __shfl_sync(0xffffffffu, nv, o + 16);
    v = e2 ? n2 : v;
    nv = statep_next(v, y, rate);
  }
  __syncwarp();  // everything is read
  // writes; where bits share a place, the last of them writes
  if (again) s.rk[found * kOrders + o] = k | 0x80000000u;
  s.ons[r] = (uint8_t)next;
  s.och[r] = (uint8_t)before;
  if (last_of_hash) *last = (uint8_t)j;
  if (last_of_state) s.spl[o * kDecSplRow + live] = nv;
  atomicAdd(&s.dw[cx * kOrders + o], delta);
  __syncwarp();
}

// Unit end, kThreads threads (t = 0..kThreads - 1): the slots' last states go
// to the slot tables, live probabilities become frozen (stretched for the
// mixer), deltas join the weights, the unit's bytes go out.  Called between two
// barriers.  Reads are issued in batches ahead of the writes.
template <int kThreads>
__device__ inline void dec_unit_end(const DecSmem &s, const DecLayout &L, const Tables *tab, uint8_t *slot,
                                    uint8_t *out, int nbits, int t) {
  constexpr int kSlots8 = kThreads >= 256 ? 2 : 8;  // slots of a thread's batch
  {
    const int o = dec_order(t & 7);
    uint8_t *tb = (o < 2 && s.t01 ? s.t01 : slot) + table_offset(o);
    for (int e0 = t; e0 < nbits * kOrders; e0 += kThreads * kSlots8) {
      uint32_t kk[kSlots8], ns[kSlots8];
CUCM_UNROLL
      for (int i = 0; i < kSlots8; i++) {
        const int e = e0 + kThreads * i;
        const bool in = e < nbits * kOrders;
        kk[i] = in ? s.rk[e] : 0x80000000u;
        ns[i] = in ? s.ons[e] : 0u;
      }
CUCM_UNROLL
      for (int i = 0; i < kSlots8; i++)
        if (!(kk[i] >> 31)) tb[kk[i]] = (uint8_t)ns[i];
    }
  }
  const int16_t *str = tab->stretch;
  constexpr int kQuads = kThreads >= 256 ? 1 : 4;  // groups of four states of a thread's batch
  for (int i0 = t; i0 < 64 * kOrders; i0 += kThreads * kQuads) {
    uint4 q[kQuads];
    uint2 d[kQuads];
CUCM_UNROLL
    for (int i = 0; i < kQuads; i++) {
      const int g = min(i0 + kThreads * i, 64 * kOrders - 1);
      q[i] = *reinterpret_cast<const uint4 *>(s.spl + (g >> 6) * kDecSplRow + 4 * (g & 63));
    }
CUCM_UNROLL
    for (int i = 0; i < kQuads; i++) {
      const uint32_t a = (uint16_t)str[q[i].x >> 20], b = (uint16_t)str[q[i].y >> 20];
      const uint32_t c = (uint16_t)str[q[i].z >> 20], e = (uint16_t)str[q[i].w >> 20];
      d[i] = make_uint2(a | (b << 16), c | (e << 16));
    }
CUCM_UNROLL
    for (int i = 0; i < kQuads; i++) {
      const int g = i0 + kThreads * i;
      if (g < 64 * kOrders) *reinterpret_cast<uint2 *>(s.spf + (g >> 6) * kDecSpfRow + 4 * (g & 63)) = d[i];
    }
  }
  int4 *w4 = reinterpret_cast<int4 *>(s.w);
  int4 *d4 = reinterpret_cast<int4 *>(s.dw);
  constexpr int kRows = (kMixCtx * kOrders / 4 + kThreads - 1) / kThreads;
  int4 a[kRows], d[kRows];
CUCM_UNROLL
  for (int i = 0; i < kRows; i++) {
    const int e = t + kThreads * i;
    if (e < kMixCtx * kOrders / 4) {
      a[i] = w4[e];
      d[i] = d4[e];
    }
  }
CUCM_UNROLL
  for (int i = 0; i < kRows; i++) {
    const int e = t + kThreads * i;
    if (e < kMixCtx * kOrders / 4) {
      w4[e] = make_int4(a[i].x + d[i].x, a[i].y + d[i].y, a[i].z + d[i].z, a[i].w + d[i].w);
      d4[e] = make_int4(0, 0, 0, 0);
    }
  }
  if (t < (nbits >> 3)) out[t] = s.outb[t];
}

// Mixer output of one node (Mixer::p, cucm_compress_v2.cu:636-644, then pr++
// below 2048, which the decoder's copy of the squash table already holds), the
// half warps with four orders each.  |sum| < 2^45, so sum >> 16 fits 32 bits.
__device__ __forceinline__ uint32_t dec_mix(const int32_t *w, int cxt, const int smp[4], int half,
                                            const uint16_t *squash) {
  const int4 a = reinterpret_cast<const int4 *>(w)[2 * cxt + half];
  const long long s0 = (long long)a.x * smp[0] + (long long)a.y * smp[1];
  const long long s1 = (long long)a.z * smp[2] + (long long)a.w * smp[3];
  long long sum = s0 + s1;
  const uint32_t lo = __shfl_xor_sync(0xffffffffu, (uint32_t)sum, 16);
  const uint32_t hi = __shfl_xor_sync(0xffffffffu, (uint32_t)(sum >> 32), 16);
  sum += (long long)((uint64_t)lo | ((uint64_t)hi << 32));
  const int idx = (int)(sum >> 16);
  return squash[max(-2047, min(2048, idx)) + 2047];
}

// A lane of a warp that predicts the nodes of a speculation tree.  Each half
// warp holds the 15 nodes (its last lane doubles the last one), the lower half
// their even orders, the upper half the odd ones, so that a round takes three
// gather instructions of 30 lines.  kKept: the slot tables are read only.
template <bool kLow, bool kKept = false>
struct DecLane {
  int half, depth;
  uint32_t pbits;
  bool recorder;
  const int16_t *spf;
  const uint8_t *low;
  const uint8_t *tables[3];

  __device__ __forceinline__ DecLane(const DecSmem &s, const uint8_t *slot, int lane) {
    half = lane >> 4;
    const int node = (lane & 15) < kDecNodes ? lane & 15 : kDecNodes - 1;
    depth = 31 - __clz(node + 1);
    pbits = (uint32_t)(node + 1 - (1 << depth));
    recorder = (lane & 15) < kDecNodes;
    spf = s.spf + 4 * half * kDecSpfRow;
    low = (kLow ? s.t01 : slot) + (half ? kOrder1Off : 0);
CUCM_UNROLL
    for (int q = 0; q < 3; q++) tables[q] = slot + table_offset(2 * q + 2 + half);
  }

  // Keys and frozen slot states of this lane's node and orders, r bits `cur`
  // into the byte after `hist`.
  __device__ __forceinline__ void gather(uint32_t cur, int r, const uint32_t hist[7], uint32_t kk[4],
                                         uint32_t st[4]) const {
    const uint32_t h0 = (1u << (r + depth)) | (cur << depth) | pbits;
    BitKeys k;
    bit_keys(h0, hist, k);
CUCM_UNROLL
    for (int q = 0; q < 4; q++) kk[q] = half ? k.k[2 * q + 1] : k.k[2 * q];
    if (kLow) st[0] = low[kk[0]];
CUCM_UNROLL
    for (int q = 0; q < 3; q++) st[q + 1] = state(tables[q] + kk[q + 1]);
    if (!kLow) st[0] = state(low + kk[0]);
  }
  static __device__ __forceinline__ uint32_t state(const uint8_t *p) {
    return kKept ? ld_kept_state(p) : ld_slot_state(p);
  }

  // Stretch, mixer context, mixer output (cucm_decompress_v2.cu:774-809).
  __device__ __forceinline__ uint32_t predict(const DecSmem &s, const uint16_t *squash, const uint32_t st[4],
                                              uint32_t c1, int smp[4], int &cxt) const {
    int olen = 0;
CUCM_UNROLL
    for (int q = 0; q < 4; q++) smp[q] = spf[q * kDecSpfRow + st[q]];
CUCM_UNROLL
    for (int q = 0; q < 4; q++) olen += (smp[q] != 1);
    olen += __shfl_xor_sync(0xffffffffu, olen, 16);
    cxt = olen + (int)(c1 >> 5) * 10;
    return dec_mix(s.w, cxt, smp, half, squash);
  }
};

// What a lane records of its node for the updating warp, if the node is on the
// path of the nibble decoded.
struct DecRecord {
  bool mine;
  uint4 key;
  uint32_t state;
  uint2 smp;
  uint32_t pc;  // pr | cxt << 16 | y << 24
};

template <bool kLow>
__device__ __forceinline__ DecRecord dec_record(const DecLane<kLow> &ln, const uint32_t kk[4], const uint32_t st[4],
                                                const int smp[4], uint32_t pr, int cxt, uint32_t nib) {
  DecRecord r;
  r.mine = ln.recorder && ln.pbits == (nib >> (4 - ln.depth));
  r.key = make_uint4(kk[0], kk[1], kk[2], kk[3]);
  r.state = st[0] | (st[1] << 8) | (st[2] << 16) | (st[3] << 24);
  r.smp = make_uint2((uint32_t)(smp[0] & 0xffff) | ((uint32_t)smp[1] << 16),
                     (uint32_t)(smp[2] & 0xffff) | ((uint32_t)smp[3] << 16));
  r.pc = pr | ((uint32_t)cxt << 16) | (((nib >> (3 - ln.depth)) & 1u) << 24);
  return r;
}

template <bool kLow>
__device__ __forceinline__ void dec_write_record(const DecSmem &s, const DecLane<kLow> &ln, const DecRecord &r,
                                                 int rd) {
  if (r.mine) {
    const int e = (rd * 4 + ln.depth) * kOrders + 4 * ln.half;
    *reinterpret_cast<uint4 *>(s.rk + e) = r.key;
    *reinterpret_cast<uint32_t *>(s.rs + e) = r.state;
    *reinterpret_cast<uint2 *>(s.rsmp + e) = r.smp;
    if (ln.half == 0) s.rpc[rd * 4 + ln.depth] = r.pc;
  }
}

// A chunk's model at its start, by kThreads threads.
template <bool kLow, int kThreads>
__device__ __forceinline__ void dec_start(const DecSmem &s, const DecLayout &L, const Tables *tab,
                                          const ModelInit *init, const uint8_t *slot, int t) {
  for (int i = t; i < 256 * kOrders; i += kThreads) {
    const int col = i >> 8, st = i & 255;
    const uint32_t v = init->statep[dec_order(col)][st];
    s.spf[col * kDecSpfRow + st] = tab->stretch[v >> 20];
    s.spl[col * kDecSplRow + st] = v;
  }
  for (int i = t; i < kMixCtx * kOrders; i += kThreads) {
    s.w[i] = init->w[(i & ~7) + dec_order(i & 7)];
    s.dw[i] = 0;
  }
  for (int i = t; i < kOrders * L.NT; i += kThreads) s.ovt[i] = (uint8_t)kDecNone;
  if (kLow) {
    // the chunk's order 0/1 tables move to shared memory for its lifetime
    const uint4 *src = reinterpret_cast<const uint4 *>(slot);
    uint4 *dst = reinterpret_cast<uint4 *>(s.t01);
    for (int i = t; i < (int)(kHashedOff / 16); i += kThreads) dst[i] = src[i];
  }
}

// Coder state of a chunk's first bytes (cucm_decompress_v2.cu:967-972).
__device__ __forceinline__ void dec_open(DecCoder &c, uint8_t *win, const uint8_t *pay, uint64_t plen, int lane) {
  c.wbase = dec_refill(win, pay, plen, 0, lane);
  c.x1 = 0;
  c.x2 = 0xffffffffu;
  c.x = dec_next4(win, (uint32_t)(0 - c.wbase));
  c.ioff = 4;
}

// The payload's next four bytes; the window moves on where it holds less than
// 16 bytes (a nibble's most, bit by bit).
__device__ __forceinline__ uint32_t dec_ahead(DecCoder &c, uint8_t *win, const uint8_t *pay, uint64_t plen, int lane) {
  if ((long long)c.ioff + 16 > c.wbase + kDecWin) c.wbase = dec_refill(win, pay, plen, c.ioff, lane);
  return dec_next4(win, (uint32_t)((long long)c.ioff - c.wbase));
}

// The bounded waits of a chunk's warps for one another.
template <class There, class Then>
__device__ __forceinline__ bool dec_wait(There there, uint32_t limit, Then then) {
  auto fenced = [&] {
    __threadfence_block();
    then();
  };
  return warp_wait(there, [](bool x) { return __all_sync(0xffffffffu, x) != 0; }, limit, fenced);
}
template <class There>
__device__ __forceinline__ bool dec_wait(There there, uint32_t limit) {
  return dec_wait(there, limit, [] {});
}

// The byte after `hist` joins it.
__device__ __forceinline__ void dec_push(uint32_t hist[7], uint32_t byte) {
CUCM_UNROLL
  for (int i = 6; i > 0; i--) hist[i] = hist[i - 1];
  hist[0] = byte;
}

// The pair's barrier: named barrier 1 + pair index, 64 threads.
__device__ __forceinline__ void pair_sync(int pair) {
  asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory");
}

// One chunk.  role 0 decodes, role 1 updates the model; lane = threadIdx & 31.
template <bool kLow>
__device__ void decompress_pair_one(const ChunkTask &t, uint8_t *slot, const DecSmem &s, const Tables *tab,
                                    const DecLayout &L, const ModelInit *init, int role, int pair,
                                    uint32_t *status, uint32_t spin_limit) {
  const int lane = threadIdx.x & 31;
  const int t64 = lane + 32 * role;
  const int U = L.U;
  const uint64_t len = t.out_cap < t.cs ? t.out_cap : t.cs;  // bytes to decode
  const uint64_t nbits = 8ull * len;
  const uint8_t *pay = t.in;
  const uint64_t plen = t.in_len;

  dec_start<kLow, 64>(s, L, tab, init, slot, t64);
  if (t64 == 0) s.prog[0] = 0;
  pair_sync(pair);

  if (role == 1) {
    // the updating warp: rounds in order, as the decoding warp publishes them
    uint32_t done = 0;
    bool ok = true;
    for (uint64_t base = 0; base < nbits; base += (uint64_t)U) {
      const int nunit = (int)(nbits - base < (uint64_t)U ? nbits - base : (uint64_t)U);
      for (int rd = 0; rd < (nunit >> 2); rd++) {
        // a plain poll: a sleep here wakes late and the updating warp
        // falls rounds behind by the unit's end
        ok = ok && dec_wait([&] { return s.prog[0] > done; }, spin_limit);
        if (!ok) break;
        dec_update_round(s, tab, L, lane, rd);
        done++;
      }
      if (!ok && lane == 0) atomicOr(status, (uint32_t)kDevTimeout);
      pair_sync(pair);
      dec_unit_end<64>(s, L, tab, slot, t.out + (base >> 3), nunit, t64);
      pair_sync(pair);
    }
    return;
  }

  DecCoder c;
  dec_open(c, s.win, pay, plen, lane);
  const DecLane<kLow> ln(s, slot, lane);
  uint32_t hist[7] = {0, 0, 0, 0, 0, 0, 0};  // completed bytes, most recent first
  uint32_t cur = 0;   // bits of the current byte
  int r = 0;          // 0 or 4
  uint32_t published = 0;

  // After a round is decoded the next round's gathers go out at once (within a
  // unit: the unit end writes the slot tables); the coder state, the payload
  // window and the decoded round's record follow while they are in flight.
  uint32_t kk[4], st[4];
  for (uint64_t base = 0; base < nbits; base += (uint64_t)U) {
    const int nunit = (int)(nbits - base < (uint64_t)U ? nbits - base : (uint64_t)U);
    const int nr = nunit >> 2;
    int obyte = 0;
    ln.gather(cur, r, hist, kk, st);
    uint32_t next = dec_ahead(c, s.win, pay, plen, lane);
    for (int rd = 0; rd < nr; rd++) {
      int smp[4], cxt;
      const uint32_t pr = ln.predict(s, tab->squash, st, hist[0], smp, cxt);
      DecPath path;
      const uint32_t nib = dec_nibble(c, path, pr << 20, next, s.win, lane);
      const DecRecord rec = dec_record(ln, kk, st, smp, pr, cxt, nib);
      cur = (cur << 4) | nib;
      r += 4;
      bool byte_done = false;
      if (r == 8) {
        byte_done = true;
        dec_push(hist, cur);
        cur = 0;
        r = 0;
      }
      if (rd + 1 < nr) ln.gather(cur, r, hist, kk, st);
      dec_settle(c, path, s.win);
      next = dec_ahead(c, s.win, pay, plen, lane);
      dec_write_record(s, ln, rec, rd);
      if (byte_done) {
        if (lane == 0) s.outb[obyte] = (uint8_t)hist[0];
        obyte++;
      }
      __syncwarp();
      published++;
      if (lane == 0) {
        __threadfence_block();
        s.prog[0] = published;
      }
    }
    pair_sync(pair);
    dec_unit_end<64>(s, L, tab, slot, t.out + (base >> 3), nunit, t64);
    pair_sync(pair);
  }
}

// Grid: chunk slots in pairs of warps; warp 2c decodes chunk slot c of the
// CTA, warp 2c + 1 updates its model.
template <bool kLow>
__global__ void __launch_bounds__(kDecMaxPairs * 64)
    decompress_pair_kernel(const ChunkTask *tasks, uint32_t ntasks, uint8_t *slots, uint32_t nslots,
                           const uint8_t *init_tables, const ModelInit *init, uint32_t *queue, uint32_t *status,
                           int unit, uint32_t spin_limit) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int pairs = blockDim.x >> 6;
  const DecLayout L = make_dec_layout(unit, pairs, kLow);
  Tables *tab = reinterpret_cast<Tables *>(smem_raw + L.off_tab);
  copy_tables(&g_tables, tab);
  __syncthreads();
  for (int i = threadIdx.x; i < 4096; i += blockDim.x) tab->squash[i] += tab->squash[i] < 2048;  // see dec_mix
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pair = warp >> 1, role = warp & 1;
  const uint32_t gs = blockIdx.x * (uint32_t)pairs + (uint32_t)pair;
  if (gs >= nslots) return;  // both warps of the pair leave together
  const DecSmem s = carve_dec(smem_raw, L, pair);
  uint8_t *slot = slots + (size_t)gs * kSlotTableBytes;
  bool fresh = true;
  for (;;) {
    if (role == 0 && lane == 0) s.prog[1] = atomicAdd(queue, 1u);
    pair_sync(pair);
    const uint32_t ti = s.prog[1];
    pair_sync(pair);
    if (ti >= ntasks) break;
    const ChunkTask t = tasks[ti];
    if (t.unit != (uint32_t)unit || t.cs == 0) {
      if (role == 0 && lane == 0) atomicOr(status, (uint32_t)kDevBadTask);
      continue;
    }
    if (!fresh) {
      uint4 *d = reinterpret_cast<uint4 *>(slot);
      const size_t nv = kSlotTableBytes / 16;
      const int t64 = lane + 32 * role;
      if (init_tables) {
        const uint4 *src = reinterpret_cast<const uint4 *>(init_tables);
        for (size_t i = t64; i < nv; i += 64) d[i] = src[i];
      } else {
        for (size_t i = t64; i < nv; i += 64) d[i] = make_uint4(0, 0, 0, 0);
      }
      pair_sync(pair);
    }
    fresh = false;
    decompress_pair_one<kLow>(t, slot, s, tab, L, init, role, pair, status, spin_limit);
  }
}
