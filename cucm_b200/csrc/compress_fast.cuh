// compress_fast.cuh -- pipelined chunk compressor for units of 32..256 bits.
//
// Included by engine_kernels.cu (shares its tables and coder helpers).
//
// The reference runs five launches per unit and a host round trip between
// them (cucm_compress_v2.cu:1067-1090).  Here one CTA of 7 warps codes a
// chunk, each warp owning one stage, all stages of consecutive units
// overlapped ("tick" t).  The numbers below are roles (kRolesAlone and
// kRolesPaired give them to physical warps):
//
//   front warps (3..6, 128 threads)
//     * keys of unit t+1 for all 8 orders (one FNV pass per bit,
//       cucm_compress_v2.cu:723-747), the unit's bits and previous bytes;
//     * slot links of unit t+1: per order, bits that touch the same slot share
//       one number, so every later touch knows it must read the state its
//       predecessor left, and know whether the slot was touched one unit
//       earlier;
//     * gathers of unit t+1's slot states from the tables in HBM;
//     * stretch, mixer context, mixer output and training of unit t-1
//       (cudamixUnit / cudaupdateMixer, cucm_compress_v2.cu:755-819) against
//       the probabilities as they stand when the previous chain has ended
//       (read from the StateMap records before the chain of unit t-1
//       starts on them).
//   walker warp (2): the bit-history side of the StateMap update for unit
//     t, in bit order, a byte (64 updates) per step: the state each update
//     sees (live), the state each prediction saw (frozen = unit-start value),
//     the next state, written through to the slot table.  It only depends on
//     the bits, never on the probabilities, so it runs a unit ahead of the
//     chain, and groups the unit's updates by state for it.
//   chain warp (0, lane = order): the StateMap probability updates of unit
//     t-1, state by state, each state's in bit order
//     (cucm_compress_v2.cu:592-601).
//   coder warp (1): the binary arithmetic coder for unit t-2.
//
// After the last data unit the coder keeps coding the stale unit buffer up
// to the chunk end, as cudaencodeUnit does (cucm_compress_v2.cu:850-852).

constexpr int kFastWarps = 7;
constexpr int kFastThreads = kFastWarps * 32;
constexpr int kFastMaxUnit = 256;
constexpr int kWChain = 0, kWCoder = 1, kWWalk = 2, kWFront = 3;
constexpr int kFrontThreads = 128;
constexpr int kSnapThreads = 32 + kFrontThreads;  // chain + front warps (barrier 1)
constexpr int kWinBytes = kFastMaxUnit / 8 + 8;    // input window of a unit (+7 history bytes)

// Role of each of a CTA's warps, 4 bits a warp.  Warp i issues from the SM's
// scheduler i % 4.  Alone on an SM, each serial role shares a scheduler with
// front warps only; where two CTAs share an SM, the chain keeps one for itself
// and coder and walker share one.  Each the other way round: 1 MiB at 64 KiB
// chunks (16 CTAs) 22.1 -> 23.7 ms, 128 MiB at 512 KiB chunks (two CTAs an SM)
// 357 -> 364 ms.
constexpr uint32_t kRolesAlone = 0x6540213u, kRolesPaired = 0x6250413u;

constexpr int kFastStageMin = 2048;

// A compress CTA keeps the whole of the tables in shared memory (reading
// stretch and squash through the read-only cache instead measured 10 %
// slower: the lookups are on the front warps' critical path).
typedef Tables FastTables;

// Row padding of the walker's [order][...] arrays: 16 bytes, so that the 8
// orders' rows start in different banks.
constexpr int kStatePad = 16, kSortPad = 8;
constexpr int kRecRow = 257;   // 256 states: the rows start in different banks, bits of one order spread over all

constexpr uint32_t kUntouched = 0xffu;  // no state: the largest is 252
constexpr int kClaimLog = 9, kClaim = 1 << kClaimLog;  // places of a claim table

struct FastLayout {
  int U, NSLOT, stage;
  int ks, ls;   // row lengths of key and of lnk / bkt
  size_t off_tab, off_rec, off_w, off_claim, off_late, off_ns, off_key, off_lnk, off_bkt, off_fsw, off_st, off_srt,
      off_fr, off_yw, off_c1, off_prm, off_win, off_stage, total;
};

__host__ __device__ constexpr FastLayout make_fast_layout(int U) {
  FastLayout L{};
  L.U = U;
  L.NSLOT = U <= 128 ? 128 : 256;  // slots per order and unit
  L.ks = U + 4;  // rows of 8 orders that start in different banks
  L.ls = U + 8;
  L.stage = next_pow2(4 * U + 1024);  // a unit codes at most 4U bytes; flushes go out in 512-byte blocks
  if (L.stage < kFastStageMin) L.stage = kFastStageMin;
  const size_t NS = (size_t)L.NSLOT;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    size_t at = o;
    o = (o + bytes + 15) & ~(size_t)15;
    return at;
  };
  L.off_tab = take(sizeof(FastTables));
  L.off_rec = take(sizeof(uint32_t) * kOrders * kRecRow);
  L.off_w = take(sizeof(int32_t) * kMixCtx * kOrders);
  L.off_claim = take((size_t)2 * kOrders * 2 * kClaim);   // claim tables [unit parity][order][round]
  L.off_late = take((size_t)2 * kOrders * (NS + 4));       // slots claimed after the rounds [unit parity][order]
  L.off_ns = take((size_t)2 * kOrders * NS);               // state written in the unit, or kUntouched
  L.off_key = take(sizeof(uint32_t) * 2 * kOrders * L.ks); // [unit parity][order][bit]
  L.off_lnk = take(sizeof(uint16_t) * 2 * kOrders * L.ls); // slot + 1 in the previous unit, or 0 [unit parity][order][bit]
  L.off_bkt = take((size_t)2 * kOrders * L.ls);            // slot in this unit
  L.off_fsw = take((size_t)2 * kOrders * U);               // gathered slot states
  L.off_st = take((size_t)kOrders * (U + kStatePad));      // live state [order][bit]
  L.off_srt = take(sizeof(uint16_t) * 2 * kOrders * (U + kSortPad));  // updates grouped by state [unit parity][order]
  L.off_fr = take((size_t)2 * U * kOrders);                // frozen state
  L.off_yw = take(sizeof(uint32_t) * 4 * (U / 32));        // bits, by unit mod 4
  L.off_c1 = take((size_t)4 * (U / 8));                    // previous byte per byte, by unit mod 4
  L.off_prm = take(sizeof(uint2) * 2 * U);                 // coder input, by unit parity
  L.off_win = take((size_t)kWinBytes);
  L.off_stage = take((size_t)L.stage);
  L.total = o;
  return L;
}

// Shared memory that a CTA takes of its SM's 228 KiB, 1 KiB of it reserved by
// the hardware.  Two CTAs share an SM at every unit: 2 * 110,032 of 233,472
// bytes at 256 bits.  What they leave is L1, in steps: at 128 bits two take 160
// KB, and 4.7 KB more a CTA moved the split from 164 to 196 KB: 128 MiB in 256
// chunks 348 -> 362 ms (it may be that gathers in flight hold L1 lines).
constexpr size_t kFastSmBytes = 228 * 1024;
__host__ __device__ constexpr size_t fast_sm_bytes(int U) { return make_fast_layout(U).total + 1024 + 64; }
static_assert(2 * fast_sm_bytes(kFastMaxUnit) <= kFastSmBytes, "two CTAs an SM");

struct FastSmem {
  FastTables *tab;
  uint32_t *rec;     // [8][kRecRow]  statep
  int32_t *w;        // [80*8]
  uint8_t *claim;    // [2][8][2][kClaim]
  uint8_t *late;     // [2][8][NSLOT + 4]: count, slots
  uint8_t *ns;       // [2][8][NSLOT]
  uint32_t *key;     // [2][8][ks]
  uint16_t *lnk;     // [2][8][ls]
  uint8_t *bkt;      // [2][8][ls]
  uint8_t *fsw;      // [2][U][8]
  uint8_t *st;       // [8][U + kStatePad]
  uint16_t *srt;     // [2][8][U + kSortPad]
  uint8_t *fr;       // [2][U][8]
  uint32_t *yw;      // [4][U/32]
  uint8_t *c1;       // [4][U/8]
  uint2 *prm;        // [2][U]
  uint8_t *win;      // [kWinBytes]
  uint8_t *stage;
};

__device__ inline FastSmem carve_fast(uint8_t *b, const FastLayout &L) {
  FastSmem s;
  s.tab = reinterpret_cast<FastTables *>(b + L.off_tab);
  s.rec = reinterpret_cast<uint32_t *>(b + L.off_rec);
  s.w = reinterpret_cast<int32_t *>(b + L.off_w);
  s.claim = b + L.off_claim;
  s.late = b + L.off_late;
  s.ns = b + L.off_ns;
  s.key = reinterpret_cast<uint32_t *>(b + L.off_key);
  s.lnk = reinterpret_cast<uint16_t *>(b + L.off_lnk);
  s.bkt = b + L.off_bkt;
  s.fsw = b + L.off_fsw;
  s.st = b + L.off_st;
  s.srt = reinterpret_cast<uint16_t *>(b + L.off_srt);
  s.fr = b + L.off_fr;
  s.yw = reinterpret_cast<uint32_t *>(b + L.off_yw);
  s.c1 = b + L.off_c1;
  s.prm = reinterpret_cast<uint2 *>(b + L.off_prm);
  s.win = b + L.off_win;
  s.stage = b + L.off_stage;
  return s;
}

__device__ __forceinline__ void named_barrier(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Barrier ids: 0 = whole CTA, 1 = chain + front (probabilities read before
// the chain updates them), 2 = front only.
__device__ __forceinline__ void front_sync() { named_barrier(2, kFrontThreads); }

__device__ __forceinline__ int fast_nvalid(uint64_t data_bits, int U, int v) {
  const uint64_t b = (uint64_t)v * U;
  return (v < 0 || b >= data_bits) ? 0 : (int)(data_bits - b < (uint64_t)U ? data_bits - b : (uint64_t)U);
}

// Input byte k of unit v's window: chunk byte v*U/8 - 7 + k, 0 outside
// [0, len).  Thread t < U/8 + 7 loads one byte.
__device__ __forceinline__ uint32_t window_load(const uint8_t *in, uint64_t len, int U, int v, int t) {
  const int64_t i = (int64_t)v * (U / 8) - 7 + t;
  return (t < U / 8 + 7 && i >= 0 && (uint64_t)i < len) ? (uint32_t)__ldg(in + i) : 0u;
}

__device__ __forceinline__ uint32_t *keys_of(const FastSmem &s, const FastLayout &L, int v) {
  return s.key + (v & 1) * kOrders * L.ks;
}

// Front: keys, bits and previous bytes of unit v from the staged window.
__device__ __forceinline__ void front_keys(const FastSmem &s, const FastLayout &L, int t, int v, int nvalid) {
  const int U = L.U;
  uint32_t *key = keys_of(s, L, v);
  uint32_t *yw = s.yw + (v & 3) * (U / 32);
  uint8_t *c1 = s.c1 + (v & 3) * (U / 8);
  for (int j0 = 0; j0 < U; j0 += kFrontThreads) {
    const int j = j0 + t;
    uint32_t y = 0;
    if (j < nvalid) {
      const int q = j >> 3, r = j & 7;
      const uint32_t cur = s.win[q + 7];
      const uint32_t h0 = (1u << r) | (cur >> (8 - r));
      const uint32_t p1 = s.win[q + 6];
      uint32_t k8[kOrders];
      uint32_t acc = (kFnvBasis ^ h0) * kFnvPrime;
      k8[0] = h0;
      k8[1] = (p1 << 8) | h0;
      acc = (acc ^ p1) * kFnvPrime;
      CUCM_UNROLL
      for (int o = 2; o < kOrders; o++) {
        acc = (acc ^ (uint32_t)s.win[q + 7 - o]) * kFnvPrime;
        k8[o] = acc & (kSlots - 1);
      }
      CUCM_UNROLL
      for (int o = 0; o < kOrders; o++) key[o * L.ks + j] = k8[o];
      y = (cur >> (7 - r)) & 1u;
      if (r == 0) c1[q] = (uint8_t)p1;
    }
    // 32 consecutive bits per warp instruction: pack them.
    const uint32_t word = __ballot_sync(0xffffffffu, y != 0);
    if ((t & 31) == 0 && j < U) yw[j >> 5] = word;
  }
}

// Slots of a unit: per order, bits that touch the same table slot share one
// number, the position of one of them, and a bit whose slot the previous unit
// touched too knows that unit's number for it.
//
// Every bit writes its position to a small claim table at a hash of its key;
// whoever's position is there afterwards is the slot's number for all bits
// with that key (they all hash to the same place), and bits that find another
// key's claim go on to a second table.  Nothing is cleared: a place is only
// read by bits that have just written it, and the previous unit's tables only
// lead to a position whose key is compared.  With 4 places per bit (units of
// 128 bits), 10-11 % of the keys of text, walk and random bytes need the second
// table and one in ~700 gets neither: those are numbered one after the other and
// listed.  At 2 places per bit (256 bits) it is 20 % and one in ~100, 18 of a
// unit's 2,048; tables twice as long take 16 KB more, and two CTAs would not fit an SM.  The
// two orders' ~12 shared-memory steps take 3,250 cycles a unit of 128 bits for a
// CTA alone; sorting each order's keys across the warp and searching the rows
// took 8,100 of the front warps' 12,000.
//
// Front warp w owns orders 2w and 2w + 1, so no other warp writes their
// tables.  E bits per lane: 32 * E >= U.
__device__ __forceinline__ uint32_t claim_at(uint32_t key, int round, int logn) {
  return (key * (round ? 0x85EBCA6Bu : 0x9E3779B1u)) >> (32 - logn);
}

template <int E>
__device__ __forceinline__ void front_links(const FastSmem &s, const FastLayout &L, int t, int v, int nvalid) {
  const int lane = t & 31, w = t >> 5;
  const uint32_t *key = keys_of(s, L, v);
  const uint32_t *pkey = keys_of(s, L, v + 1);
  uint16_t *lnk = s.lnk + (v & 1) * kOrders * L.ls;
  uint8_t *bkt = s.bkt + (v & 1) * kOrders * L.ls;
  uint32_t k[2][E];
  int num[2][E], prev[2][E];  // slot here; slot + 1 in the previous unit
  uint8_t *claim[2], *pclaim[2];
  CUCM_UNROLL
  for (int h = 0; h < 2; h++) {
    const int o = 2 * w + h;
    claim[h] = s.claim + ((v & 1) * kOrders + o) * 2 * kClaim;
    pclaim[h] = s.claim + (((v + 1) & 1) * kOrders + o) * 2 * kClaim;
    CUCM_UNROLL
    for (int i = 0; i < E; i++) {
      const int j = lane + 32 * i;
      k[h][i] = j < nvalid ? key[o * L.ks + j] : 0u;
    }
  }
  // (in all of this the loads of a step stand before its stores: the compiler
  // keeps their order, and a load behind a store waits its turn)
  CUCM_UNROLL
  for (int h = 0; h < 2; h++) {
    CUCM_UNROLL
    for (int i = 0; i < E; i++)
      if (lane + 32 * i < nvalid) claim[h][claim_at(k[h][i], 0, kClaimLog)] = (uint8_t)(lane + 32 * i);
  }
  __syncwarp();
  uint32_t open = 0;   // bits of this lane that still need a number: bit E * h + i
  uint32_t loose = 0;  // ... whose key the previous unit's first table does not have
  CUCM_UNROLL
  for (int h = 0; h < 2; h++) {
    const int o = 2 * w + h;
    CUCM_UNROLL
    for (int i = 0; i < E; i++) {
      const int j = lane + 32 * i;
      const uint32_t at = claim_at(k[h][i], 0, kClaimLog);
      num[h][i] = claim[h][at];
      const int p = pclaim[h][at];
      const bool here = key[o * L.ks + num[h][i]] == k[h][i];
      const bool there = v > 0 && pkey[o * L.ks + p] == k[h][i];
      prev[h][i] = there ? p + 1 : 0;
      if (j < nvalid && !here) open |= 1u << (E * h + i);
      if (j < nvalid && !there) loose |= 1u << (E * h + i);
    }
  }
  // second tables: every bit looks, the open ones claim
  CUCM_UNROLL
  for (int h = 0; h < 2; h++) {
    CUCM_UNROLL
    for (int i = 0; i < E; i++)
      if (open >> (E * h + i) & 1u) claim[h][kClaim + claim_at(k[h][i], 1, kClaimLog)] = (uint8_t)(lane + 32 * i);
  }
  __syncwarp();
  CUCM_UNROLL
  for (int h = 0; h < 2; h++) {
    const int o = 2 * w + h;
    CUCM_UNROLL
    for (int i = 0; i < E; i++) {
      const uint32_t bit = 1u << (E * h + i);
      const uint32_t at = kClaim + claim_at(k[h][i], 1, kClaimLog);
      const int n = claim[h][at], p = pclaim[h][at];
      const bool here = key[o * L.ks + n] == k[h][i];
      const bool there = pkey[o * L.ks + p] == k[h][i];
      const bool take = (open & bit) && here, tie = v > 0 && (loose & bit) && there;
      num[h][i] = take ? n : num[h][i];
      prev[h][i] = tie ? p + 1 : prev[h][i];
      open &= take ? ~bit : ~0u;
      loose &= tie ? ~bit : ~0u;
    }
  }
  // bits without a claim: the first one's position for all with its key
  uint8_t *late = s.late + ((v & 1) * kOrders + 2 * w) * (L.NSLOT + 4);
  const uint8_t *plate = s.late + (((v + 1) & 1) * kOrders + 2 * w) * (L.NSLOT + 4);
  int nlate[2] = {0, 0};
  if (__any_sync(0xffffffffu, open != 0)) {
    CUCM_UNROLL
    for (int h = 0; h < 2; h++) {
      CUCM_UNROLL
      for (int i = 0; i < E; i++) {
        uint32_t m;
        while ((m = __ballot_sync(0xffffffffu, open >> (E * h + i) & 1u)) != 0) {
          const int src = __ffs(m) - 1;
          const uint32_t kk = __shfl_sync(0xffffffffu, k[h][i], src);
          const int n = src + 32 * i;
          CUCM_UNROLL
          for (int q = 0; q < E; q++)
            if ((open >> (E * h + q) & 1u) && k[h][q] == kk) {
              num[h][q] = n;
              open &= ~(1u << (E * h + q));
            }
          if (lane == 0) late[h * (L.NSLOT + 4) + 4 + nlate[h]] = (uint8_t)n;
          nlate[h]++;
        }
      }
    }
  }
  CUCM_UNROLL
  for (int h = 0; h < 2; h++) {
    const int o = 2 * w + h;
    const int np = v > 0 ? plate[h * (L.NSLOT + 4)] : 0;
    for (int q = 0; q < np; q++) {
      const int n = plate[h * (L.NSLOT + 4) + 4 + q];
      const uint32_t kk = pkey[o * L.ks + n];
      CUCM_UNROLL
      for (int i = 0; i < E; i++)
        if ((loose >> (E * h + i) & 1u) && k[h][i] == kk) prev[h][i] = n + 1;
    }
    if (lane == 0) late[h * (L.NSLOT + 4)] = (uint8_t)nlate[h];
    CUCM_UNROLL
    for (int i = 0; i < E; i++) {
      const int j = lane + 32 * i;
      if (j < nvalid) {
        bkt[o * L.ls + j] = (uint8_t)num[h][i];
        lnk[o * L.ls + j] = (uint16_t)prev[h][i];
      }
    }
  }
}

// Long units: E = the unit's 32-bit words, so that no lane works on padding (160
// bits in 256 chunks, 7.6 ms with E = 8, 6.4 so; 192 bits 8.3 and 7.9).  Up to
// 128 bits E = 4: four more copies of the code cost units of 128 bits 1 %.
template <int GR>
__device__ __forceinline__ void front_links_unit(const FastSmem &s, const FastLayout &L, int t, int v, int nvalid) {
  if (GR == 8) {
    front_links<4>(s, L, t, v, nvalid);
    return;
  }
  switch (L.U >> 5) {
    case 5: front_links<5>(s, L, t, v, nvalid); break;
    case 6: front_links<6>(s, L, t, v, nvalid); break;
    case 7: front_links<7>(s, L, t, v, nvalid); break;
    default: front_links<8>(s, L, t, v, nvalid); break;
  }
}

// Walker: bit-history updates of unit v in bit order, a byte per step.  The 8
// keys of a byte and an order are never alike: the bits share the previous
// bytes and differ in the partial byte, and both steps of the hash, the XOR
// with a byte and the product with an odd number, are one-to-one on its low 25
// bits.  So the 64 updates of a byte (lane: order lane & 7, bits lane >> 3 and
// (lane >> 3) + 4) are independent and run together.  Per update: the state it
// sees (live: an earlier touch in this unit, else the frozen unit-start state
// -- from the previous unit's table when linked), the next state, written
// through to the slot table.  It only depends on the bits, never on the
// probabilities, so it runs a unit ahead of the chain.  All that a step reads
// but its slots' live states is read a step ahead, so a step waits for two
// shared-memory loads one after the other, the live state and its successor.
struct WalkByte {
  uint32_t b[2], k[2], f[2], y[2];  // slot, key, frozen state, bit
};

__device__ __forceinline__ void walk_unit(const FastSmem &s, const FastLayout &L, uint8_t *slot, int lane, int v,
                                          int n) {
  const int U = L.U, NS = L.NSLOT;
  const int o = lane & 7, r0 = lane >> 3;
  const uint32_t *key = keys_of(s, L, v) + o * L.ks;
  const uint16_t *lnk = s.lnk + ((v & 1) * kOrders + o) * L.ls;
  const uint8_t *bkt = s.bkt + ((v & 1) * kOrders + o) * L.ls;
  const uint8_t *fsb = s.fsw + (v & 1) * U * kOrders + o;
  const uint32_t *yw = s.yw + (v & 3) * (U / 32);
  uint8_t *st = s.st + o * (U + kStatePad);
  uint8_t *fr = s.fr + (v & 1) * U * kOrders + o;
  uint8_t *ns_cur = s.ns + ((v & 1) * kOrders + o) * NS;
  const uint8_t *ns_prev = s.ns + (((v + 1) & 1) * kOrders + o) * NS;
  uint8_t *tab = slot + table_offset(o);
  const FastTables *tb = s.tab;
  auto ahead = [&](int j, WalkByte &w) {
    const uint32_t yword = yw[j >> 5];
CUCM_UNROLL
    for (int h = 0; h < 2; h++) {
      const int jj = j + r0 + 4 * h;
      w.b[h] = bkt[jj];
      w.k[h] = key[jj];
      const uint32_t c = lnk[jj];
      const uint32_t g = fsb[jj * kOrders];
      w.f[h] = c ? (uint32_t)ns_prev[c - 1] : g;
      w.y[h] = (yword >> (jj & 31)) & 1u;
    }
  };
  WalkByte w;
  ahead(0, w);
  for (int j = 0; j < n; j += 8) {
    const WalkByte c = w;
    const uint32_t n0 = ns_cur[c.b[0]], n1 = ns_cur[c.b[1]];
    if (j + 8 < n) ahead(j + 8, w);
    const uint32_t l0 = n0 != kUntouched ? n0 : c.f[0];
    const uint32_t l1 = n1 != kUntouched ? n1 : c.f[1];
    const uint32_t s0 = tb->nex[l0][c.y[0]], s1 = tb->nex[l1][c.y[1]];
    ns_cur[c.b[0]] = (uint8_t)s0;
    ns_cur[c.b[1]] = (uint8_t)s1;
    __syncwarp();
    const int j0 = j + r0, j1 = j0 + 4;
    st[j0] = (uint8_t)l0;
    st[j1] = (uint8_t)l1;
    fr[j0 * kOrders] = (uint8_t)c.f[0];
    fr[j1 * kOrders] = (uint8_t)c.f[1];
    tab[c.k[0]] = (uint8_t)s0;  // write-through; later touches overwrite it
    tab[c.k[1]] = (uint8_t)s1;
  }
  __syncwarp();
}

// Walker: groups unit v's StateMap updates by state for the chain warp.  Per
// order and 128 bits, the updates (state << 8 | bit << 1 | y) in ascending
// order: states apart, the updates of one state in bit order.  Lane = (order
// lane & 7, quarter lane >> 3) sorts its 32 bits, two 16-bit keys to a
// register, then the quarters are merged across lanes.  Updates of different
// states of an order never meet, so this is all the order the chain needs.
__device__ __forceinline__ void sort_ce(uint32_t &a, uint32_t &b) {
  const uint32_t m = __vminu2(a, b);
  b = __vmaxu2(a, b);
  a = m;
}
__device__ __forceinline__ uint32_t swap_halves(uint32_t a) { return __byte_perm(a, 0, 0x1032); }

// 32 keys of a lane, key k in the low half and key 16 + k in the high half of
// r[k]: the last steps of a bitonic merge, distances 16, 8, 4, 2, 1.
__device__ __forceinline__ void sort_merge32(uint32_t (&r)[16], bool halves) {
  if (halves) {
CUCM_UNROLL
    for (int k = 0; k < 16; k++) {
      const uint32_t w = swap_halves(r[k]);
      r[k] = __byte_perm(__vminu2(r[k], w), __vmaxu2(r[k], w), 0x5410);
    }
  }
CUCM_UNROLL
  for (int d = 8; d > 0; d >>= 1)
CUCM_UNROLL
    for (int k = 0; k < 16; k++)
      if ((k & d) == 0) sort_ce(r[k], r[k | d]);
}

// This lane's keys against those of lane ^ lanes in reverse (a first merge
// step) or position by position (a later one): the smaller or larger ones.
__device__ __forceinline__ void sort_cross(uint32_t (&r)[16], int lanes, bool reverse, bool low) {
  uint32_t w[16];
CUCM_UNROLL
  for (int k = 0; k < 16; k++) w[k] = __shfl_xor_sync(0xffffffffu, r[k], lanes);
CUCM_UNROLL
  for (int k = 0; k < 16; k++) {
    const uint32_t x = reverse ? swap_halves(w[15 - k]) : w[k];
    r[k] = low ? __vminu2(r[k], x) : __vmaxu2(r[k], x);
  }
}

__device__ __forceinline__ void walk_sort(const FastSmem &s, const FastLayout &L, int lane, int v, int n) {
  const int U = L.U;
  const int o = lane & 7, q = lane >> 3;
  const uint32_t *yw = s.yw + (v & 3) * (U / 32);
  for (int j0 = 0; j0 < n; j0 += 128) {
    const int jq = j0 + 32 * q;  // first bit of this lane
    const int have = n - jq;     // a multiple of 8
    uint32_t r[16];
    if (have > 0) {
      const uint32_t y = yw[jq >> 5];
      const uint4 *src = reinterpret_cast<const uint4 *>(s.st + o * (U + kStatePad) + jq);
      const uint4 a = src[0], b = src[1];
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
CUCM_UNROLL
      for (int k = 0; k < 16; k++) {  // bits 2k and 2k + 1
        const uint32_t st = __byte_perm(w[k >> 1], 0, k & 1 ? 0x3424 : 0x1404);
        const uint32_t bits = (uint32_t)(32 * q) * 0x20002u + (uint32_t)(4 * k) + ((uint32_t)(4 * k + 2) << 16);
        r[k] = st | bits | ((y >> (2 * k)) & 1u) | (((y >> (2 * k + 1)) & 1u) << 16);
        if (2 * k >= have) r[k] = 0xffffffffu;
      }
    } else {
CUCM_UNROLL
      for (int k = 0; k < 16; k++) r[k] = 0xffffffffu;
    }
    // the low and the high halves, 16 keys each (Batcher's merge exchange)
CUCM_UNROLL
    for (int p = 1; p < 16; p *= 2)
CUCM_UNROLL
      for (int k = p; k >= 1; k /= 2)
CUCM_UNROLL
        for (int i = 0; i < 16; i++)
          if (i + k < 16 && i >= k % p && (i - k % p) % (2 * k) < k && i / (2 * p) == (i + k) / (2 * p))
            sort_ce(r[i], r[i + k]);
    // the two halves of a lane
CUCM_UNROLL
    for (int k = 0; k < 8; k++) {
      const uint32_t w = swap_halves(r[15 - k]);
      const uint32_t m = __vminu2(r[k], w), x = __vmaxu2(r[k], w);
      r[k] = __byte_perm(m, x, 0x5410);
      r[15 - k] = __byte_perm(m, x, 0x7632);
    }
    sort_merge32(r, false);
    if (n - j0 > 32) {
      sort_cross(r, 8, true, (q & 1) == 0);
      sort_merge32(r, true);
    }
    if (n - j0 > 64) {
      sort_cross(r, 24, true, q < 2);
      sort_cross(r, 8, false, (q & 1) == 0);
      sort_merge32(r, true);
    }
    if (have > 0) {
      uint4 *dst = reinterpret_cast<uint4 *>(s.srt + ((v & 1) * kOrders + o) * (U + kSortPad) + jq);
CUCM_UNROLL
      for (int h = 0; h < 4; h++) {
        const uint32_t sel = h < 2 ? 0x5410 : 0x7632;
        const int k = 8 * (h & 1);
        dst[h] = make_uint4(__byte_perm(r[k], r[k + 1], sel), __byte_perm(r[k + 2], r[k + 3], sel),
                            __byte_perm(r[k + 4], r[k + 5], sel), __byte_perm(r[k + 6], r[k + 7], sel));
      }
    }
  }
}

// Chain (lane = order): StateMap probability updates of unit v
// (cucm_compress_v2.cu:592-601), state by state in the order walk_sort left
// them.  The updates of one state follow one another with its probability in
// a register; everything else -- the probability a state starts from, its
// count, which only ever grows by one per update, and so each update's
// adaptation rate -- is known ahead, and read a block of 8 updates early.
// Seven dependent operations a step; the ~35 instructions of a step bound it
// (80 cycles, against 110 for the bits in order with every record stored and
// the next one forwarded or loaded).  Working the operands out with all 32
// lanes first, for 8 lanes to run through, measured the same (units of 128
// bits) or 14 % slower (256).
struct ChainBlock {
  uint32_t at[8];   // record index | 0x8000 where a state begins
  uint32_t v[8];    // probability the state begins with
  uint32_t d[8];    // -rate
  uint32_t k[8];    // (y << 19) * rate
  uint32_t inc;     // bit i: the count still grows
};

__device__ __forceinline__ void chain_block(ChainBlock &b, const uint32_t *rec, const uint16_t *dt, const uint4 &e4,
                                            uint32_t &prev, uint32_t &cnt) {
  const uint32_t w[4] = {e4.x, e4.y, e4.z, e4.w};
  uint32_t e[8];
  b.inc = 0;
CUCM_UNROLL
  for (int i = 0; i < 8; i++) {
    e[i] = i & 1 ? w[i >> 1] >> 16 : w[i >> 1] & 0xffffu;
    b.at[i] = e[i] >> 8;
    b.v[i] = rec[b.at[i]];
  }
CUCM_UNROLL
  for (int i = 0; i < 8; i++) {
    const bool first = (e[i] ^ prev) >= 256u;
    prev = e[i];
    cnt = first ? b.v[i] & 1023u : min(cnt + 1, 1023u);
    if (first) b.at[i] |= 0x8000u;
    const uint32_t r = dt[cnt];
    b.d[i] = 0u - r;
    b.k[i] = (e[i] & 1u) ? r << 19 : 0u;
    if (cnt < 1023u) b.inc |= 1u << i;
  }
}

__device__ __forceinline__ void chain_run(const ChainBlock &b, uint32_t *rec, uint32_t &val) {
CUCM_UNROLL
  for (int i = 0; i < 8; i++) {
    const uint32_t x = (b.at[i] & 0x8000u) ? b.v[i] : val;
    // (err >> 3) * rate with err = (y << 22) - (x >> 10)
    const uint32_t t = ((x >> 10) + 7u) >> 3;
    val = x + (((b.k[i] + t * b.d[i]) & 0xfffffc00u) | ((b.inc >> i) & 1u));
    rec[b.at[i] & 0x7fffu] = val;
  }
}

__device__ __forceinline__ void fast_chain(const FastSmem &s, const FastLayout &L, int o, int v, int n) {
  uint32_t *rec = s.rec + o * kRecRow;
  const uint16_t *dt = s.tab->dt;
  const uint4 *src = reinterpret_cast<const uint4 *>(s.srt + ((v & 1) * kOrders + o) * (L.U + kSortPad));
  for (int j0 = 0; j0 < n; j0 += 128) {
    const int nb = (n - j0 < 128 ? n - j0 : 128) >> 3;  // blocks (n is a multiple of 8)
    uint32_t prev = 0x10000u, cnt = 0, val = 0;
    ChainBlock cur, nxt;
    chain_block(cur, rec, dt, src[0], prev, cnt);
    for (int i = 1; i < nb; i++) {
      // only states that begin in the next block use what is read here, and
      // no earlier block has touched those
      chain_block(nxt, rec, dt, src[i], prev, cnt);
      chain_run(cur, rec, val);
      cur = nxt;
    }
    chain_run(cur, rec, val);
    src += 16;
  }
}

// Front: stretched probabilities of unit v's bits (thread t: bits t and
// t + 128) as the records stand when the previous chain has ended, read
// before the chain of unit v changes them.
__device__ __forceinline__ void front_probs(const FastSmem &s, const FastLayout &L, int t, int v, int nvalid,
                                            int (&smps)[2][kOrders]) {
  const int U = L.U;
  const uint8_t *fr = s.fr + (v & 1) * U * kOrders;
  CUCM_UNROLL
  for (int h = 0; h < 2; h++) {
    const int j = t + h * kFrontThreads;
    if (j < U && j < nvalid) {
      const uint64_t f8 = *reinterpret_cast<const uint64_t *>(fr + j * kOrders);
      CUCM_UNROLL
      for (int o = 0; o < kOrders; o++) {
        const uint32_t stt = (uint32_t)(f8 >> (8 * o)) & 0xffu;
        smps[h][o] = s.tab->stretch[s.rec[o * kRecRow + stt] >> 20];
      }
    }
  }
}

// Front: predictions, mixer output and training of unit v from the
// probabilities front_probs read; thread t handles bits t and t + 128.
__device__ __forceinline__ void front_mix(const FastSmem &s, const FastLayout &L, int t, int v, int nvalid,
                                          int (&smps)[2][kOrders]) {
  const int U = L.U;
  const uint32_t *yw = s.yw + (v & 3) * (U / 32);
  const uint8_t *c1 = s.c1 + (v & 3) * (U / 8);
  uint2 *prm = s.prm + (v & 1) * U;
  const uint2 *prm_old = s.prm + ((v + 1) & 1) * U;
  int cxs[2] = {0, 0}, errs[2] = {0, 0};
  bool has[2] = {false, false};
  CUCM_UNROLL
  for (int h = 0; h < 2; h++) {
    const int j = t + h * kFrontThreads;
    if (j < U) {
      if (j < nvalid) {
        int olen = 0;
        CUCM_UNROLL
        for (int o = 0; o < kOrders; o++) olen += (smps[h][o] != 1);
        const int cx = olen + (c1[j >> 3] >> 5) * 10;
        const int pr = mix_pr(s.w, cx, smps[h], s.tab);
        const int y = (yw[j >> 5] >> (j & 31)) & 1;
        prm[j] = coder_entry((uint32_t)((pr << 1) | y));
        cxs[h] = cx;
        errs[h] = ((y << 12) - pr) * 7;
        has[h] = true;
      } else {
        prm[j] = prm_old[j];  // stale entry, re-coded as the reference does
      }
    }
  }
  front_sync();  // every weight read before any update
  // Lane l adds its order (l + i) % 8 at step i: the bits of a warp mostly
  // share a few rows, and the same order at a time would send all 32 adds to
  // those rows' one word (and 4 banks).
  CUCM_UNROLL
  for (int h = 0; h < 2; h++) {
    if (has[h]) {
      int d[kOrders];
      CUCM_UNROLL
      for (int o = 0; o < kOrders; o++) d[o] = (int)(((long long)errs[h] * smps[h][o]) >> 16);
      CUCM_UNROLL
      for (int k = 1; k < kOrders; k <<= 1) {
        int e[kOrders];
        CUCM_UNROLL
        for (int o = 0; o < kOrders; o++) e[o] = (t & k) ? d[(o + k) & 7] : d[o];
        CUCM_UNROLL
        for (int o = 0; o < kOrders; o++) d[o] = e[o];
      }
      CUCM_UNROLL
      for (int i = 0; i < kOrders; i++) atomicAdd(&s.w[cxs[h] * kOrders + ((t + i) & 7)], d[i]);
    }
  }
}

// Front: table words holding the slot states of unit v, into registers.
// Thread t takes the 8 orders of bits t and t + 128; GR is 8 for units up to
// 128 bits and 16 up to 256.
template <int GR>
__device__ __forceinline__ void front_gather(const FastSmem &s, const FastLayout &L, const uint8_t *slot, int t,
                                             int v, int nvalid, uint32_t g[GR]) {
  const uint32_t *key = keys_of(s, L, v);
  CUCM_UNROLL
  for (int i = 0; i < GR; i++) {
    const int j = t + (i >> 3) * kFrontThreads, o = i & 7;
    if (j < nvalid) {
      const uint32_t k = key[o * L.ks + j];
      g[i] = __ldcg(reinterpret_cast<const uint32_t *>(slot + table_offset(o) + (k & ~3u)));
    }
  }
}

template <int GR>
__device__ __forceinline__ void front_store_gather(const FastSmem &s, const FastLayout &L, int t, int v, int nvalid,
                                                   const uint32_t g[GR]) {
  const uint32_t *key = keys_of(s, L, v);
  uint8_t *fsb = s.fsw + (v & 1) * kOrders * L.U;
  CUCM_UNROLL
  for (int h = 0; h < GR / 8; h++) {
    const int j = t + h * kFrontThreads;
    if (j < nvalid) {
      uint32_t b[kOrders];
      CUCM_UNROLL
      for (int o = 0; o < kOrders; o++) b[o] = (g[8 * h + o] >> (8 * (key[o * L.ks + j] & 3))) & 0xffu;
      *reinterpret_cast<uint2 *>(fsb + j * kOrders) =
          make_uint2(b[0] | b[1] << 8 | b[2] << 16 | b[3] << 24, b[4] | b[5] << 8 | b[6] << 16 | b[7] << 24);
    }
  }
}

constexpr uint64_t kTailOffloadBits = 4096;  // shorter stale tails are coded in place

template <int GR>
__device__ void compress_fast_one(const ChunkTask &t, uint8_t *slot, const FastSmem &s, const FastLayout &L,
                                  const ModelInit *init, uint32_t *status, TailTask *tails, uint32_t *tail_count,
                                  uint32_t roles) {
  const int tid = threadIdx.x;
  const int pw = tid >> 5, lane = tid & 31;
  const int warp = (int)((roles >> (4 * pw)) & 15u);
  const int U = L.U;
  const uint64_t len = t.in_len < t.cs ? t.in_len : t.cs;
  const uint64_t total_bits = 8ull * t.cs;
  const uint64_t data_bits = 8ull * len;
  const int nU = (int)((data_bits + U - 1) / U);
  const bool front = warp >= kWFront;
  const int ft = (warp - kWFront) * 32 + lane;
  auto ncode_of = [&](int v) -> int {
    const uint64_t b = (uint64_t)v * U;
    return b >= total_bits ? 0 : (int)(total_bits - b < (uint64_t)U ? total_bits - b : (uint64_t)U);
  };

  for (int i = tid; i < kOrders * 256; i += blockDim.x) s.rec[(i >> 8) * kRecRow + (i & 255)] = init->statep[i >> 8][i & 255];
  for (int i = tid; i < kMixCtx * kOrders; i += blockDim.x) s.w[i] = init->w[i];
  for (int i = tid; i < 2 * U; i += blockDim.x) s.prm[i] = coder_entry(0);  // cucm_compress_v2.cu:1039-1040
  for (int i = tid; i < 4 * kOrders * kClaim; i += blockDim.x) s.claim[i] = 0;  // (any position is a valid one)

  Coder c{0u, 0xffffffffu, 0, 0};
  uint32_t g[GR];
  uint32_t wbyte = 0;
  __syncthreads();

  // Prologue: keys, links and gathers of unit 0.
  if (front) {
    wbyte = window_load(t.in, len, U, 0, ft);
    if (ft < U / 8 + 7) s.win[ft] = (uint8_t)wbyte;
    front_sync();
    front_keys(s, L, ft, 0, fast_nvalid(data_bits, U, 0));
    if (nU > 1) wbyte = window_load(t.in, len, U, 1, ft);
    front_sync();
    front_links_unit<GR>(s, L, ft, 0, fast_nvalid(data_bits, U, 0));
    front_gather<GR>(s, L, slot, ft, 0, fast_nvalid(data_bits, U, 0), g);
    front_store_gather<GR>(s, L, ft, 0, fast_nvalid(data_bits, U, 0), g);
  }
  __syncthreads();

  for (int tau = 0; tau < nU + 2; tau++) {
    const int um = tau - 1;
    const int nv1 = fast_nvalid(data_bits, U, tau + 1);
    int smps[2][kOrders];
    if (warp == kWChain || front) {
      if (front && um >= 0 && um < nU) front_probs(s, L, ft, um, fast_nvalid(data_bits, U, um), smps);
      named_barrier(1, kSnapThreads);
    }
    // keys and gathers of unit tau+1; the gathers land while the front mixes
    // and links (keys a tick earlier, so that the gathers can go out first:
    // within 2 % either way, and a third unit's keys to keep)
    if (front && tau + 1 < nU) {
      if (ft < U / 8 + 7) s.win[ft] = (uint8_t)wbyte;
      front_sync();
      front_keys(s, L, ft, tau + 1, nv1);
      if (tau + 2 < nU) wbyte = window_load(t.in, len, U, tau + 2, ft);
      front_sync();
      front_gather<GR>(s, L, slot, ft, tau + 1, nv1, g);
    }
    if (warp == kWChain) {
      if (um >= 0 && um < nU && lane < kOrders) fast_chain(s, L, lane, um, fast_nvalid(data_bits, U, um));
    } else if (warp == kWCoder) {
      const int uc = tau - 2;
      if (uc >= 0 && uc < nU) {
        coder_run_p(c, s.prm + (uc & 1) * U, s.stage, L.stage, ncode_of(uc));
        coder_flush_p(c, s.stage, L.stage, t.out, t.out_cap);
      }
    } else if (warp == kWWalk) {
      if (tau < nU) {
        uint4 *z4 = reinterpret_cast<uint4 *>(s.ns + (tau & 1) * kOrders * L.NSLOT);
        for (int i = lane; i < kOrders * L.NSLOT / 16; i += 32) z4[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
        __syncwarp();
        walk_unit(s, L, slot, lane, tau, fast_nvalid(data_bits, U, tau));
        walk_sort(s, L, lane, tau, fast_nvalid(data_bits, U, tau));
      }
    } else {
      if (um >= 0 && um < nU) front_mix(s, L, ft, um, fast_nvalid(data_bits, U, um), smps);
      if (tau + 1 < nU) {
        front_links_unit<GR>(s, L, ft, tau + 1, nv1);
        front_store_gather<GR>(s, L, ft, tau + 1, nv1, g);
      }
    }
    __syncthreads();
  }

  if (warp == kWCoder) {
    const uint2 *last = s.prm + ((nU - 1) & 1) * U;
    const uint64_t coded = (uint64_t)nU * U;
    const uint64_t left = total_bits > coded ? total_bits - coded : 0;
    if (tails && left >= kTailOffloadBits) {
      // the stale tail goes to the tail pass: the ring drains to the
      // payload, the coder state and the unit buffer to a tail task, and the
      // CTA moves on to its next chunk
      const uint32_t mask = (uint32_t)L.stage - 1;
      for (uint64_t i = c.flushed + lane; i < c.head; i += 32)
        if (i < t.out_cap) t.out[i] = s.stage[(uint32_t)i & mask];
      uint32_t k = 0;
      if (lane == 0) k = atomicAdd(tail_count, 1u);
      k = __shfl_sync(0xffffffffu, k, 0);
      TailTask &T = tails[k];
      for (int j = lane; j < U; j += 32) T.prm[j] = (uint16_t)coder_entry_u16(last[j]);
      if (lane == 0) {
        T.out = t.out;
        T.cap = t.out_cap;
        T.result = t.result;
        T.head = c.head;
        T.bits = left;
        T.x1 = c.x1;
        T.x2 = c.x2;
        T.unit = (uint32_t)U;
      }
      __syncwarp();
    } else {
      for (int v = nU;; v++) {
        const int n = ncode_of(v);
        if (n <= 0) break;
        coder_run_p(c, last, s.stage, L.stage, n);
        coder_flush_p(c, s.stage, L.stage, t.out, t.out_cap);
      }
      coder_finish_p(c, s.stage, L.stage, t.out, t.out_cap, t.result);
      if (lane == 0 && c.head > t.out_cap) atomicOr(status, (uint32_t)kDevOverflow);
    }
  }
  __syncthreads();
}

// Persistent CTA: chunks from the work queue, one after the other, each in
// this CTA's slot tables (restored to the initial model between chunks).
template <int GR>
__device__ __forceinline__ void compress_fast_loop(const ChunkTask *tasks, uint32_t ntasks, uint8_t *slots,
                                                   const uint8_t *init_tables, const ModelInit *init,
                                                   uint32_t *queue, uint32_t *status, int unit, TailTask *tails,
                                                   uint32_t *tail_count, uint32_t roles) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const FastLayout L = make_fast_layout(unit);
  const FastSmem s = carve_fast(smem_raw, L);
  uint8_t *slot = slots + (size_t)blockIdx.x * kSlotTableBytes;
  copy_tables(&g_tables, s.tab);
  __shared__ uint32_t s_task;
  bool fresh = true;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_task = atomicAdd(queue, 1u);
    __syncthreads();
    const uint32_t ti = s_task;
    if (ti >= ntasks) break;
    const ChunkTask t = tasks[ti];
    if (t.unit != (uint32_t)unit || t.cs == 0 || t.in_len == 0) {
      if (threadIdx.x == 0) {
        atomicOr(status, (uint32_t)kDevBadTask);
        *t.result = ~0ull;
      }
      continue;
    }
    if (!fresh) {
      reset_slot(slot, init_tables);
      __syncthreads();
    }
    fresh = false;
    compress_fast_one<GR>(t, slot, s, L, init, status, tails, tail_count, roles);
  }
}

// Units up to 128 bits.  (Capping the registers at 96 so that three CTAs
// share an SM made each CTA 35-44 % slower: more CTAs did not pay for it.)
__global__ void __launch_bounds__(kFastThreads, 2)
    compress_fast_kernel(const ChunkTask *tasks, uint32_t ntasks, uint8_t *slots, const uint8_t *init_tables,
                         const ModelInit *init, uint32_t *queue, uint32_t *status, int unit, TailTask *tails,
                         uint32_t *tail_count, uint32_t roles) {
  compress_fast_loop<8>(tasks, ntasks, slots, init_tables, init, queue, status, unit, tails, tail_count, roles);
}

// Units of 160..256 bits: 16 gathers a thread, 44 bytes spilled at the 128
// registers of two CTAs.
__global__ void __launch_bounds__(kFastThreads, 2)
    compress_fast_kernel_wide(const ChunkTask *tasks, uint32_t ntasks, uint8_t *slots, const uint8_t *init_tables,
                              const ModelInit *init, uint32_t *queue, uint32_t *status, int unit, TailTask *tails,
                              uint32_t *tail_count, uint32_t roles) {
  compress_fast_loop<16>(tasks, ntasks, slots, init_tables, init, queue, status, unit, tails, tail_count, roles);
}

// One chunk, task passed by value, tables at `slot` (no work queue); the
// stale tail is coded in place.
template <int GR>
__global__ void __launch_bounds__(kFastThreads, 2)
    compress_fast_single_kernel(const ChunkTask t, uint8_t *slot, const ModelInit *init, uint32_t *status) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const FastLayout L = make_fast_layout((int)t.unit);
  const FastSmem s = carve_fast(smem_raw, L);
  copy_tables(&g_tables, s.tab);
  __syncthreads();
  compress_fast_one<GR>(t, slot, s, L, init, status, nullptr, nullptr, kRolesAlone);
}

// The tail pass: one thread per handed-over chunk codes its stale tail (the
// unit buffer again and again up to the chunk end), writes the bytes, the
// flush byte (cucm_compress_v2.cu:902) and the payload length.  `lanes`
// chunks share a warp, each with its unit buffer in a row of shared memory
// (rows 16 bytes apart in the banks).
// One 20 KB buffer at 1 MiB chunks (8.2 million stale bits): 424 -> 260 ms
// against a test after every bit.
inline size_t tail_smem_bytes(int unit, int lanes) {
  return (size_t)lanes * ((size_t)(unit + 2) * sizeof(uint2) + kLaneRing + 4);
}

__global__ void __launch_bounds__(32) compress_tail_kernel(const TailTask *tails, const uint32_t *count,
                                                           uint32_t *status, int unit, int lanes) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int lane = threadIdx.x;
  const uint32_t i = blockIdx.x * (uint32_t)lanes + lane;
  if (lane >= lanes || i >= *count) return;
  const TailTask &T = tails[i];
  uint2 *ent = reinterpret_cast<uint2 *>(smem_raw) + (unit + 2) * lane;
  uint8_t *ring = lane_ring(smem_raw + (size_t)(unit + 2) * lanes * sizeof(uint2), lane);
  for (int j = 0; j < unit; j++) ent[j] = coder_entry(T.prm[j]);
  uint32_t x1 = T.x1, x2 = T.x2;
  const uint64_t cap = T.cap;
  uint64_t base = T.head;  // payload offset of ring position 0
  uint8_t *out = T.out;
  uint32_t head = 0, from = 0;  // bytes since base: produced, written
  uint64_t left = T.bits;
  int j = 0;
  for (; left >= kCoderGroup; left -= kCoderGroup) {
    coder_group_at(ent + j, x1, x2, head, ring, kLaneRing - 1);
    j = j + kCoderGroup == unit ? 0 : j + kCoderGroup;
    if (lane_flush_due(from, head)) lane_flush(ring, base, from, head, out, cap);
  }
  for (int k = 0; k < (int)left; k++) coder_step(ent[j + k], x1, x2, head, ring, kLaneRing - 1);
  ring[head & (kLaneRing - 1)] = (uint8_t)(x1 >> 24);
  head++;
  lane_flush(ring, base, from, head, out, cap);
  base += head;  // (what is left of the last ring)
  *T.result = base;
  if (base > cap) atomicOr(status, (uint32_t)kDevOverflow);
}
