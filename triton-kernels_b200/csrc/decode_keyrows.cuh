// Decode with 17 to 64 q rows per KV head, keys as the rows of the tensor-core tiles.  Part of decode.cu, inside its namespaces.
//
// decode_umma_kernel pads the q rows to the 128 rows of a tcgen05 tile; with 40 rows two thirds of its multiplications, and of the
// accumulator traffic in tensor memory, are padding, and long batches run at the board's power limit (1.37 GHz).  Here a tile is 128
// keys, which are the rows of both products' A operands, read from shared memory where the copies put them, and the q rows are the
// columns (padded to a multiple of 16):
//   S^T = K Q^T   (128 keys x N, A = K tile K-major, B = Q rows K-major)
//   O^T += V^T P^T (128 or 64 elements x N, A = V tile MN-major, B = P, a row of 128 bytes per key in shared memory, MN-major)
// A tile of 128 keys is 2 x 8 MMAs of N columns instead of 2 x 16 of 64 and 128.
//
// Persistent, one CTA to an SM, 24 warps:
//   warps 0-15  softmax: warp w holds the keys of TMEM lane quadrant w % 4 (thread = key) and one or two chunks of eight columns, those
//               of share w / 4.  Exponentials against each column's standing reference, sums per thread and column, P to shared memory.
//               The four warps of a share agree by one barrier with a vote per tile that no exponential was too large for its
//               reference; if one was, and on a unit's first tile, they work out the columns' maxima.
//   warps 16-19 output: read a finished unit's O out of tensor memory, normalise, store, draw the ticket
//   warp 20     MMA issuer, TMEM owner;  warp 21 copies Q and K;  warp 22 copies V;  warp 23 draws the units
// Scores, accumulators, Q and the units' sums exist twice, so that the first tiles of a unit are under way while the last one is
// being finished.  K and V tiles share one ring in the order in which they are consumed: K_0, K_1, V_0, K_2, V_1, ...
// Planner, records, partials and merges are decode_umma_kernel's.
//
// What bounds it: the copies, at head_dim 128.  A tile of 64 KB arrives in some 2 100 cycles; the softmax of 40 columns takes about 1 300, the
// issuing warp 1 350, both beside them.  A unit costs 2.5 us in which its first tile is looked at twice, its sums are added up and the ring
// runs full; the softmax warps' code of those parts runs once a unit, at five cycles an instruction.  Against decode_umma_kernel, us, 40 rows:
// 32 x 1 000 to 33 000 keys in 16-key pages, eight heads, D 128 321 -> 287 (336 -> 299 on another box); 20 x 1 000 to 30 000 236 -> 201;
// 200 x 300 to 4 000 of two heads, 32 rows, 110 -> 88; 15 x 2 000 42 -> 33; D 64, 128 x 500 to 8 000 282 -> 257.
// With eight softmax warps of up to 32 columns D 64 takes 279 there, D 128 the same.  K of the next unit is asked for whenever it
// arrives before the last P does; zeroing V rows behind a short sequence in place of leaving out the steps without a key
// cost the issuing warp 3 000 cycles a unit.
constexpr int kKrTile = 128;
constexpr int kKrMaxRows = 64;
constexpr int kKrThreads = 768;
constexpr int kKrSoftmaxWarps = 16, kKrOutWarp = 16, kKrMmaWarp = 20, kKrKeyWarp = 21, kKrValueWarp = 22, kKrDrawWarp = 23;
constexpr int kKrShares = kKrSoftmaxWarps / 4, kKrShareCols = kKrMaxRows / kKrShares;
constexpr int kKrRingBytes = 160 * 1024;
constexpr int kKrMaxSlots = 10;
constexpr float kKrMaxWeight = 1024.0f;      // P fits 16 bits, and the reference lies at most ten powers of two below the maximum

// A wait asks for a phase by its parity, so a barrier must not complete its next phase before all who wait for this one have seen
// it.  Beside each: what keeps that (g: a tile of the CTA, r: a unit, those of an even and an odd number having barriers of their own).
struct __align__(16) KrCtrl {
  uint64_t full[kKrMaxSlots];    // copies -> MMA warp: a tile.  The next one's copies wait for `empty`
  // MMA warp -> copies, softmax warps (commit): a tile is consumed.  The next one here comes by copies that waited for this.  The softmax warps
  // wait for V of g - 1 before P of g; the next tile in its slot, K of g + 3 at the earliest, is asked for behind P of g + 1
  uint64_t empty[kKrMaxSlots];
  uint64_t q_full[2];     // copies -> MMA warp: a unit's Q.  r + 2 waits for q_empty of r
  uint64_t q_empty[2];    // MMA warp -> copies (commit, every unit).  r + 2 needs q_full of r + 2
  uint64_t s_full[2];     // MMA warp -> softmax warps (commit): scores of a tile.  g + 2 is asked for after P of g
  uint64_t p_ready;       // softmax warps -> MMA warp: P of a tile.  P of g + 1 waits for the product of g
  uint64_t o_done[2];     // MMA warp -> output warps (commit): a unit's last, with or without keys.  r + 2 waits for o_free of r
  uint64_t o_free[2];     // output warps -> MMA, softmax warps: the accumulator and the sums have been read.  r + 2 needs o_done and l_ready of r + 2
  uint64_t l_ready[2];    // softmax warps -> output warps: a unit's sums and references.  r + 2 waits for o_free of r
  uint64_t rows_out;      // output warps, all of them on both sides: a cut unit's partial rows are written and fenced
  uint64_t drained;       // once
  uint64_t may_draw[2];   // copies of K -> scheduler: the end of a unit (of that parity) is near.  Units behind r are published after the wait in r
  // scheduler -> all others, and back: a unit's record.  r + 4 waits for all of them to be done with r
  uint64_t unit_full[kUmmaUnitRing], unit_empty[kUmmaUnitRing];
  UmmaUnit unit[kUmmaUnitRing];
  int unit_ring[kUmmaUnitRing];
  int published;
  uint32_t tmem_base;
  int abort_flag, abort_round;
  int ready, n_reserved, n_claimed;
  int claimed[kUmmaMaxClaims];
  // a softmax warp's own copies, by column of its share: minus the reference; what a moved reference scales by
  __align__(16) float ref[kKrSoftmaxWarps][kKrShareCols];
  __align__(16) float scale[kKrSoftmaxWarps][kKrShareCols];
  float peak[2][kKrShares][4][kKrShareCols];     // maxima by tile parity, share, quadrant, column
  float sums[2][4][kKrMaxRows];                  // a unit's sums by unit parity, quadrant, column
  float refs[2][kKrMaxRows];                     // ... and references
  __align__(16) float inv[4][kKrMaxRows];    // an output warp's own copy: one over the sums
  unsigned hidden[kKrShares][17];      // by share: columns whose draft is one of the first so many
};

template <int D> struct KrPlan {
  static constexpr int kBlocks = D / 64;
  static constexpr int kTileBytes = kKrTile * D * 2;
  static constexpr int kSlots = kKrRingBytes / kTileBytes;
  static constexpr int kQBytes = kBlocks * kKrMaxRows * 128;
  static constexpr int kQOff = kKrRingBytes;
  static constexpr int kPOff = kQOff + 2 * kQBytes;
  static constexpr int kCtrlOff = kPOff + kKrTile * 128;
  static constexpr int kTotal = kCtrlOff + static_cast<int>(sizeof(KrCtrl)) + 1024;
  static_assert(kSlots <= kKrMaxSlots && kTotal <= 227 * 1024, "shared memory");
};

// Copies of one operand's tiles; see PageAhead for the entries of pages.
struct KrCopies {
  const CUtensorMap* map;
  const int* table;
  int lane, box_shift, page_shift, page_size;
  bool paged, whole;           // whole: a box brings both column blocks (make_kv_groups_map)
  int head, row0, t_begin, t_end;
  int now, next;
  __device__ __forceinline__ void read(int first_box, int& e) const {
    const int t = t_begin + ((first_box + lane) << box_shift);
    e = t < t_end ? __ldcg(table + (page_shift >= 0 ? t >> page_shift : t / page_size)) : kNoPage;
  }
  __device__ __forceinline__ void start(const DecodeParams& p, const UmmaUnit& w, const int* tables) {
    t_begin = w.t_begin;
    t_end = w.t_end;
    head = w.h;
    row0 = static_cast<int>(w.seq_start);
    if (p.layout == B200ATTN_DENSE) { head = 0; row0 = static_cast<int>((static_cast<long long>(w.b) * p.kv_heads + w.h) * p.max_kv); }
    if (!paged) return;
    table = tables + static_cast<long long>(w.b) * p.table_stride;
    if (p.num_pages <= 0 && t_begin < t_end && lane == 0) p.header[0] = DEV_ERR_PAGE_RANGE;
    read(0, now);
    read(32, next);
  }
  // the keys of tile `tile` that the unit has, to `dst`
  template <int D> __device__ __forceinline__ void issue(const DecodeParams& p, int tile, uint32_t dst, uint32_t bar) {
    constexpr int kBlocks = D / 64;
    const int t0 = t_begin + tile * kKrTile;
    const int boxes = kKrTile >> box_shift, box_rows = 1 << box_shift;
    int n = min(boxes, (t_end - t0 + box_rows - 1) >> box_shift);
    int row = row0 + t0 + (lane << box_shift);
    if (paged) {
      if (((tile * boxes) & 31) == 0 && tile > 0) { now = next; read(tile * boxes + 32, next); }
      if (p.num_pages <= 0) n = 0;
      const int page = __shfl_sync(0xffffffffu, now, (tile * boxes + lane) & 31);
      if (lane < n) {
        // an entry outside the cache is reported and replaced by page 0: never dereferenced, output stays finite
        const bool bad = page < 0 || page >= p.num_pages;
        if (bad) p.header[0] = DEV_ERR_PAGE_RANGE;
        const int t = t0 + (lane << box_shift);
        row = (bad ? 0 : page) * page_size + (page_shift >= 0 ? t & (page_size - 1) : t % page_size);
      }
    }
    if (lane == 0) {
      if (n > 0) ptx::mbar_arrive_expect_tx(bar, static_cast<uint32_t>(n * box_rows * 128 * kBlocks));
      else ptx::mbar_arrive(bar);
    }
    __syncwarp();
    if (lane < n) {
      const uint32_t to = dst + lane * box_rows * 128 * (whole ? kBlocks : 1);
      if (whole) {
        ptx::tma_load_5d(to, map, bar, 0, 0, 0, row >> 3, head);
      } else {
#pragma unroll
        for (int c = 0; c < kBlocks; ++c) ptx::tma_load_3d(to + c * kKrTile * 128, map, bar, c * 64, head, row);
      }
    }
  }
};

// Reduces 16 columns, of which every lane holds a row, over the warp: lanes l and l + 16 end up with column l.
template <typename Op> __device__ __forceinline__ float column_reduce(float (&f)[16], int lane, Op op) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float got = __shfl_xor_sync(0xffffffffu, up ? f[i] : f[i + o], o);
      f[i] = op(up ? f[i + o] : f[i], got);
    }
  }
  return op(f[0], __shfl_xor_sync(0xffffffffu, f[0], 16));
}
// first chunk of eight columns of share s, of `chunks`
__device__ __forceinline__ int share_start(int chunks, int s) { return (chunks * s + kKrShares - 1) / kKrShares; }

// whether the copies of pages of `box_rows` rows (the largest power of two that divides the page size, at most 64) suit
constexpr bool keyrows_boxes(int box_rows) { return box_rows >= 8; }

template <typename T, int D, typename OutT>
__global__ void __launch_bounds__(kKrThreads, 1) decode_keyrows_kernel(const __grid_constant__ CUtensorMap tm_q,
                                                                       const __grid_constant__ CUtensorMap tm_k,
                                                                       const __grid_constant__ CUtensorMap tm_v,
                                                                       const DecodeParams p) {
  using namespace ptx;
  using Plan = KrPlan<D>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  KrCtrl* ctrl = reinterpret_cast<KrCtrl*>(smem + Plan::kCtrlOff);
  const uint32_t smem_base = smem_u32(smem);
  constexpr int kSlots = Plan::kSlots;
  constexpr int kSCol = 0, kOCol = 2 * kKrMaxRows;      // TMEM columns: two score tiles, two accumulators

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int R = p.rows;
  const int cols = (R + 15) & ~15;                      // columns of the MMAs
  const int chunks = (R + 7) >> 3;                      // of eight columns
  const bool whole = D == 128 && p.layout == B200ATTN_PAGED;          // layout of the tiles: see KrCopies

  if (tid == 0) {
    for (int i = 0; i < kSlots; ++i) { mbar_init(smem_u32(&ctrl->full[i]), 1); mbar_init(smem_u32(&ctrl->empty[i]), 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&ctrl->q_full[i]), 1);
      mbar_init(smem_u32(&ctrl->q_empty[i]), 1);
      mbar_init(smem_u32(&ctrl->may_draw[i]), 1);
      mbar_init(smem_u32(&ctrl->s_full[i]), 1);
      mbar_init(smem_u32(&ctrl->o_done[i]), 1);
      mbar_init(smem_u32(&ctrl->o_free[i]), 4);
      mbar_init(smem_u32(&ctrl->l_ready[i]), kKrSoftmaxWarps);
    }
    mbar_init(smem_u32(&ctrl->p_ready), kKrSoftmaxWarps);
    mbar_init(smem_u32(&ctrl->rows_out), 4);
    mbar_init(smem_u32(&ctrl->drained), 1);
    for (int i = 0; i < kUmmaUnitRing; ++i) {
      mbar_init(smem_u32(&ctrl->unit_full[i]), 1);
      mbar_init(smem_u32(&ctrl->unit_empty[i]), kKrSoftmaxWarps + 4 + 3);
    }
    ctrl->published = 0;
    ctrl->abort_flag = 0;
    ctrl->abort_round = 0x7fffffff;
    mbar_fence_init();
  }
  if (tid >= 32 && tid < 32 + 17 * kKrShares) {
    const int share = (tid - 32) / 17, drafts = (tid - 32) % 17;
    unsigned bits = 0;
    int draft = share_start(chunks, share) * 8 % p.q_len;
    for (int i = 0; i < kKrShareCols; ++i) {
      if (draft < drafts) bits |= 1u << i;
      if (++draft == p.q_len) draft = 0;
    }
    ctrl->hidden[share][drafts] = bits;
  }
  if (warp == kKrMmaWarp) {
    tmem_alloc(smem_u32(&ctrl->tmem_base), 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctrl->tmem_base;
  volatile int* abort_flag = &ctrl->abort_flag;
  // (no launch_dependents here: see decode_umma_kernel)
  ptx::grid_dep_wait();      // the planner's records are complete and visible from here on
  const int G = static_cast<int>(gridDim.x), me = static_cast<int>(blockIdx.x);
  const int n_units = p.header[2] * p.kv_heads;
  // Units are handed out as in decode_umma_kernel.  unit_at(r): the CTA's r-th unit, n_units or more when there is none, -1 when the
  // (bounded) wait for the scheduler ran out; its record lies in the ring beside it.
  auto unit_at = [&](int r) -> int {
    if (!warp_wait(smem_u32(&ctrl->unit_full[r % kUmmaUnitRing]), (r / kUmmaUnitRing) & 1)) return -1;
    return *reinterpret_cast<volatile int*>(&ctrl->unit_ring[r % kUmmaUnitRing]);
  };
  auto unit_done = [&](int r) {   // this warp will not read slot r again
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctrl->unit_empty[r % kUmmaUnitRing]));
  };
  auto rows_of = [&](const UmmaUnit& w) {
    return (static_cast<long long>(w.b) * p.q_heads + static_cast<long long>(w.h) * p.head_stride + p.head0) * p.q_len;
  };
  auto tiles_of = [](const UmmaUnit& w) { return w.t_end > w.t_begin ? (w.t_end - w.t_begin + kKrTile - 1) / kKrTile : 0; };
  // places in the ring of the K and the V tile number g of this CTA
  auto key_place = [](int g) { return g == 0 ? 0 : 2 * g - 1; };
  auto value_place = [](int g) { return 2 * g + 2; };
  auto copies_for = [&](const CUtensorMap* map) {
    KrCopies c;
    c.map = map;
    c.table = nullptr;
    c.lane = lane;
    c.box_shift = p.box_shift;
    c.page_shift = p.page_shift;
    c.page_size = p.page_size;
    c.paged = p.layout == B200ATTN_PAGED;
    c.whole = whole;
    c.head = c.row0 = c.t_begin = c.t_end = 0;
    c.now = c.next = kNoPage;
    return c;
  };
  // the ring slot of a place, once what it held has been consumed
  auto slot_free = [&](int place) -> bool {
    const int use = place / kSlots;
    return use == 0 || (warp_wait(smem_u32(&ctrl->empty[place % kSlots]), (use - 1) & 1) && !*abort_flag);
  };
  // bounded drain of this warp's copies still in flight before the CTA may exit
  auto drain = [&](auto place_of, int g) {
    for (int t = max(0, g - (kSlots + 1) / 2); t < g; ++t) {
      const int place = place_of(t);
      mbar_wait(smem_u32(&ctrl->full[place % kSlots]), (place / kSlots) & 1);
    }
  };

  if (warp == kKrDrawWarp) {
    // =========================== scheduler ===========================
    auto publish = [&](int rr, int u, const UmmaUnit& w) {            // lane 0
      ctrl->unit_ring[rr % kUmmaUnitRing] = u;
      ctrl->unit[rr % kUmmaUnitRing] = w;
      ctrl->published = rr + 1;
      mbar_arrive(smem_u32(&ctrl->unit_full[rr % kUmmaUnitRing]));
    };
    // Dealt out (slots > 0): the CTA's units are the items of its slot, in order.  Else its first unit is its own index, and the others
    // are drawn.  That takes two trips to L2, so a unit is drawn when the copies of the one before near their end, and behind a short
    // unit one earlier.
    const int slots = p.header[5];
    int u = me, u_end = n_units;
    if (slots > 0) {
      const int slot = me / p.kv_heads;
      const int* slot_first = reinterpret_cast<const int*>(p.item_info + 2 * static_cast<long long>(p.max_items)) - (slots + 1);
      u = n_units;
      if (slot < slots) {
        u = __ldcg(slot_first + slot) * p.kv_heads + me % p.kv_heads;
        u_end = __ldcg(slot_first + slot + 1) * p.kv_heads;
      }
    }
    bool ok = true;
    for (int r = 0; ok; ++r) {
      if (u >= u_end) u = n_units;
      UmmaUnit w = {};
      if (u < n_units) w = umma_unit(p, u);
      if (r >= kUmmaUnitRing)
        ok = warp_wait(smem_u32(&ctrl->unit_empty[r % kUmmaUnitRing]), (r / kUmmaUnitRing - 1) & 1) && !*abort_flag;
      if (!ok) break;
      if (lane == 0) publish(r, u, w);
      __syncwarp();
      if (u >= n_units) break;
      if (slots > 0) {
        u += p.kv_heads;
      } else {
        const int behind = tiles_of(w) <= 2 ? r - 1 : r;
        if (behind >= 0) ok = warp_wait(smem_u32(&ctrl->may_draw[behind & 1]), (behind >> 1) & 1) && !*abort_flag;
        if (!ok) break;
        if (lane == 0) u = min(G + atomicAdd(p.header + 4, 1), n_units);
        u = __shfl_sync(0xffffffffu, u, 0);
      }
    }
    if (!ok && lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
  } else if (warp == kKrKeyWarp) {
    // =========================== copies of Q and K ===========================
    if (lane == 0) { prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_k); }
    bool ok = true;
    int g = 0, q_uses = 0;
    KrCopies copies = copies_for(&tm_k);
    for (int r = 0; ok; ++r) {
      const int u = unit_at(r);
      if (u < 0) { ok = false; break; }
      if (u >= n_units) break;
      const UmmaUnit w = ctrl->unit[r % kUmmaUnitRing];
      unit_done(r);
      copies.start(p, w, p.k_table);
      const int n = tiles_of(w);
      // Q rows (an empty unit only takes its turn)
      if (r >= 2) ok = warp_wait(smem_u32(&ctrl->q_empty[r & 1]), ((r >> 1) - 1) & 1) && !*abort_flag;
      if (!ok) break;
      if (lane == 0) {
        const uint32_t bar = smem_u32(&ctrl->q_full[r & 1]);
        if (n > 0) {
          mbar_arrive_expect_tx(bar, static_cast<uint32_t>(Plan::kBlocks * cols * 128));
          for (int c = 0; c < Plan::kBlocks; ++c)
            tma_load_3d(smem_base + Plan::kQOff + (r & 1) * Plan::kQBytes + c * kKrMaxRows * 128, &tm_q, bar, c * 64, 0,
                        static_cast<int>(rows_of(w)));
        } else {
          mbar_arrive(bar);
        }
      }
      q_uses = r + 1;
      __syncwarp();
      const int near = max(0, n - 3);
      if (n == 0 && lane == 0) mbar_arrive(smem_u32(&ctrl->may_draw[r & 1]));
      for (int tile = 0; tile < n; ++tile, ++g) {
        const int place = key_place(g);
        ok = slot_free(place);
        if (!ok) break;
        if (tile == near && lane == 0) mbar_arrive(smem_u32(&ctrl->may_draw[r & 1]));
        copies.template issue<D>(p, tile, smem_base + place % kSlots * Plan::kTileBytes, smem_u32(&ctrl->full[place % kSlots]));
      }
    }
    if (!ok) {
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
      drain(key_place, g);
      for (int i = max(0, q_uses - 2); i < q_uses; ++i) mbar_wait(smem_u32(&ctrl->q_full[i & 1]), (i >> 1) & 1);
    }
  } else if (warp == kKrValueWarp) {
    // =========================== copies of V ===========================
    if (lane == 0) prefetch_tensormap(&tm_v);
    bool ok = true;
    int g = 0;
    KrCopies copies = copies_for(&tm_v);
    for (int r = 0; ok; ++r) {
      const int u = unit_at(r);
      if (u < 0) { ok = false; break; }
      if (u >= n_units) break;
      const UmmaUnit w = ctrl->unit[r % kUmmaUnitRing];
      unit_done(r);
      copies.start(p, w, p.v_table);
      const int n = tiles_of(w);
      for (int tile = 0; tile < n; ++tile, ++g) {
        const int place = value_place(g);
        ok = slot_free(place);
        if (!ok) break;
        copies.template issue<D>(p, tile, smem_base + place % kSlots * Plan::kTileBytes, smem_u32(&ctrl->full[place % kSlots]));
      }
    }
    if (!ok) {
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
      drain(value_place, g);
    }
  } else if (warp == kKrMmaWarp) {
    // =========================== MMA issuer ===========================
    constexpr int kFmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
    const uint32_t idesc_s = make_idesc_f16(kKrTile, 0, kFmt, 0) | static_cast<uint32_t>(cols >> 3) << 17;
    const uint32_t idesc_o = make_idesc_f16(kKrTile, 0, kFmt, 1, 1) | static_cast<uint32_t>(cols >> 3) << 17;
    // tiles lie in groups of eight keys, both column blocks of a group together, or a column block after the other; at head_dim
    // 64 the upper 64 rows of O^T are a block's worth of other bytes of this CTA's shared memory, which nobody reads out
    const uint32_t group = whole ? 2048 : 1024;
    const uint32_t block = whole || D == 64 ? 1024 : kKrTile * 128;
    const uint64_t kdesc = make_smem_desc_sw128(smem_base, 16, group);
    const uint64_t vdesc = make_smem_desc_sw128(smem_base, block, group);
    const uint64_t qdesc = make_smem_desc_sw128(smem_base + Plan::kQOff, 16);
    const uint64_t pdesc = make_smem_desc_sw128(smem_base + Plan::kPOff, 1024);
    const uint64_t k_block = block >> 4, v_step = 2 * group >> 4;
    const uint32_t lead = elect_one();
    bool ok = true, ahead = false;               // ahead: the unit's first scores have been asked for
    int g = 0;                                   // tiles consumed so far, over all units
    // scores of tile number gi, a tile of unit r
    auto issue_s = [&](int gi, int r, bool last) -> bool {
      const int place = key_place(gi), slot = place % kSlots;
      const bool good = mbar_wait_ready(smem_u32(&ctrl->full[slot]), (place / kSlots) & 1);
      tc_fence_after();
      mma_keys_by_rows<D / 16>(tmem + kSCol + (gi & 1) * kKrMaxRows, kdesc + static_cast<uint64_t>(slot * Plan::kTileBytes >> 4),
                               qdesc + static_cast<uint64_t>((r & 1) * Plan::kQBytes >> 4), idesc_s, k_block, lead);
      mma_commit_lead(smem_u32(&ctrl->s_full[gi & 1]), lead);
      mma_commit_lead(smem_u32(&ctrl->empty[slot]), lead);
      if (last) mma_commit_lead(smem_u32(&ctrl->q_empty[r & 1]), lead);
      return good;
    };
    for (int r = 0; ok; ++r) {
      const int u = unit_at(r);
      if (u < 0) { ok = false; break; }
      if (u >= n_units) break;
      const UmmaUnit& w = ctrl->unit[r % kUmmaUnitRing];
      const int n = tiles_of(w), t_begin = w.t_begin, t_end = w.t_end;
      if (!ahead) {
        ok = warp_wait(smem_u32(&ctrl->q_full[r & 1]), (r >> 1) & 1) && !*abort_flag;
        if (!ok) break;
        if (n > 0) ok = __all_sync(0xffffffffu, issue_s(g, r, n == 1));
        else mma_commit_lead(smem_u32(&ctrl->q_empty[r & 1]), lead);
        if (!ok) break;
      }
      ahead = false;
      if (n == 0) {
        // (like a unit with keys, whose first product waits for this: else o_done completes twice before its waiters have looked)
        if (r >= 2) ok = warp_wait(smem_u32(&ctrl->o_free[r & 1]), ((r >> 1) - 1) & 1) && !*abort_flag;
        if (!ok) break;
        mma_commit_lead(smem_u32(&ctrl->o_done[r & 1]), lead);
      }
      for (int tile = 0; tile < n && ok; ++tile, ++g) {
        const bool last = tile + 1 == n;
        bool good = true;
        if (!last) good = issue_s(g + 1, r, tile + 2 == n);
        const int place = value_place(g), slot = place % kSlots;
        good = mbar_wait_ready(smem_u32(&ctrl->full[slot]), (place / kSlots) & 1) && good;
        const int valid = t_end - (t_begin + tile * kKrTile);
        const int steps = valid < kKrTile ? (valid + 15) >> 4 : kKrTile / 16;      // of sixteen keys
        if (valid & 15 && valid < kKrTile) {
          // The last step's keys past the unit's end carry P == 0 but their V rows may hold anything: zero them so 0 * x stays 0.  (Steps
          // without a key are left out: zeroing a tile of 20 keys took this warp 3 000 cycles.)
          unsigned char* vbuf = smem + slot * Plan::kTileBytes;
          for (int i = lane; i < (steps * 16 - valid) * 8; i += 32) {
            const int key = valid + (i >> 3);
#pragma unroll
            for (int c = 0; c < Plan::kBlocks; ++c)
              *reinterpret_cast<uint4*>(vbuf + (key >> 3) * group + c * block + (key & 7) * 128 + (i & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_proxy_async_smem();
          __syncwarp();
        }
        if (last) {
          // The next unit's first scores, if what they need arrives before this tile's P does
          const int at = (r + 1) % kUmmaUnitRing, next_place = key_place(g + 1);
          int n2 = -1;
          for (uint32_t tries = 0; tries < kWaitTries && !__all_sync(0xffffffffu, mbar_test(smem_u32(&ctrl->p_ready), g & 1)); ++tries) {
            if (n2 == 0 || ahead) break;
            if (n2 < 0) {
              if (!__all_sync(0xffffffffu, mbar_test(smem_u32(&ctrl->unit_full[at]), ((r + 1) / kUmmaUnitRing) & 1))) continue;
              n2 = *reinterpret_cast<volatile int*>(&ctrl->unit_ring[at]) < n_units ? tiles_of(ctrl->unit[at]) : 0;
            }
            if (n2 > 0 && __all_sync(0xffffffffu, mbar_test(smem_u32(&ctrl->q_full[(r + 1) & 1]), ((r + 1) >> 1) & 1) &&
                                                      mbar_test(smem_u32(&ctrl->full[next_place % kSlots]), (next_place / kSlots) & 1))) {
              good = issue_s(g + 1, r + 1, n2 == 1) && good;
              ahead = true;
            }
          }
        }
        good = mbar_wait_ready(smem_u32(&ctrl->p_ready), g & 1) && good;
        if (tile == 0 && r >= 2) good = mbar_wait(smem_u32(&ctrl->o_free[r & 1]), ((r >> 1) - 1) & 1) && good;
        tc_fence_after();
        mma_values_by_weights(tmem + kOCol + (r & 1) * kKrMaxRows, vdesc + static_cast<uint64_t>(slot * Plan::kTileBytes >> 4), pdesc,
                              idesc_o, v_step, tile > 0 ? 1u : 0u, steps, lead);
        mma_commit_lead(smem_u32(&ctrl->empty[slot]), lead);      // (the softmax warps wait for it too)
        if (last) mma_commit_lead(smem_u32(&ctrl->o_done[r & 1]), lead);
        ok = __all_sync(0xffffffffu, good);
      }
      if (ok) unit_done(r);
    }
    if (!ok) {
      // (the other warps may have gone on since: no unit of the ring is known to be right)
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; ctrl->abort_round = 0; }
      mma_commit_lead(smem_u32(&ctrl->drained), lead);
      warp_wait(smem_u32(&ctrl->drained), 0);
    }
  } else if (warp < kKrSoftmaxWarps) {
    // =========================== softmax warps: thread = key ===========================
    const int quad = warp & 3, share = warp >> 2, key = quad * 32 + lane;
    const int col0 = share_start(chunks, share) * 8, my_chunks = share_start(chunks, share + 1) - col0 / 8;
    const int bar_id = 1 + share;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const float sl2 = p.scale_log2;
    const uint64_t sl2_2 = pack_f2(sl2, sl2);
    const uint32_t p_row = smem_base + Plan::kPOff + key * 128;
    const int col = lane & 15;       // the column whose reference this lane keeps
    float* const my_ref = ctrl->ref[warp];
    float* const my_scale = ctrl->scale[warp];
    // The four warps of a share take the same way through everything below: whatever makes one leave (a wait that ran out) is
    // voted on at a barrier that all of them come to.  One that does not even know its unit has a vote of its own, which the others meet
    // at the first barrier of a unit, or behind the last.
    bool fine = true;
    int g = 0;
    // tile number t's product with V (its slot cannot have been used and given back once more: that takes P of later tiles)
    auto product_done = [&](int t) -> bool {
      const int place = value_place(t);
      return mbar_wait_ready(smem_u32(&ctrl->empty[place % kSlots]), (place / kSlots) & 1);
    };
    for (int r = 0;; ++r) {
      const int u = unit_at(r);
      fine = fine && u >= 0;
      if (u < 0 || u >= n_units) { fine = !named_bar_any(bar_id, 128, !fine); break; }
      const UmmaUnit& w = ctrl->unit[r % kUmmaUnitRing];
      const int n = tiles_of(w), t_begin = w.t_begin, t_end = w.t_end;
      const int first_lim = p.causal ? min(t_end - 1, w.len - p.q_len) : t_end - 1;      // last key that all rows see
      const int lim0 = w.len - p.q_len;
      uint64_t sums[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) sums[i] = 0;
      float m_col = -INFINITY;         // the reference of column `lane % 16` of this share
      bool unset = true;               // some column has none yet
      bool lost = false;
      for (int tile = 0; tile < n; ++tile, ++g) {
        fine = mbar_wait_ready(smem_u32(&ctrl->s_full[g & 1]), (g >> 1) & 1) && fine;
        tc_fence_after();
        const int t0 = t_begin + tile * kKrTile;
        const uint32_t tS = tmem + kSCol + (g & 1) * kKrMaxRows + lane_off + col0;
        uint32_t v[16];
        auto load_scores = [&]() {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (c < my_chunks) tmem_ld8(tS + c * 8, v + c * 8);
            else {
#pragma unroll
              for (int i = 0; i < 8; ++i) v[c * 8 + i] = 0u;
            }
          }
          tmem_wait_ld_regs(v);
          if (t0 + kKrTile - 1 > first_lim) {
            // hidden keys are -inf: beyond the unit, or to drafts that come before them
            const int before = p.causal ? min(max(t0 + key - lim0, 0), p.q_len) : 0;
            const unsigned hide = t0 + key >= t_end ? 0xffffffffu : ctrl->hidden[share][before];
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (hide >> i & 1u) v[i] = 0xff800000u;
          }
        };
        float top;       // the largest exponential
        auto exponentials = [&]() {
          top = 0.f;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (c >= my_chunks) continue;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const float4 neg = *reinterpret_cast<const float4*>(my_ref + c * 8 + i * 4);
              uint32_t* x = v + c * 8 + i * 4;
              float a, b, d, e;
              unpack_f2(fma_f2(pack_f2(__uint_as_float(x[0]), __uint_as_float(x[1])), sl2_2, pack_f2(neg.x, neg.y)), a, b);
              unpack_f2(fma_f2(pack_f2(__uint_as_float(x[2]), __uint_as_float(x[3])), sl2_2, pack_f2(neg.z, neg.w)), d, e);
              a = fast_exp2(a); b = fast_exp2(b); d = fast_exp2(d); e = fast_exp2(e);
              top = max3(top, a, b);
              top = max3(top, d, e);
              x[0] = __float_as_uint(a); x[1] = __float_as_uint(b); x[2] = __float_as_uint(d); x[3] = __float_as_uint(e);
            }
          }
        };
        load_scores();
        bool move = unset;
        if (!move) {
          exponentials();
          move = named_bar_any(bar_id, 128, !fine || !(top <= kKrMaxWeight));
          if (move) load_scores();
        }
        if (move) {
          // a reference that moves (or is set: the unit's first tile)
          float (*const peak)[kKrShareCols] = ctrl->peak[g & 1][share];
          float m[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) m[i] = __uint_as_float(v[i]);
          peak[quad][col] = column_reduce(m, lane, [](float a, float b) { return fmaxf(a, b); });
          lost = named_bar_any(bar_id, 128, !fine);
          if (lost) break;
          const float mx = fmaxf(fmaxf(peak[0][col], peak[1][col]), fmaxf(peak[2][col], peak[3][col])) * sl2;
          const bool real = col < my_chunks * 8 && col0 + col < R;
          const bool need = real && (mx - m_col) > kMoveThreshold;        // (false for NaN / (-inf)-(-inf))
          float alpha = 1.f;
          if (need) { alpha = fast_exp2(m_col - mx); m_col = mx; }
          __syncwarp();
          my_ref[col] = !real ? -INFINITY : m_col == -INFINITY ? 0.f : -m_col;       // (columns beyond the rows weigh nothing)
          my_scale[col] = alpha;
          __syncwarp();
          unset = __any_sync(0xffffffffu, real && m_col == -INFINITY);
          if (tile > 0 && __any_sync(0xffffffffu, need)) {
            fine = product_done(g - 1) && fine;
            tc_fence_after();
            const uint32_t tO = tmem + kOCol + (r & 1) * kKrMaxRows + lane_off + col0;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              if (c >= my_chunks) continue;
              uint32_t ov[8];
              tmem_ld8(tO + c * 8, ov);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 8; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * my_scale[c * 8 + i]);
              tmem_st8(tO + c * 8, ov);
#pragma unroll
              for (int i = 0; i < 4; ++i) sums[c * 4 + i] = mul_f2(sums[c * 4 + i], pack_f2(my_scale[c * 8 + 2 * i], my_scale[c * 8 + 2 * i + 1]));
            }
            tmem_wait_st();
          }
          exponentials();
        }
        // P goes where the tile before had it, when its product is done
        if (g > 0) fine = product_done(g - 1) && fine;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (c >= my_chunks) continue;
          const uint32_t* x = v + c * 8;
          uint32_t pk[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) pk[i] = ElemTraits<T>::pack2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1]));
          const uint32_t to = p_row + (((col0 >> 3) + c) ^ (key & 7)) * 16;
          asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(to), "r"(pk[0]), "r"(pk[1]), "r"(pk[2]), "r"(pk[3]) : "memory");
        }
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->p_ready));
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (c >= my_chunks) continue;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            sums[c * 4 + i] = add_f2(sums[c * 4 + i], pack_f2(__uint_as_float(v[c * 8 + 2 * i]), __uint_as_float(v[c * 8 + 2 * i + 1])));
        }
      }
      if (lost) { fine = false; break; }
      // sums over the quadrant's keys: lane l ends up with those of column l
      float f[16];
#pragma unroll
      for (int i = 0; i < 8; ++i) unpack_f2(sums[i], f[2 * i], f[2 * i + 1]);
      const float total = column_reduce(f, lane, [](float a, float b) { return a + b; });
      if (r >= 2) fine = mbar_wait(smem_u32(&ctrl->o_free[r & 1]), ((r >> 1) - 1) & 1) && fine;
      if (col < my_chunks * 8) {
        ctrl->sums[r & 1][quad][col0 + col] = total;
        if (quad == 0) ctrl->refs[r & 1][col0 + col] = m_col;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->l_ready[r & 1]));
      unit_done(r);
    }
    if (!__all_sync(0xffffffffu, fine) && lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; atomicMin(&ctrl->abort_round, 0); }
  } else if (warp < kKrOutWarp + 4) {
    // =========================== output warps: thread = element of the rows ===========================
    const int quad = warp - kKrOutWarp, d = quad * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    float* const inv = ctrl->inv[quad];
    bool ok = true;
    int r = 0, merges = 0;
    for (; ok; ++r) {
      const int u = unit_at(r);
      if (u < 0) { ok = false; break; }
      if (u >= n_units) break;
      const UmmaUnit w = ctrl->unit[r % kUmmaUnitRing];
      const bool has = tiles_of(w) > 0, single = w.n_chunks == 1;
      ok = warp_wait(smem_u32(&ctrl->l_ready[r & 1]), (r >> 1) & 1) && !*abort_flag;
      if (!ok) break;
      const long long slot = (static_cast<long long>(w.item0) + w.c) * p.kv_heads + w.h;
      for (int col = lane; col < R; col += 32) {
        const float (&s)[4][kKrMaxRows] = ctrl->sums[r & 1];
        const float l = (s[0][col] + s[1][col]) + (s[2][col] + s[3][col]);
        if (single) inv[col] = l > 0.f ? 1.f / l : 0.f;
        else if (quad == 0)
          *reinterpret_cast<float2*>(p.part_ml + (slot * R + col) * 2) = make_float2(ctrl->refs[r & 1][col], l);
      }
      __syncwarp();
      ok = warp_wait(smem_u32(&ctrl->o_done[r & 1]), (r >> 1) & 1) && !*abort_flag;
      if (!ok) break;
      tc_fence_after();
      const long long row0 = rows_of(w);
      if (d < D) {
        const uint32_t tO = tmem + kOCol + (r & 1) * kKrMaxRows + lane_off;
        auto write = [&](auto* to, auto convert) {
          for (int c = 0; c < R; c += 16, to += 16 * D) {
            uint32_t ov[16];
            float4 by[4];
            if (has) {
              tmem_ld16(tO + c, ov);
              tmem_wait_ld_regs(ov);
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) ov[i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) by[i] = *reinterpret_cast<const float4*>(inv + c + 4 * i);
            const float* const scale = &by[0].x;
            if (c + 16 <= R) {
#pragma unroll
              for (int i = 0; i < 16; ++i) to[i * D] = convert(__uint_as_float(ov[i]), scale[i]);
            } else {
#pragma unroll
              for (int i = 0; i < 15; ++i)
                if (c + i < R) to[i * D] = convert(__uint_as_float(ov[i]), scale[i]);
            }
          }
        };
        if (single) write(static_cast<OutT*>(p.out) + row0 * D + d, [](float x, float scale) { return ElemTraits<OutT>::from_float(x * scale); });
        else write(p.part_o + slot * R * D + d, [](float x, float) { return x; });
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->o_free[r & 1]));
      if (!single) {
        // Publish the partial; merges are claimed in the teardown.
        __threadfence();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->rows_out));
        // (all four warps: one that went on could arrive for its next unit in the place of one that still writes this unit's rows.  The
        // accumulator and the sums are given back already, so nothing but these warps waits)
        ok = warp_wait(smem_u32(&ctrl->rows_out), merges & 1) && !*abort_flag;
        if (!ok) break;
        if (quad == 0 && lane == 0) {
          __threadfence();
          atomicAdd(p.counters + w.b * p.kv_heads + w.h, 1);
          atomicAdd(p.header + 3, 1);              // tickets drawn and not merged yet (a hint for the teardown)
        }
        ++merges;
      }
      unit_done(r);
    }
    if (!ok) {
      atomicMin(&ctrl->abort_round, r);
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
    }
  }
  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == kKrMmaWarp) { tc_fence_after(); tmem_dealloc(tmem, 256); }
  claim_merges<OutT, D>(p, ctrl, me);
  if (ctrl->abort_flag) poison_units<OutT, D>(p, ctrl, n_units, [&](int r) { return ctrl->unit[r % kUmmaUnitRing]; });
}
