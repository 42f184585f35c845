// LUT GEMM for batches of 9 to a few hundred rows (batched decode, short prompts) on tcgen05.
//
// Such a launch is a stream of codes with little arithmetic per code: at 64 rows a 128 x 64 chunk of
// 4-bit codes (4 KB of HBM, 177 cycles of an SM's share; 128 wavefronts of lookups) feeds four MMAs of
// 128 x 64 x 16, and these bound it: an MMA with its A operand in tensor memory takes about 60 cycles
// whatever its width up to 128 columns (238 cycles per chunk at 16 to 64 tokens, 257 at 128, measured alone),
// and the kernel takes 257 at 64 tokens. The whole-tile kernel of gemm_tc.cu took 680 to 790 cycles per
// chunk here: eight lookup warps, each of them a serial chain of about 1450 cycles per chunk
// (measured with the SM clock: 500 waiting for its own code load, 390 looking up and storing, 150 for
// the next load and its cursor, the rest barriers), one tile per SM whatever the tile count.
//
// What is different here:
//  * Codes arrive by bulk copies (one contiguous chunk each) into a deep ring of shared memory that a
//    producer warp fills ahead, before it needs anything of the previous kernel; a lookup warp's chain
//    is barrier, two 16-byte reads, 32 lookups, two tensor-memory stores.
//  * Sixteen lookup warps: four row quarters x four stages of two chunks in flight.
//  * A tile is cut along K over a thread-block cluster; the CTAs exchange their sums through
//    distributed shared memory (each finishes a share of the tokens, adding the parts in ascending-k
//    order), so a 4096-row projection fills the GPU without a workspace, and tiles that do not divide
//    by the SM count cost less.
//  * Two accumulator halves, and eight epilogue warps of their own: a tile's exchange and stores run under
//    the next tile's MMAs.
//  * Sums in chains: the tensor core truncates where it adds to its fp32 accumulator, so a sum's error
//    grows with the number of MMAs behind one another (share of fp16 results that are not the rounding of
//    the 64-bit sum, K = 4096: 1.72e-2 for one chain, 0.95e-2 for two, 0.52e-2 for four). A tile's
//    k-blocks therefore go to several accumulators one after the other, which the epilogue adds in fp32,
//    ascending: as many as keep every chain as short as in the kernel that would serve the launch
//    otherwise (`chain_limit`: the tile kernel's warps at up to 16 rows, the cut tiles of gemm_tc.cu
//    above). Where they do not fit into half of the columns, a tile takes both halves and the next tile's
//    MMAs start when they have been read.
// Weights are the A operand in tensor memory, tokens (up to 128 per tile) the B operand in shared
// memory, as in gemm_tc.cu. All waits are bounded, and a wait that depends on the activations starts after
// the previous kernel has ended (an exchange may keep that one waiting for a peer for up to a second): the
// lookup warps' second stage, the code producer's second round of its ring, the MMA issuer.
//
// The gated form (kModeGated, up to 16 tokens): a cluster takes a row tile of gate and then the same row
// tile of up, and an epilogue thread, which finishes the same eight outputs of both, holds the finished
// gate values in registers: silu(gate) * up stays fp32 until its one rounding, as in the decode kernels.
//
// Warps: 0-15 lookup (row quarter = warp % 4; every fourth stage of two chunks belongs to group warp / 4),
// 16 code producer, 17 activation producer, 18 MMA issuer, 19-26 epilogue.
#include <cstdlib>
#include <mutex>

#include "gemm_parts.cuh"

namespace b200lut {

__device__ int g_cluster_status = 0;

int gemm_cluster_status_take() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_cluster_status, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(g_cluster_status, &zero, sizeof(int));
  return v;
}

namespace {

constexpr int kCLookupWarps = 16;
constexpr int kCGroups = 4;
constexpr int kCCodeWarp = kCLookupWarps, kCXWarp = kCLookupWarps + 1, kCMmaWarp = kCLookupWarps + 2,
              kCEpiWarp = kCLookupWarps + 3;
constexpr int kCEpiWarps = 8;
constexpr int kCThreads = (kCEpiWarp + kCEpiWarps) * 32;
constexpr int kCMaxNT = 128;
constexpr int kCMaxSplit = 8;
constexpr int kCStages = 4;               // operand stages in tensor memory, two k-blocks (64 columns) each
constexpr uint32_t kCTmemCols = 512;
constexpr uint32_t kCACol = 256;          // behind two accumulators of up to 128 columns
constexpr int kCMaxXSlots = 4;            // activation slots of two k-blocks
constexpr int kCMinCodeSlots = kCGroups, kCMaxCodeSlots = 8;    // code slots of two chunks
constexpr uint32_t kCTableAbs = 2048;     // pair table: offset inside the CTA's shared window
constexpr uint32_t kCWindowMask = 0x3FFFFu;
constexpr uint32_t kCDynBytes = 231424;   // dynamic shared memory per CTA
constexpr uint32_t kCWindowEnd = 1024 + kCDynBytes;

struct ClusterParams {
  // what every role reads first, close together: a launch's parameters start out in no cache
  int split, clusters, tiles_each, tiles_more;   // CTAs per cluster; clusters; whole share of tiles (gated form:
                                                 // pairs of tiles), clusters with one more
  int kb_each, kb_more;                          // k-blocks per CTA of a cluster, CTAs (the first ones) with one more
  int quads_each, quads_more;                    // token quads that a CTA finishes, likewise
  int NT, m_tiles, G, gs, M, nx, nc;             // tokens per tile, token tiles, ..., activation slots, code slots
  int chain, halves;                             // k-blocks per accumulator (1 or even); 2: tiles alternate between the halves
  uint32_t slot_bytes, x_off, c_off, e_off, s_off;   // offsets inside the shared window
  uint32_t e_quad, e_rows8;                          // exchange slots: bytes from quad to quad, from eight rows to the next eight
  int nsegs;
  long long wait_cycles;
  PersistSeg seg[kPMaxSeg];
  float* acc_out;              // first stream of two: fp32 sums instead of outputs
  const float* acc_in;         // second stream: sums to add
  long long ld_acc;
};

// Keeps a value in a register: without it the compiler reads launch parameters back from the constant
// bank (indexed, for a projection of a merged launch) at every use inside the loops.
__device__ __forceinline__ void pin(int& v) { asm volatile("" : "+r"(v)); }
__device__ __forceinline__ void pin(uint32_t& v) { asm volatile("" : "+r"(v)); }
__device__ __forceinline__ void pin(long long& v) { asm volatile("" : "+l"(v)); }
template <typename P>
__device__ __forceinline__ void pin(P*& v) { asm volatile("" : "+l"(v)); }

// Pair-table lookup: the table's place in the window is the immediate.
__device__ __forceinline__ uint32_t lds32_table(uint32_t addr) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1+2048];" : "=r"(v) : "r"(addr));
  return v;
}
static_assert(kCTableAbs == 2048, "the immediate in lds32_table is the table's offset");

__device__ __forceinline__ uint4 lds128v(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// 16 bytes into another CTA's shared memory, reported to that CTA's barrier `bar` when they are there
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t bar, const uint32_t (&v)[4]) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];" ::"r"(addr),
               "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}

// The 2 * BITS words of a lane's string that hold row slabs 2q and 2q + 1 of the chunk at `slot`.
// A lane's 32 bytes of a plane are two 16-byte halves; lanes 4..7 of every eight read the other half
// first, so that the eight lanes of a wavefront cover 128 distinct bytes.
template <int BITS>
__device__ __forceinline__ void load_codes(uint32_t (&w)[2 * BITS], uint32_t slot, int q, int lane) {
  const uint32_t a = slot + lane * 32;
  if constexpr (BITS >= 3) {
    const uint32_t first = 2 * BITS * q / 4;                  // 16-byte piece: plane first / 2, half first % 2
    const uint32_t p0 = a + (first >> 1) * 1024 + (first & 1) * 16;
    const uint32_t p1 = a + ((first + 1) >> 1) * 1024 + ((first + 1) & 1) * 16;
    const bool swap = (lane >> 2) & 1;
    const uint4 u = lds128v(swap ? p1 : p0), v = lds128v(swap ? p0 : p1);
    const uint4 lo = swap ? v : u, hi = swap ? u : v;
    const uint32_t all[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    if constexpr (BITS == 4) {
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = all[i];
    } else {
#pragma unroll
      for (int i = 0; i < 6; ++i) w[i] = (q & 1) ? all[i + 2] : all[i];
    }
  } else if constexpr (BITS == 2) {
    const uint4 u = lds128v(a + (q >> 1) * 1024 + (q & 1) * 16);
    w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w;
  } else {
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(a + q * 8));
  }
}


constexpr int kModePlain = 0, kModeResidual = 1, kModeGated = 2;
constexpr int kCGatedMaxNT = 16;          // one piece of eight outputs per epilogue thread and tile

template <typename T, int BITS, int MODE>
__global__ void __launch_bounds__(kCThreads, 1)
gemm_tc_persistent_kernel_clusters(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap tmap,
                                   const ClusterParams p) {
  constexpr bool RES = MODE == kModeResidual, GATED = MODE == kModeGated;
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t low = smem_u32(smem) & kCWindowMask, win = smem_u32(smem) - low;
  const uint32_t ctrl = win + 1024;
  // barriers: operand stage full / done (4 + 4), code slot full / empty (8 + 8), accumulator full / read
  // (2 + 2), exchange full / free
  const uint32_t bar_full = ctrl, bar_done = ctrl + 32, bar_cfull = ctrl + 64, bar_cempty = ctrl + 128,
                 bar_dfull = ctrl + 192, bar_dempty = ctrl + 208, bar_efull = ctrl + 224, bar_efree = ctrl + 232;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + (1024 + 256 - low));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + (1024 + 260 - low));
  uint8_t* tbl_ptr = smem + (kCTableAbs - low);

  const int S = p.split;
  const int rank = S > 1 ? int(tc::cluster_ctarank()) : 0;
  const int cid = S > 1 ? int(tc::cluster_id()) : int(blockIdx.x);
  const int c0 = rank * p.kb_each + (rank < p.kb_more ? rank : p.kb_more);     // this CTA's k-blocks of every tile:
  const int len = p.kb_each + (rank < p.kb_more ? 1 : 0);
  const int lenc = !RES || c0 + len <= p.G ? len : (p.G > c0 ? p.G - c0 : 0);  // with codes,
  const int lenr = len - lenc;                                                 // and the residual's, which close the tile
  const int pc = (lenc + 1) & ~1, lp = pc + ((lenr + 1) & ~1);                 // both start a stage of their own
  constexpr int kUnit = GATED ? 2 : 1;             // tiles of a unit of the schedule
  const int t0 = kUnit * (cid * p.tiles_each + (cid < p.tiles_more ? cid : p.tiles_more));
  // Never seen: the layout starts at the window's first dynamic byte. Such a CTA does no work.
  const bool bad_window = low != 1024;
  const int ntile = bad_window ? 0 : kUnit * (p.tiles_each + (cid < p.tiles_more ? 1 : 0));
  const long long lim = p.wait_cycles;
  int nl = kTileRows / p.gs;
  if (nl < 1) nl = 1;
  // the gated form has one token tile, and tiles 2r and 2r + 1 are row tile r of gate and of up
  auto row_of = [&](int tile) {
    if constexpr (GATED) return (tile & 1 ? p.seg[1].row0 : 0) + (tile >> 1);
    else return p.m_tiles == 1 ? tile : tile / p.m_tiles;
  };
  auto tok_of = [&](int tile) { return GATED || p.m_tiles == 1 ? 0 : (tile % p.m_tiles) * p.NT; };

  asm volatile("griddepcontrol.launch_dependents;");
  // The code producer sets up its own barriers and does not wait for the block: its first copies are
  // under way while the others meet.
  uint32_t first_palette = 0;      // the first tile's palette entry of this lane: requested before the barriers are met
  if (warp == kCCodeWarp) {
    if (lane < 16) tc::mbar_init(bar_cfull + 8 * lane, lane < 8 ? 1u : 4u);    // this warp (and its bytes) / four lookup warps
    if (lane == 0) {
      *abort_flag = bad_window ? 1 : 0;
      if (bad_window) atomicCAS(&g_cluster_status, tc::kStatusOk, tc::kStatusWaitLoad);
    }
    tc::mbar_init_fence();
    __syncwarp();
  } else if (warp == kCXWarp) {
    // full x 4 (four lookup warps + this warp and its bytes), done x 4 (commit), accumulator full x 2 (commit)
    // / read x 2, exchange full (this CTA's own expectation and the bytes) / free
    if (lane < 8) tc::mbar_init(bar_full + 8 * lane, lane < 4 ? 5u : 1u);
    else if (lane < 14)
      tc::mbar_init(bar_dfull + 8 * (lane - 8), lane < 10 ? 1u
                                                : lane < 12 ? uint32_t(kCEpiWarps)
                                                : lane < 13 ? 1u
                                                            : uint32_t((S > 1 ? S - 1 : 1) * kCEpiWarps));
    tc::mbar_init_fence();
    if (lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
  } else if (warp == kCMmaWarp) {
    tc::tmem_alloc(ctrl + 256, kCTmemCols);
  } else if (warp < kCLookupWarps && ntile > 0) {
    const int row = row_of(t0);
    const PersistSeg sd = segment_of_row(p, row);
    first_palette = palette_fetch(sd.lut, BITS, sd.n_groups, (row - sd.row0) * kTileRows, p.gs, nl);
  }
  tc::fence_before_sync();
  if (S > 1) {
    tc::cluster_arrive();                        // every CTA's barriers exist before anyone signals across
    if (warp != kCCodeWarp) tc::cluster_wait();
  } else if (warp == kCCodeWarp) {
    asm volatile("bar.arrive 2, %0;" ::"n"(kCThreads) : "memory");
  } else {
    asm volatile("bar.sync 2, %0;" ::"n"(kCThreads) : "memory");
  }
  tc::fence_after_sync();
  const uint32_t tmem = warp == kCCodeWarp ? 0u : *tmem_slot;

  if (warp < kCLookupWarps) {
    // ---- lookup: codes -> palette pairs -> tensor memory -------------------------------------------
    // A warp serves its 32 rows of every fourth stage, so its operand stage never changes.
    const int q = warp & 3, grp = warp >> 2;
    const int sp = lp >> 1;                        // stages per tile
    int table_row = -1, slot = grp, nc = p.nc;
    uint32_t cphase = 0, slot_bytes = p.slot_bytes, codes = win + p.c_off, dphase = 1;
    int st = grp;                                  // this warp's next stage, counted from the start
    pin(nc); pin(slot_bytes); pin(codes);
    const uint32_t dst = tmem + (uint32_t(32 * q) << 16) + kCACol + 64u * uint32_t(grp);
    for (int t = 0; t < ntile; ++t) {
      const int row = row_of(t0 + t);
      if (row != table_row) {
        uint32_t lv = first_palette;
        if (t > 0) {
          const PersistSeg sd = segment_of_row(p, row);
          lv = palette_fetch(sd.lut, BITS, sd.n_groups, (row - sd.row0) * kTileRows, p.gs, nl);
        }
        if (table_row >= 0) asm volatile("bar.sync 1, %0;" ::"n"(kCLookupWarps * 32) : "memory");
        table_store_shfl<kCLookupWarps * 32>(tbl_ptr, lv, BITS, nl);
        asm volatile("bar.sync 1, %0;" ::"n"(kCLookupWarps * 32) : "memory");
        table_row = row;
      }
      uint32_t token;                              // defined after the table's barrier; part of every address
      asm volatile("mov.u32 %0, 0;" : "=r"(token));
      const uint32_t base = (win + lane * 4 + (nl == 2 && q >= 2 ? 128u : 0u)) + token;
      for (; st < (t + 1) * sp; st += kCGroups) {
        const int j = 2 * (st - t * sp);           // the stage's first k-block of the tile
        const bool coded = !RES || j < lenc;
        uint32_t w[2][2 * BITS];
        tc::mbar_wait(bar_cfull + 8 * slot, cphase, abort_flag, &g_cluster_status, tc::kStatusWaitLoad, lim);
        if (coded) {                               // an odd last k-block: the second read returns what the slot held before
          load_codes<BITS>(w[0], codes + uint32_t(slot) * slot_bytes, q, lane);
          load_codes<BITS>(w[1], codes + uint32_t(slot) * slot_bytes + 1024 * BITS, q, lane);
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar_cempty + 8 * slot);
        slot += kCGroups;
        if (slot >= nc) { slot -= nc; cphase ^= 1u; }
        if (st == grp + kCGroups) asm volatile("griddepcontrol.wait;" ::: "memory");   // the first wait for an MMA
        tc::mbar_wait(bar_done + 8 * grp, dphase, abort_flag, &g_cluster_status, tc::kStatusWaitEmpty, lim);
        dphase ^= 1u;
        tc::fence_after_sync();
        if (coded) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
#pragma unroll
            for (int sl = 0; sl < 2; ++sl) {
              uint32_t r[16];
#pragma unroll
              for (int kt = 0; kt < 4; ++kt) {     // fields 0, 2, 1, 3: the store's register order
                r[4 * kt + 0] = lds32_table(slab_field_addr<BITS>(w[k], sl, 4 * kt + 0, base));
                r[4 * kt + 1] = lds32_table(slab_field_addr<BITS>(w[k], sl, 4 * kt + 2, base));
                r[4 * kt + 2] = lds32_table(slab_field_addr<BITS>(w[k], sl, 4 * kt + 1, base));
                r[4 * kt + 3] = lds32_table(slab_field_addr<BITS>(w[k], sl, 4 * kt + 3, base));
              }
              tc::tmem_st_16x256b_x4(dst + (uint32_t(16 * sl) << 16) + 32u * k, r);
            }
          }
        } else {
          // 128 columns of the tile's resA rows as they are (the store's register order, see gemm_tc.cu)
          const PersistSeg sd = segment_of_row(p, row);
#pragma unroll 1
          for (int k = 0; k < 2; ++k) {
            const int kk = (c0 + lenc + j - pc + k - p.G) * kChunkK + 4 * (lane & 3);
#pragma unroll 1
            for (int sl = 0; sl < 2; ++sl) {
              const int n = (row - sd.row0) * kTileRows + 32 * q + 16 * sl + (lane >> 2);
              const uint16_t* ra = sd.resA + size_t(n) * sd.res_rank + kk;
              const uint16_t* rb = ra + size_t(8) * sd.res_rank;
              uint32_t r[16];
#pragma unroll
              for (int kt = 0; kt < 4; ++kt) {
                uint2 lo = make_uint2(0u, 0u), hi = make_uint2(0u, 0u);
                if (sd.resA != nullptr && kk + 16 * kt < sd.res_rank) {
                  lo = __ldg(reinterpret_cast<const uint2*>(ra + 16 * kt));
                  hi = __ldg(reinterpret_cast<const uint2*>(rb + 16 * kt));
                }
                r[4 * kt + 0] = lo.x; r[4 * kt + 1] = lo.y; r[4 * kt + 2] = hi.x; r[4 * kt + 3] = hi.y;
              }
              tc::tmem_st_16x256b_x4(dst + (uint32_t(16 * sl) << 16) + 32u * k, r);
            }
          }
        }
        tc::wait_st();
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar_full + 8 * grp);
      }
    }
  } else if (warp == kCCodeWarp) {
    // ---- codes: one bulk copy per stage, as far ahead as the ring reaches ------------------------------
    if (tc::elect_one()) {
      uint64_t policy;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
      int nc = p.nc, slot = 0;
      uint32_t phase = 1, slot_bytes = p.slot_bytes, codes = win + p.c_off;   // a new barrier's previous phase reads as done
      pin(nc); pin(slot_bytes); pin(codes);
      bool ok = true;
      for (int t = 0; t < ntile && ok; ++t) {
        const int row = row_of(t0 + t);
        const PersistSeg sd = segment_of_row(p, row);
        const uint8_t* src = sd.packed + (size_t(row - sd.row0) * p.G + c0) * (1024 * BITS);
        for (int left = lenc, j = 0; j < lp; j += 2, left -= 2, src += 2 * 1024 * BITS) {
          const uint32_t bar = bar_cfull + 8 * slot;
          ok = tc::mbar_wait(bar_cempty + 8 * slot, phase, abort_flag, &g_cluster_status, tc::kStatusWaitEmpty, lim);
          if (!ok) break;
          if (RES && left <= 0) {
            tc::mbar_arrive(bar);                                  // nothing but residual k-blocks
          } else {
            const uint32_t bytes = uint32_t(left < 2 ? left : 2) * (1024 * BITS);
            tc::mbar_expect_tx(bar, bytes);
            bulk_load(codes + uint32_t(slot) * slot_bytes, src, bytes, bar, policy);
          }
          if (++slot == nc) {
            if (phase) asm volatile("griddepcontrol.wait;" ::: "memory");   // from here on slots come back from the lookups
            slot = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
    if (S > 1) tc::cluster_wait();               // of the start
  } else if (warp == kCXWarp) {
    // ---- activations: one load per operand stage (two k-blocks) ----------------------------------------
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (tc::elect_one()) {
      uint32_t bytes = uint32_t(p.NT) * 256u, dst0 = win + p.x_off;
      int nx = p.nx, slot = 0, st = 0;
      pin(bytes); pin(dst0); pin(nx);
      bool ok = true;
      for (int t = 0; t < ntile && ok; ++t) {
        const int m0 = tok_of(t0 + t);
        const int tblk = RES ? segment_of_row(p, row_of(t0 + t)).t_col0 / kChunkK + c0 + lenc - p.G : 0;
        for (int j = 0; j < lp; j += 2, ++st) {
          const int prev = st - nx;                                // the stage that used this slot before
          if (prev >= 0)
            ok = tc::mbar_wait(bar_done + 8 * (prev & (kCStages - 1)), uint32_t(prev / kCStages) & 1u, abort_flag,
                               &g_cluster_status, tc::kStatusWaitEmpty, lim);
          if (!ok) break;
          const uint32_t bar = bar_full + 8 * (st & (kCStages - 1));
          tc::mbar_expect_tx(bar, bytes);
          if (!RES || j < lenc) tma_load_3d(dst0 + uint32_t(slot) * bytes, &xmap, bar, 0, m0, c0 + j);
          else tma_load_3d(dst0 + uint32_t(slot) * bytes, &tmap, bar, 0, m0, tblk + j - pc);
          if (++slot == nx) slot = 0;
        }
      }
    }
    __syncwarp();
  } else if (warp == kCMmaWarp) {
    // ---- MMA issuer: a short loop, eight MMAs and one commit per stage ------------------------------------
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (tc::elect_one()) {
      constexpr uint32_t kFmt = DType<T>::id == B200LUT_BF16 ? 1u : 0u;
      const uint32_t idesc = tc::instr_desc(kFmt, 128, uint32_t(p.NT));
      const uint64_t dt = tc::smem_desc(0u, 16u, 1024u, 2u);
      const uint32_t xhi = uint32_t(dt >> 32), x0 = uint32_t(dt) + ((win + p.x_off) >> 4);
      uint32_t half = uint32_t(p.NT) * 8u;                  // one k-block of activations in descriptor units
      int nx = p.nx, slot = 0;
      pin(half); pin(nx);
      const int alt = p.halves - 1;                         // 1: tile t in half t & 1
      uint32_t st = 0, xlo = x0;
      // A chain's first k-block overwrites its accumulator. Chains are whole stages, or single k-blocks: then
      // the stage's second one has the next accumulator. (Loop-invariant values and a count: with the chains
      // in a loop of their own 12288 x 4096, 3 bits, 16 rows took 13.0 instead of 12.4 us.)
      const bool one = p.chain == 1;
      const uint32_t next = half >> 3, next_half = one ? next : 0u, add_half = one ? 0u : 1u, jump = next + next_half;
      for (int t = 0; t < ntile; ++t) {
        const int buf = t & alt;
        if (t > alt)                   // the half's last tile must have been read
          tc::mbar_wait(bar_dempty + 8 * buf, uint32_t((t >> alt) - 1) & 1u, abort_flag, &g_cluster_status,
                        tc::kStatusWaitDone, lim);
        uint32_t acc = tmem + uint32_t(buf * kCMaxNT), add = 0u;
        int left = p.chain;
        for (int j = 0; j < lp; j += 2, ++st) {
          const uint32_t u = st & (kCStages - 1);
          const bool second = !RES || j < pc ? j + 1 < lenc : j - pc + 1 < lenr;
          tc::mbar_wait(bar_full + 8 * u, (st / kCStages) & 1u, abort_flag, &g_cluster_status, tc::kStatusWaitFull, lim);
          tc::fence_after_sync();
          tc::mma_ts_kblock(acc, tmem + kCACol + 64u * u, xlo, xhi, idesc, add);
          if (second) tc::mma_ts_kblock(acc + next_half, tmem + kCACol + 64u * u + 32u, xlo + half, xhi, idesc, add_half);
          tc::mma_commit(bar_done + 8 * u);
          add = 1u;
          if ((left -= 2) <= 0) { left = p.chain; acc += jump; add = 0u; }
          xlo += 2 * half;
          if (++slot == nx) { slot = 0; xlo = x0; }
        }
        tc::mma_commit(bar_dfull + 8 * buf);
      }
    }
    __syncwarp();
  } else {
    // ---- epilogue: tensor memory (+ the cluster's other parts) -> bias -> one rounding -> global --------
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int q = warp & 3, h = (warp - kCEpiWarp) >> 2, row_in = 32 * q + lane;   // lane quarter, half of the columns
    // Token quads (four columns): CTA r of the cluster finishes quads [first(r), first(r + 1)).
    auto first = [&](int r) { return r * p.quads_each + (r < p.quads_more ? r : p.quads_more); };
    const int mine0 = first(rank), mine1 = first(rank + 1);
    // Has this warp quads of its half to send? Where no other CTA's share is wider than two quads, the warps of
    // the second half have none, and nobody waits for them: the exchange may be a tile or two ahead of them.
    const bool sends = p.quads_each + (p.quads_more > (rank < p.quads_more ? 1 : 0) ? 1 : 0) > 2 * h;
    uint32_t e_quad = p.e_quad;
    pin(e_quad);
    const uint32_t slot_stride = uint32_t(p.quads_each + (p.quads_more ? 1 : 0)) * e_quad;   // of the widest share
    const uint32_t exch = win + p.e_off + uint32_t(row_in >> 3) * p.e_rows8 + uint32_t(row_in & 7) * 16u;
    const uint32_t stage = win + p.s_off + uint32_t(warp - kCEpiWarp) * 512u;   // 8 tokens x 32 rows
    const int alt = p.halves - 1;
    // accumulators of this CTA's tiles (the residual's k-blocks start a stage of their own),
    int chains = (p.chain == 1 ? len : lp + p.chain - 1) / p.chain;
    const uint32_t chain_cols = uint32_t(p.NT);                    // and the columns from one to the next
    pin(chains);
    // Quads b and, with `both`, b + 1 of the accumulators at `acc`: their chains' sums, ascending in k.
    auto read_quads = [&](uint32_t acc, int b, bool both, uint32_t (&r)[2][4]) {
      const uint32_t a = acc + uint32_t(4 * b);
      tmem_ld_32x32b_x4(a, r[0]);
      if (both) tmem_ld_32x32b_x4(a + 4u, r[1]);
      tc::wait_ld();
#pragma unroll 1
      for (int i = 1; i < chains; ++i) {
        uint32_t u[2][4];
        tmem_ld_32x32b_x4(a + uint32_t(i) * chain_cols, u[0]);
        if (both) tmem_ld_32x32b_x4(a + uint32_t(i) * chain_cols + 4u, u[1]);
        tc::wait_ld();
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (e == 0 || both) r[e][j] = __float_as_uint(__uint_as_float(r[e][j]) + __uint_as_float(u[e][j]));
      }
    };
    float* acc_out = p.acc_out;
    const float* acc_in = p.acc_in;
    float gate[8];                                                 // gated form: what the last (gate) tile came to
    for (int t = 0; t < ntile; ++t) {
      const int row = row_of(t0 + t), m0 = tok_of(t0 + t);
      const PersistSeg sd = segment_of_row(p, row);
      const int n = (row - sd.row0) * kTileRows + 32 * q;          // first of the warp's 32 rows
      uint16_t* out = (GATED ? p.seg[0].out : sd.out) + n;
      long long ldo = GATED ? p.seg[0].ldo : sd.ldo;
      int M = p.M;
      pin(out); pin(ldo); pin(M);
      const bool vec = (GATED ? p.seg[0].out_aligned : sd.out_aligned) != 0;
      const float bias = sd.bias ? DType<T>::to_float(sd.bias[n + lane]) : 0.f;
      const int buf = t & alt;
      const uint32_t acc = tmem + (uint32_t(32 * q) << 16) + uint32_t(buf * kCMaxNT);
      auto release = [&]() {                                       // this warp has read the tile's accumulators
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar_dempty + 8 * buf);
      };
      if (S > 1 && warp == kCEpiWarp && lane == 0)                 // what the others will write here for this tile
        tc::mbar_expect_tx(bar_efull, uint32_t((S - 1) * (mine1 - mine0) * kTileRows) * 16u);
      tc::mbar_wait(bar_dfull + 8 * buf, uint32_t(t >> alt) & 1u, abort_flag, &g_cluster_status, tc::kStatusWaitDone, lim);
      tc::fence_after_sync();
      if (S > 1) {
        // The others have read this CTA's parts of the last tile. A warp that sends nothing overwrites nothing,
        // and must not wait here: the phase it asks for could be two back, which reads as not complete.
        // A warp that sends cannot miss one, as the next phase needs what it sends.
        if (t > 0 && sends)
          tc::mbar_wait_cluster(bar_efree, uint32_t(t - 1) & 1u, abort_flag, &g_cluster_status, tc::kStatusWaitDone, lim);
        for (int k = 1; k < S; ++k) {
          const int d = rank + k < S ? rank + k : rank + k - S;
          const int b0 = first(d), b1 = first(d + 1);
          const uint32_t bar = map_rank(bar_efull, uint32_t(d));
          // this CTA's slot among d's sources
          uint32_t dst = map_rank(exch, uint32_t(d)) + uint32_t(rank < d ? rank : rank - 1) * slot_stride +
                         uint32_t(2 * h) * e_quad;
          for (int b = b0 + 2 * h; b < b1; b += 4, dst += 4u * e_quad) {
            uint32_t r[2][4];
            read_quads(acc, b, b + 1 < b1, r);
            st_async_v4(dst, bar, r[0]);
            if (b + 1 < b1) st_async_v4(dst + e_quad, bar, r[1]);
          }
        }
        tc::mbar_wait_cluster(bar_efull, uint32_t(t) & 1u, abort_flag, &g_cluster_status, tc::kStatusWaitFull, lim);
      }
      if (mine0 + 2 * h >= mine1) release();
      for (int b = mine0 + 2 * h; b < mine1; b += 4) {             // 8 tokens of the warp's 32 rows at a time
        const bool both = b + 1 < mine1;
        uint32_t own[2][4];
        read_quads(acc, b, both, own);
        if (b + 4 >= mine1) release();
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = S == 1 ? __uint_as_float(own[j >> 2][j & 3]) : 0.f;
        if (S > 1) {
          uint32_t e = exch + uint32_t(b - mine0) * e_quad;
          for (int r = 0; r < S; ++r) {            // ascending k
            if (r == rank) {
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j] += __uint_as_float(own[j >> 2][j & 3]);
            } else {
              const uint4 a = lds128v(e);
              v[0] += __uint_as_float(a.x); v[1] += __uint_as_float(a.y);
              v[2] += __uint_as_float(a.z); v[3] += __uint_as_float(a.w);
              if (both) {
                const uint4 c = lds128v(e + e_quad);
                v[4] += __uint_as_float(c.x); v[5] += __uint_as_float(c.y);
                v[6] += __uint_as_float(c.z); v[7] += __uint_as_float(c.w);
              }
              e += slot_stride;
            }
          }
        }
        if constexpr (GATED) {
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] += bias;
          if ((t & 1) == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) gate[j] = v[j];
            continue;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = gate[j] / (1.f + __expf(-gate[j])) * v[j];
        }
        const int tok0 = m0 + 4 * b, most = both ? 8 : 4;
        const int ntok = M - tok0 < most ? M - tok0 : most;         // tokens of this piece that exist
        if (!GATED && acc_out) {                   // first stream of two: raw fp32 sums
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < ntok) __stcg(acc_out + (tok0 + j) * p.ld_acc + n + lane, v[j]);
          continue;
        }
        if (!GATED && acc_in) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < ntok) v[j] += __ldcg(acc_in + (tok0 + j) * p.ld_acc + n + lane);
        }
        if (vec) {
          // [token][32 rows] in the warp's staging slice, then 16 bytes per lane: eight tokens a store
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(stage + uint32_t(j * 64 + lane * 2)),
                         "h"(DType<T>::from_float(GATED ? v[j] : v[j] + bias))
                         : "memory");
          __syncwarp();
          const int j = lane >> 2;
          if (j < ntok) *reinterpret_cast<uint4*>(out + (tok0 + j) * ldo + 8 * (lane & 3)) = lds128v(stage + uint32_t(lane * 16));
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < ntok) out[(tok0 + j) * ldo + lane] = DType<T>::from_float(GATED ? v[j] : v[j] + bias);
        }
      }
      if (S > 1 && t + 1 < ntile) {
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        __syncwarp();
        if (lane < S && lane != rank) tc::mbar_arrive_cluster(map_rank(bar_efree, uint32_t(lane)));
      }
    }
  }
  // A wait has given up: copies into this CTA's memory, sums sent to other CTAs and MMAs may be under way with
  // nobody to wait for them. They take microseconds; every thread that ends its role after the flag was set
  // stays for 100000 cycles (50 us), so the CTA leaves, and frees its tensor memory, behind all of them.
  __syncwarp();
  if (__any_sync(0xffffffffu, *abort_flag != 0)) {
    const long long t0 = clock64();
    while (clock64() - t0 < 100000) { }
    __syncwarp();
  }
  tc::fence_before_sync();
  // A CTA must not leave while another's sums are on their way to it. It has waited for all of them —
  // unless a wait gave up, so the CTAs meet; by now every arrival of the others is near.
  if (S > 1) {
    tc::cluster_arrive();
    tc::cluster_wait();
  } else {
    __syncthreads();
  }
  if (warp == kCMmaWarp) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, kCTmemCols);
  }
}

// ---- host -------------------------------------------------------------------------------------------

struct ClusterPlan {
  int split, clusters, NT, m_tiles, tiles, nx, nc, chains, chain, halves;
  uint32_t slot_bytes, x_off, c_off, e_off, s_off, e_quad, e_rows8, smem_bytes;
};

// Shared memory of a launch; false when it does not fit: pair table, activation slots (1 KB-aligned),
// exchange slots, the epilogue's staging slices, code slots. One palette per tile (group_size >= 128)
// uses only one 128-byte half of every 256-byte entry of the table; at 4 bits the exchange goes into the
// other half when it fits (up to 16 quads), which leaves a 128-token tile a third activation slot.
bool cluster_layout(int bits, int group_size, ClusterPlan* c) {
  const int quads = c->NT / 4, widest = (quads + c->split - 1) / c->split;
  const int held = c->split > 1 ? (c->split - 1) * widest : 0;           // quads of other CTAs' sums
  const bool in_table = bits == 4 && group_size >= kTileRows && held <= 16;
  const uint32_t after_table = kCTableAbs + (256u << (2 * bits)), x_off = (after_table + 1023u) & ~1023u;
  const uint32_t exch = in_table ? 0u : uint32_t(held) * kTileRows * 16u;
  const uint32_t xslot = uint32_t(c->NT) * 256u, fixed = x_off + exch + kCEpiWarps * 512u;
  c->slot_bytes = 2 * 1024u * uint32_t(bits);
  // as many slots of each kind as fit, the longer latency (codes, from HBM) first
  c->nx = 2;
  c->nc = kCMinCodeSlots;
  auto fits = [&](int nx, int nc) { return fixed + uint32_t(nx) * xslot + uint32_t(nc) * c->slot_bytes <= kCWindowEnd; };
  if (!fits(c->nx, c->nc)) return false;
  for (bool more = true; more;) {
    more = false;
    if (c->nx < kCMaxXSlots && fits(c->nx + 1, c->nc)) { ++c->nx; more = true; }
    if (c->nc < kCMaxCodeSlots && fits(c->nx, c->nc + 1)) { ++c->nc; more = true; }
  }
  c->x_off = x_off;
  c->e_off = in_table ? kCTableAbs + 128u : c->x_off + uint32_t(c->nx) * xslot;
  c->e_quad = in_table ? kTileRows * 32u : kTileRows * 16u;
  c->e_rows8 = in_table ? 256u : 128u;
  c->s_off = c->x_off + uint32_t(c->nx) * xslot + exch;
  c->c_off = c->s_off + kCEpiWarps * 512u;
  c->smem_bytes = c->c_off + uint32_t(c->nc) * c->slot_bytes - 1024u;
  return true;
}

// The activation rows as [K / 64][M][64]: one load brings two k-blocks of a token tile.
int encode_x_map3(CUtensorMap* map, const void* x, int64_t ldx, int M, int K, int dtype, int NT) {
  EncodeTiledFn enc = encode_fn();
  B200LUT_REQUIRE(enc != nullptr, B200LUT_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[3] = {cuuint64_t(kChunkK), cuuint64_t(M), cuuint64_t(K / kChunkK)};
  const cuuint64_t strides[2] = {cuuint64_t(ldx) * 2, cuuint64_t(kChunkK) * 2};
  const cuuint32_t box[3] = {cuuint32_t(kChunkK), cuuint32_t(NT), 2};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, dtype == B200LUT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                         const_cast<void*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B200LUT_REQUIRE(r == CUDA_SUCCESS, B200LUT_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", int(r));
  return B200LUT_OK;
}

template <typename T, int BITS, int MODE>
int configure(int dev) {
  static bool done[64] = {false};
  if (dev < 64 && done[dev]) return B200LUT_OK;
  auto kern = gemm_tc_persistent_kernel_clusters<T, BITS, MODE>;
  B200LUT_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kCDynBytes)));
  if (dev < 64) done[dev] = true;
  return B200LUT_OK;
}

template <typename T, int BITS, int MODE>
int launch_cluster(const CUtensorMap& xmap, const CUtensorMap& tmap, const ClusterParams& p, uint32_t smem, bool pdl,
                   cudaStream_t stream) {
  int dev = 0;
  B200LUT_CUDA_OK(cudaGetDevice(&dev));
  if (int rc = configure<T, BITS, MODE>(dev)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(p.clusters * p.split), 1, 1);
  cfg.blockDim = dim3(kCThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (p.split > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = unsigned(p.split);
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = unsigned(na);
  auto kern = gemm_tc_persistent_kernel_clusters<T, BITS, MODE>;
  B200LUT_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, xmap, tmap, p));
  return B200LUT_OK;
}

// Clusters of `split` CTAs (one per SM) that can be resident at once, per device; measured once.
int max_clusters(int split) {
  static std::mutex mu;
  static int cache[64][kCMaxSplit + 1] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lock(mu);
  int& n = cache[dev][split];
  if (n) return n;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 0;
  if (split == 1) return n = sms;
  auto kern = gemm_tc_persistent_kernel_clusters<__nv_bfloat16, 4, kModePlain>;
  if (configure<__nv_bfloat16, 4, kModePlain>(dev) != B200LUT_OK) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(split), 1, 1);
  cfg.blockDim = dim3(kCThreads, 1, 1);
  cfg.dynamicSmemBytes = kCDynBytes;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(split);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int got = 0;
  if (cudaOccupancyMaxActiveClusters(&got, kern, &cfg) != cudaSuccess || got < 1) {
    (void)cudaGetLastError();
    got = -1;
  }
  return n = got;
}

// The cut of K that finishes first, by a fit (microseconds) to launches measured at 2048 to 24576 rows,
// K = 4096 and 12288, 24 to 1024 tokens, cuts of 1 to 8: a k-block of the busiest cluster, what a launch
// costs besides, what the exchange adds, and what is lost when the launch fills more than half of the
// SMs (below that, its start and end run beside its neighbours' in the stream). With K cut, a cluster's
// next tile cannot end before the exchange of the last one has made its way around (kExchange: 16 rows of
// 24576 x 4096, a gate/up pair, cuts of 1 / 2 / 3 / 8 over 2 / 4 / 4 to 6 / 12 tiles, 20.5 / 23.2 / 32.2 /
// 57.7 us): short parts of many tiles lose what the even split gains. With that term in the cost the pair
// takes 20.7 us instead of 30.9, 248320 x 4096 at 16 rows 126 instead of 144, and the Q/K/V launch of 333
// tokens and its residual 53 instead of 84. `unit` tiles go to a
// cluster together; c.tiles counts units. `chain_limit`: the most of the G k-blocks that one accumulator may
// take; a cut whose chains do not fit into the accumulators' columns is out. (The residual's `extra` k-blocks
// lengthen a chain, as they do in the kernel the limit comes from.)
bool plan_cluster(int M, int rows, int G, int extra, int bits, int group_size, bool whole_tiles, int unit, int chain_limit,
                  ClusterPlan* best) {
  const int Gx = G + extra;
  const int m_tiles = (M + kCMaxNT - 1) / kCMaxNT;
  const int per = (M + m_tiles - 1) / m_tiles, NT = (per + 15) / 16 * 16;
  const int sms = max_clusters(1);
  const double kblock = 0.112 + 4.7e-6 * NT * NT;
  double least = 0;
  bool found = false;
  constexpr double kExchange = 3.9, kDrain = 0.5;
  for (int s = 1; s <= (whole_tiles ? 1 : kCMaxSplit); ++s) {
    if (s > 1 && Gx < 4 * s) break;
    ClusterPlan c = {};
    c.split = s; c.NT = NT; c.m_tiles = m_tiles; c.tiles = rows * m_tiles / unit;
    // chains of whole stages (two k-blocks), or of single k-blocks; the residual's start a stage of their own
    const int len = (Gx + s - 1) / s, coded = (G + s - 1) / s;
    const int limit = chain_limit >= coded ? (coded + 1) & ~1 : chain_limit > 1 ? chain_limit & ~1 : 1;
    c.chains = limit == 1 ? len : (coded + limit - 1) / limit;
    c.chain = limit == 1 ? 1 : (((len + (extra ? 2 : 0) + c.chains - 1) / c.chains) + 1) & ~1;
    if (c.chains * NT > 2 * kCMaxNT) continue;
    c.halves = c.chains * NT > kCMaxNT ? 1 : 2;
    const int fit = max_clusters(s);
    if (fit < 1 || !cluster_layout(bits, group_size, &c)) continue;
    c.clusters = c.tiles < fit ? c.tiles : fit;
    const int rounds = unit * ((c.tiles + c.clusters - 1) / c.clusters);
    double crowd = (c.clusters * s - sms / 2) / (s > 1 ? 0.27 * sms : 0.5 * sms);
    crowd = crowd < 0 ? 0 : (crowd > 1 ? 1 : crowd);
    const double tile = double(len) * kblock, next = s > 1 && tile < kExchange ? kExchange : tile;
    const double cost = tile + (rounds - 1) * (next + (c.halves == 1 ? kDrain : 0.0)) + 3.2 +
                        (s > 1 ? 0.9 + 0.1 * s : 0.0) + 3.0 * crowd;
    if (!found || cost < least) { *best = c; least = cost; found = true; }
  }
  return found;
}

}  // namespace

long long gemm_wait_cycles() {
  const char* e = getenv("B200LUT_WAIT_MS");
  if (!e) return tc::kWaitCycles;
  const long ms = atol(e);
  return (ms < 1 ? 1 : ms > 1000 ? 1000 : ms) * 2000000ll;
}

bool cluster_gemm_serves(int M, int row_tiles, int K, int bits, int group_size, int chain_limit) {
  ClusterPlan c = {};
  return M >= 1 && group_size >= 64 && K >= 2 * kChunkK &&
         plan_cluster(M, row_tiles, K / kChunkK, 0, bits, group_size, false, 1, chain_limit, &c);
}

// `nseg` projections that share x (one code stream each, one code width and group size, at most two
// palettes per 128-row tile); whole_tiles: K is not cut; gated: the projections are (gate, up) of one
// size, at most 16 rows, and segs[0].out becomes silu(gate) * up. *served is false, and nothing has been launched, for other shapes.
int cluster_gemm(const void* x, int64_t ldx, int M, int K, int dtype, const b200lut_segment* segs, int nseg, bool pdl,
                 void* stream, float* acc_out, const float* acc_in, long long ld_acc, long long wait_cycles, bool whole_tiles, bool gated,
                 int chain_limit, bool* served) {
  *served = false;
  ClusterParams p = {};
  int rows = 0, extra = 0;
  const uint16_t* t_base = nullptr;
  long long t_ld = 0;
  for (int i = 0; i < nseg; ++i) {
    const b200lut_segment& s = segs[i];
    PersistSeg& d = p.seg[i];
    d.packed = static_cast<const uint8_t*>(s.packed);
    d.lut = static_cast<const uint16_t*>(s.lut);
    d.bias = static_cast<const uint16_t*>(s.bias);
    d.out = static_cast<uint16_t*>(s.out);
    d.ldo = s.ldo;
    d.out_aligned = (aligned16(s.out) && s.ldo % 8 == 0) ? 1 : 0;
    d.row0 = rows;
    d.n_groups = s.n_groups;
    rows += s.N / kTileRows;
    if (s.res_rank > 0) {
      if (!t_base) { t_base = static_cast<const uint16_t*>(s.res_t); t_ld = s.res_ldt; }
      d.resA = static_cast<const uint16_t*>(s.resA);
      d.res_rank = s.res_rank;
      const long long col0 = static_cast<const uint16_t*>(s.res_t) - t_base;
      const int blocks = (s.res_rank + kChunkK - 1) / kChunkK;
      // loads take whole 64-column blocks of one t matrix; what else there is, the general kernel takes or refuses
      if (s.res_ldt != t_ld || col0 < 0 || col0 % kChunkK || col0 + (long long)blocks * kChunkK > t_ld) return B200LUT_OK;
      d.t_col0 = int(col0);
      if (blocks > extra) extra = blocks;
    }
  }
  if (gated && (M > kCGatedMaxNT || nseg != 2 || segs[0].N != segs[1].N || extra || acc_out || acc_in)) return B200LUT_OK;
  p.nsegs = nseg;
  p.M = M; p.G = K / kChunkK; p.gs = segs[0].group_size;
  const int Gx = p.G + extra;
  ClusterPlan c = {};
  if (segs[0].group_size < 64 ||
      !plan_cluster(M, rows, p.G, extra, segs[0].bits, p.gs, whole_tiles, gated ? 2 : 1, whole_tiles ? p.G : chain_limit, &c))
    return B200LUT_OK;
  p.NT = c.NT; p.m_tiles = c.m_tiles; p.split = c.split; p.clusters = c.clusters;
  p.tiles_each = c.tiles / c.clusters; p.tiles_more = c.tiles % c.clusters;
  p.kb_each = Gx / c.split; p.kb_more = Gx % c.split;
  p.halves = c.halves; p.chain = c.chain;
  p.quads_each = c.NT / 4 / c.split; p.quads_more = c.NT / 4 % c.split;
  p.nx = c.nx; p.nc = c.nc; p.slot_bytes = c.slot_bytes;
  p.x_off = c.x_off; p.c_off = c.c_off; p.e_off = c.e_off; p.s_off = c.s_off; p.e_quad = c.e_quad; p.e_rows8 = c.e_rows8;
  p.wait_cycles = wait_cycles;
  p.acc_out = acc_out; p.acc_in = acc_in; p.ld_acc = ld_acc;
  CUtensorMap xmap, tmap;
  if (int rc = encode_x_map3(&xmap, x, ldx, M, K, dtype, p.NT)) return rc;
  if (extra) {
    if (int rc = encode_x_map3(&tmap, t_base, t_ld, M, int(t_ld), dtype, p.NT)) return rc;
  } else {
    tmap = xmap;
  }
  *served = true;
#define B200LUT_CLUSTER_AS(B, MODE)                                                                         \
  (dtype == B200LUT_BF16 ? launch_cluster<__nv_bfloat16, B, MODE>(xmap, tmap, p, c.smem_bytes, pdl, cudaStream_t(stream)) \
                         : launch_cluster<__half, B, MODE>(xmap, tmap, p, c.smem_bytes, pdl, cudaStream_t(stream)))
#define B200LUT_CLUSTER(B)                             \
  (extra   ? B200LUT_CLUSTER_AS(B, kModeResidual)      \
   : gated ? B200LUT_CLUSTER_AS(B, kModeGated)         \
           : B200LUT_CLUSTER_AS(B, kModePlain))
  switch (segs[0].bits) {
    case 4: return B200LUT_CLUSTER(4);
    case 3: return B200LUT_CLUSTER(3);
    case 2: return B200LUT_CLUSTER(2);
    default: return B200LUT_CLUSTER(1);
  }
#undef B200LUT_CLUSTER
#undef B200LUT_CLUSTER_AS
}

}  // namespace b200lut
