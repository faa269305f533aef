// Dense contraction kernel for sm_100a:  D[b, m, n] = epilogue( sum_k A[b, m, k] * B[b, n, k] )
//
// One persistent CTA per SM, warp specialised:
//   warp 0      TMA producer: cp.async.bulk.tensor loads of A and B tiles (128-byte swizzle)
//               into a B200_STAGES-deep shared-memory ring, completion on mbarriers
//   warp 1      owns tensor memory (tcgen05.alloc) and issues tcgen05.mma (kind::f16 or
//               kind::tf32, fp32 accumulators in TMEM); tcgen05.commit releases ring slots
//               and publishes finished accumulators
//   warps 2..   epilogue: tcgen05.ld of the accumulator (one TMEM lane = one output row per
//               thread), the routine's generated epilogue expression, global stores
// Two accumulator buffers in TMEM let the epilogue of tile i overlap the main loop of
// tile i+1.  Every wait is bounded: a wait that does not complete within ~2 s raises the
// device status word, all roles drain and the CTA frees its tensor memory and returns.
//
// The translation unit that includes this text defines:
//   B200_GEMM_NAME            kernel symbol
//   B200_BM (128), B200_BN    tile extents (B200_BN multiple of 16, <= 256)
//   B200_BK                   k elements per ring slot (128 bytes worth)
//   B200_UMMA_K               k elements per tcgen05.mma (16 for 16-bit inputs, 8 for tf32)
//   B200_ELEM_BYTES           operand element size
//   B200_STAGES               ring depth
//   B200_EPI_WARPS            4, 8 or 16 (a multiple of 4: one warp per TMEM lane quarter and column part)
//   B200_STAGING_BYTES        bytes of one staging tile (32 rows x chunk columns of the widest output)
//   B200_STAGING_TILES        staging tiles per epilogue warp (2 when outputs leave as TMA stores and shared memory allows)
//   B200_EPI_PROLOGUE         declarations at the top of the epilogue role (pointers to the output tensor maps)
//   B200_LOAD_TILE_BYTES      bytes of the per-warp tile that receives a row operand's chunk by TMA (0: none)
//   B200_A_KMAJOR/B_KMAJOR    1: k is the contiguous axis of the operand, 0: m/n is
//   B200_IDESC                tcgen05 instruction descriptor (formats, majors, M, N)
//   B200_TMEM_COLS            power of two >= 2*B200_BN (and >= 32)
//   B200_CLUSTER_K            > 1: CTAs that share the k blocks of a tile (undefined: one); B200_WARP_COLS: columns a warp finishes
//   B200_BLOCK / B200_GRID    the kernel's block index and block count (a device function of a launch group: its share)
//   B200_EPI_PARAMS           extra kernel parameters (node pointers) of the epilogue
//   B200_EPILOGUE_ROW(...)    statement block evaluated per (row, 32-column chunk), see below
#ifndef B200_GEMM_SM100_CUH
#define B200_GEMM_SM100_CUH

#ifndef B200_TC_SM100_CUH
#include "tc_sm100.cuh"
#endif
// The shape is part of what is compiled: B200_M / _N / _K, batch extents B200_B0 (outer) and B200_B1 (inner),
// B200_A_B0 .. B200_B_B1 (1 when the operand varies along that batch axis), B200_TILES_M / _N.  Tile coordinates
// are quotients by these; as kernel arguments they cost the producer seven chained divisions, about 0.3 us,
// before its first copy.
struct b200_gemm_shape {
  unsigned int tma_out;         // != 0: the epilogue's row-contiguous outputs leave as TMA stores (their maps are valid)
};


__device__ __forceinline__ void b200_tmem_ld_chunk(unsigned int taddr, unsigned int* r) {
#if B200_EPI_CHUNK == 64
  b200_tmem_ld32(taddr, r);
  b200_tmem_ld32(taddr + 32u, r + 32);
#elif B200_EPI_CHUNK == 32
  b200_tmem_ld32(taddr, r);
#else
  b200_tmem_ld16(taddr, r);
#endif
}

// Developer aid: with -DB200_TRACE, CTA 0 records nanoseconds since its start at a few points
// into words 2..15 of the device status buffer (printed by the host when B200_TRACE is set).
#ifdef B200_TRACE
#define B200_TR(slot) do { if (blockIdx.x == 0) status[slot] = (unsigned int)(b200_now_ns() - b200_t0); } while (0)
#else
#define B200_TR(slot) do { } while (0)
#endif

// per CTA: 128 rows of A; all of the tile's B columns, or half of them in pair mode
#define B200_CTA_M 128
#define B200_CTA_N (B200_BN / (1 + B200_CTA_PAIR))
#define B200_A_TILE_BYTES (B200_CTA_M * B200_BK * B200_ELEM_BYTES)
// Rows of A that are staged.  A contraction of fewer than 128 rows copies those alone, in whole swizzle groups of
// eight (k-major) or chunks of 128 bytes (m-major): what the copies fill with zeros beyond M also passes through
// the 64 bytes a clock that an SM takes in, which bound 37 rows of 784-1024-1024 (2.8 us for 13 k blocks of
// 128 x 16 tiles).  The rest of the tile stays as it is: it only reaches accumulator rows that nobody reads.
#if B200_M >= B200_CTA_M
#define B200_A_ROWS B200_CTA_M
#elif B200_A_KMAJOR
#define B200_A_ROWS ((B200_M + 7) / 8 * 8)
#else
#define B200_A_ROWS ((B200_M + B200_ROW_ELEMS - 1) / B200_ROW_ELEMS * B200_ROW_ELEMS)
#endif
#define B200_STAGE_COPY_BYTES ((B200_A_ROWS * B200_BK * B200_ELEM_BYTES + B200_B_TILE_BYTES) * (1 + B200_PAIRS))
#define B200_B_TILE_BYTES (B200_CTA_N * B200_BK * B200_ELEM_BYTES)
// B200_PAIRS: single-precision operands as tf32 pairs, x = hi + lo, stored by the gathering kernel as two
// segments of B200_SEG positions along k.  A ring slot then holds both parts of both operands, and each
// is used twice: hi lo + lo hi + hi hi.  (Three passes over segments of 3 k positions, as if k were
// three times as long, moved half as many bytes again into shared memory per product and were bound by
// that: 665 cycles per k block of a 128 x 128 tile.)
#ifndef B200_PAIRS
#define B200_PAIRS 0
#define B200_SEG 0
#endif
#define B200_STAGE_BYTES ((B200_A_TILE_BYTES + B200_B_TILE_BYTES) * (1 + B200_PAIRS))
#define B200_B_AT (B200_A_TILE_BYTES * (1 + B200_PAIRS))   // where a slot's B tile (or pair of tiles) begins
#define B200_THREADS (64 + 32 * B200_EPI_WARPS)
// elements of the contiguous axis covered by one 128-byte swizzle row
#define B200_ROW_ELEMS (128 / B200_ELEM_BYTES)
#ifndef B200_EPI_CHUNK
#if B200_BN >= 32
#define B200_EPI_CHUNK 32
#else
#define B200_EPI_CHUNK 16
#endif
#endif
#ifndef B200_RASTER
#define B200_RASTER 8
#endif
// B200_SPLITK work units per tile, each over its own slice of the k blocks (the epilogue then adds
// its partial tile to the output with reductions in global memory)
#ifndef B200_SPLITK
#define B200_SPLITK 1
#endif
// B200_FLUSH > 0: the accumulator leaves tensor memory every B200_FLUSH k blocks and is summed in the
// epilogue threads' registers.  The tensor cores cut every addition into the accumulator off instead of
// rounding it, which after n MMAs has moved a sum by about n 2^-25 of itself towards zero: too much for
// operands that travel as tf32 pairs and are meant to keep single precision (3e-6 at K = 131, growing
// with K).  Short runs that are added up with rounding stay within what a chain of fp32 additions does.
#ifndef B200_FLUSH
#define B200_FLUSH 0
#endif
// B200_CLUSTER_K > 1: few tiles, and most of the time of each is its walk along k (a k block of a 128 x 16 tile
// brings 18 KB into the SM at some 60 bytes a clock, whatever little is multiplied with it).  A cluster of 2 or 4
// CTAs shares a tile, each CTA taking a slice of its k blocks; every CTA then finishes 128 / B200_CLUSTER_K of the
// tile's rows: the epilogue warps hand the rows of their tensor-memory quarter to the CTA that finishes
// them, into its shared memory (column groups of four, a lane's row next to its neighbours': 512 bytes an
// instruction), where its barrier counts the bytes.  The partials are added in the order of the slices.
// The exchange is what it costs: some 16 bytes a clock leave an SM this way, 0.35 us for 16 columns, 0.75 for 32, 1.3 for
// 64 (bulk copies out of shared memory: 0.5, 1.0, 1.6).  Runs back to back without
// and with clusters: 128 rows of 2048-2048-2048-10 24.3 -> 17.8 us; 64 of 4096-4096-256-10 27.5 -> 18.1; 37 of 784-1024-1024-10 16.8 -> 14.9.
// A cluster takes one tile: the grid has B200_CLUSTER_K CTAs for each.
#if B200_CLUSTER_K > 1
#define B200_X_GROUPS (4 / B200_CLUSTER_K)                 // groups of 32 rows that a CTA finishes
#define B200_X_BYTES (4 * 32 * B200_BN * 4)                // partials on their way: CLUSTER_K x X_GROUPS x 32 rows x BN columns
#else
#define B200_X_BYTES 0
#endif
// columns of the tile that an epilogue warp works on
#ifndef B200_WARP_COLS
#define B200_WARP_COLS (B200_BN / (B200_EPI_WARPS / 4))
#endif

// Contractions that do not depend on one another and together leave SMs idle run as one launch: a kernel that calls this
// one, compiled once for each of them as a device function, by ranges of its blocks.  B200_BLOCK / B200_GRID are then the
// function's parameters.
#ifndef B200_KERNEL_HEAD
#define B200_KERNEL_HEAD extern "C" __global__ void __launch_bounds__(B200_THREADS, 1) B200_GEMM_NAME
#define B200_TMAP_PARAM const __grid_constant__ b200_tmap
#define B200_BLOCK_PARAMS
#define B200_BLOCK blockIdx.x
#define B200_GRID gridDim.x
#endif

B200_KERNEL_HEAD(B200_TMAP_PARAM map_a, B200_TMAP_PARAM map_b, const b200_gemm_shape shape, unsigned int* status B200_BLOCK_PARAMS B200_EPI_PARAMS) {
  extern __shared__ unsigned char b200_dyn_smem[];
  // tiles need 1024-byte alignment for the 128-byte swizzle pattern
  const unsigned int smem_base = (b200_smem_addr(b200_dyn_smem) + 1023u) & ~1023u;
  unsigned char* smem_gen = b200_dyn_smem + (smem_base - b200_smem_addr(b200_dyn_smem));
  const unsigned int tiles_at = smem_base;
  // the epilogue warps' staging tiles follow the ring (1024-byte aligned, as the swizzled TMA stores want);
  // barriers and bookkeeping live after them
  constexpr unsigned int x_offset = B200_STAGES * B200_STAGE_BYTES + B200_EPI_WARPS * (B200_STAGING_TILES * B200_STAGING_BYTES + B200_LOAD_TILE_BYTES);
  unsigned long long* bars = (unsigned long long*)(smem_gen + x_offset + B200_X_BYTES);
  const unsigned int bar_full = b200_smem_addr(bars);                          // [STAGES]
  const unsigned int bar_empty = bar_full + 8u * B200_STAGES;                  // [STAGES]
  const unsigned int bar_acc_full = bar_empty + 8u * B200_STAGES;              // [2]
  const unsigned int bar_acc_empty = bar_acc_full + 16u;                       // [2]
  const unsigned int bar_load = bar_acc_empty + 16u;                           // [EPI_WARPS]: row operands loaded by TMA
  const unsigned int bar_x = bar_load + 8u * B200_EPI_WARPS;                   // [1]: partials of the other CTAs of a cluster
  volatile unsigned int* tmem_slot = (volatile unsigned int*)(bars + 2 * B200_STAGES + 5 + B200_EPI_WARPS);
  volatile unsigned int* abort_flag = tmem_slot + 1;

  // the next kernel in the stream may be placed as soon as every CTA of this one is running
  asm volatile("griddepcontrol.launch_dependents;");
  const unsigned int warp = threadIdx.x >> 5;
  const unsigned int lane = threadIdx.x & 31u;
#ifdef B200_TRACE
  const unsigned long long b200_t0 = b200_now_ns();
  B200_TRE(-1);
#endif

  if (threadIdx.x == 32) {
    // the descriptors are fetched while the barriers and the tensor memory are being set up
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_b) : "memory");
  }
  if (threadIdx.x == 0) {
    for (unsigned int s = 0; s < B200_STAGES; ++s) {
      b200_mbar_init(bar_full + 8u * s, 1);
      b200_mbar_init(bar_empty + 8u * s, 1);
    }
    for (unsigned int a = 0; a < 2; ++a) {
      b200_mbar_init(bar_acc_full + 8u * a, 1);
      // the leader's accumulator buffer is free again when the epilogue warps of both CTAs are done with it
      b200_mbar_init(bar_acc_empty + 8u * a, B200_EPI_WARPS * (1 + B200_CTA_PAIR));
    }
    for (unsigned int w = 0; w < B200_EPI_WARPS; ++w) b200_mbar_init(bar_load + 8u * w, 1);
    b200_mbar_init(bar_x, 1);
#if B200_CLUSTER_K > 1
    b200_mbar_expect_tx(bar_x, B200_X_BYTES);   // the partials of all CTAs of the cluster, this one's included
#endif
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc." B200_CG ".sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(b200_smem_addr((const void*)tmem_slot)),
                 "r"((unsigned int)B200_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit." B200_CG ".sync.aligned;" ::: "memory");
  }
  // Set-up touches no global memory and is over, block-wide barrier included, before the grids ahead of this one
  // end; the threads that read or write global memory (the producer, the epilogue) then wait for those grids
  // themselves, right ahead of their first access, and no limited wait begins before that.  The MMA issuer goes
  // straight to its first operands, however long those grids take: should operands never come, it is the epilogue
  // that finds out, and ends this wait too.
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  b200_cluster_sync();   // the peer's barriers are initialised before anything is signalled on them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned int tmem_base = *tmem_slot;
  const unsigned int cta_rank = b200_cta_rank();
  const unsigned int k_rank = b200_k_rank();
  // tiles are taken by CTA pairs in pair mode, by clusters that share the k blocks, by single CTAs otherwise
  constexpr unsigned int ctas_per_worker = B200_CTA_PAIR ? 2 : B200_CLUSTER_K;
  const unsigned int worker = B200_BLOCK / ctas_per_worker, n_workers = B200_GRID / ctas_per_worker;
  if (threadIdx.x == 0) B200_TR(2);   // set-up done

  constexpr unsigned int tiles_per_batch = B200_TILES_M * B200_TILES_N;
  constexpr unsigned int total_tiles = tiles_per_batch * B200_B0 * B200_B1;
  constexpr unsigned int k_blocks = (B200_K + B200_BK - 1) / B200_BK;
  constexpr unsigned int total_units = total_tiles * B200_SPLITK;
  constexpr unsigned int k_slices = B200_SPLITK * B200_CLUSTER_K;   // (one of the two is 1)

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (b200_elect()) {
      unsigned int slot = 0, phase = 0;
      bool live = true;
      asm volatile("griddepcontrol.wait;" ::: "memory");
      for (unsigned int unit = worker; live && unit < total_units; unit += n_workers) {
        const unsigned int tile = unit % total_tiles, split = unit / total_tiles * B200_CLUSTER_K + k_rank;
        const unsigned int kb0 = split * k_blocks / k_slices, kb1 = (split + 1u) * k_blocks / k_slices;
        const unsigned int bidx = tile / tiles_per_batch;
        const unsigned int t = tile - bidx * tiles_per_batch;
        // consecutive tiles walk down m first so that a wave of CTAs shares few B tiles
        const unsigned int group = t / (B200_RASTER * B200_TILES_N);
        const unsigned int first_m = group * B200_RASTER;
        const unsigned int rows = min((unsigned int)B200_RASTER, B200_TILES_M - first_m);
        const unsigned int r = t - group * B200_RASTER * B200_TILES_N;
        const unsigned int mt = first_m + r % rows;
        const unsigned int nt = r / rows;
        const unsigned int b0 = bidx / B200_B1, b1 = bidx - b0 * B200_B1;
        // this CTA's rows of A and its share of the tile's B columns
        const int m0 = (int)(mt * B200_BM + cta_rank * B200_CTA_M), n0 = (int)(nt * B200_BN + cta_rank * B200_CTA_N);
        for (unsigned int kb = kb0; kb < kb1; ++kb) {
#ifdef B200_INJECT_NO_LOADS
          // failure-detection test only: the producer loads nothing, so the waits for operands can
          // never be satisfied and must run out (no copy or MMA is ever in flight in this build)
          continue;
#endif
          if (!b200_wait(bar_empty + 8u * slot, phase ^ 1u, abort_flag, status, 1u)) { live = false; break; }
          // both CTAs' copies complete on the leader's barrier; the leader announces the bytes of both
          const unsigned int full = b200_map_to_cta(bar_full + 8u * slot, 0u);   // (the barrier itself when not paired)
          if (cta_rank == 0u) b200_mbar_expect_tx(bar_full + 8u * slot, B200_STAGE_COPY_BYTES * (1 + B200_CTA_PAIR));
          const unsigned int sa = tiles_at + slot * B200_STAGE_BYTES;
          const unsigned int sb = sa + B200_B_AT;
#pragma unroll
          for (int part = 0; part < 1 + B200_PAIRS; ++part) {
          const int k0 = (int)(kb * B200_BK) + part * B200_SEG;
          const unsigned int pa = sa + part * B200_A_TILE_BYTES, pb = sb + part * B200_B_TILE_BYTES;
#if B200_A_KMAJOR
          b200_tma_load_4d(pa, &map_a, full, k0, m0, (int)(b1 * B200_A_B1), (int)(b0 * B200_A_B0));
#else
#pragma unroll
          for (int c = 0; c < (int)B200_A_ROWS / B200_ROW_ELEMS; ++c)
            b200_tma_load_4d(pa + c * (B200_ROW_ELEMS * B200_BK * B200_ELEM_BYTES), &map_a, full, m0 + c * B200_ROW_ELEMS, k0,
                             (int)(b1 * B200_A_B1), (int)(b0 * B200_A_B0));
#endif
#if B200_B_KMAJOR
          b200_tma_load_4d(pb, &map_b, full, k0, n0, (int)(b1 * B200_B_B1), (int)(b0 * B200_B_B0));
#else
#pragma unroll
          for (int c = 0; c < B200_CTA_N / B200_ROW_ELEMS; ++c)
            b200_tma_load_4d(pb + c * (B200_ROW_ELEMS * B200_BK * B200_ELEM_BYTES), &map_b, full, n0 + c * B200_ROW_ELEMS, k0,
                             (int)(b1 * B200_B_B1), (int)(b0 * B200_B_B0));
#endif
          }
          if (unit == worker && kb == kb0) B200_TR(3);   // first loads issued
          if (++slot == B200_STAGES) { slot = 0; phase ^= 1u; }
        }
      }
      B200_TR(4);   // producer done
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (the leader CTA of a pair)
    if (cta_rank == 0u && b200_elect()) {
      unsigned int slot = 0, phase = 0, acc = 0, acc_phase = 0;
      bool live = true;
      // operand descriptors of ring slot 0.  k-major: rows of 128 bytes, 8-row groups 1024 bytes
      // apart.  m/n-major: 64-element (128-byte) chunks of m/n, k rows 128 bytes apart, 8-row groups
      // 1024 bytes apart, chunks one box apart.
#if B200_A_KMAJOR
      const unsigned long long desc_a0 = b200_smem_desc(tiles_at, 16u, 1024u);
#else
      const unsigned long long desc_a0 = b200_smem_desc(tiles_at, B200_ROW_ELEMS * B200_BK * B200_ELEM_BYTES, B200_MN_GROUP_BYTES, B200_MN_SWIZZLE);
#endif
#if B200_B_KMAJOR
      const unsigned long long desc_b0 = b200_smem_desc(tiles_at + B200_B_AT, 16u, 1024u);
#else
      const unsigned long long desc_b0 =
          b200_smem_desc(tiles_at + B200_B_AT, B200_ROW_ELEMS * B200_BK * B200_ELEM_BYTES, B200_MN_GROUP_BYTES, B200_MN_SWIZZLE);
#endif
      for (unsigned int unit = worker; live && unit < total_units; unit += n_workers) {
        const unsigned int split = unit / total_tiles * B200_CLUSTER_K + k_rank;
        const unsigned int kb0 = split * k_blocks / k_slices, kb1 = (split + 1u) * k_blocks / k_slices;
        for (unsigned int kbf = kb0; live && kbf < kb1;) {
          // one run of k blocks into one accumulator buffer: the whole unit, or B200_FLUSH blocks of it
          const unsigned int kbe = B200_FLUSH ? min(kbf + (unsigned int)B200_FLUSH, kb1) : kb1;
          if (!b200_wait(bar_acc_empty + 8u * acc, acc_phase ^ 1u, abort_flag, status, 2u)) { live = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned int d_tmem = tmem_base + acc * B200_BN;
          for (unsigned int kb = kbf; kb < kbe; ++kb) {
            if (!b200_wait_aborted(bar_full + 8u * slot, phase, abort_flag)) { live = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (unit == worker && kb == kb0) B200_TR(5);   // first operands landed
            // descriptors of this slot: the start-address field (bits 0-13, address >> 4) moves, the rest is fixed
            const unsigned long long da0 = desc_a0 + (unsigned long long)((slot * B200_STAGE_BYTES) >> 4);
            const unsigned long long db0 = desc_b0 + (unsigned long long)((slot * B200_STAGE_BYTES) >> 4);
#pragma unroll
            for (unsigned int p = 0; p < 1 + 2 * B200_PAIRS; ++p) {
              // the parts multiplied: both as stored, or (A hi, B lo), (A lo, B hi), (A hi, B hi)
              const unsigned long long dap = da0 + (unsigned long long)((p == 1u ? B200_A_TILE_BYTES : 0u) >> 4);
              const unsigned long long dbp = db0 + (unsigned long long)((B200_PAIRS && p == 0u ? B200_B_TILE_BYTES : 0u) >> 4);
#pragma unroll
              for (unsigned int ks = 0; ks < B200_BK / B200_UMMA_K; ++ks) {
                // a k step moves UMMA_K elements along a k-major row, or UMMA_K rows of 128 bytes in the m/n-major form
                const unsigned long long da = dap + (unsigned long long)((ks * (B200_A_KMAJOR ? B200_UMMA_K * B200_ELEM_BYTES : B200_UMMA_K * 128u)) >> 4);
                const unsigned long long db = dbp + (unsigned long long)((ks * (B200_B_KMAJOR ? B200_UMMA_K * B200_ELEM_BYTES : B200_UMMA_K * 128u)) >> 4);
                b200_umma(d_tmem, da, db, (unsigned int)B200_IDESC, (kb != kbf || ks != 0u || p != 0u) ? 1u : 0u);
              }
            }
            b200_umma_commit(bar_empty + 8u * slot);  // frees the slot once these MMAs retire
            if (++slot == B200_STAGES) { slot = 0; phase ^= 1u; }
          }
          if (live) b200_umma_commit(bar_acc_full + 8u * acc);
          if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
          kbf = kbe;
        }
        if (unit == worker) B200_TR(6);                  // tile 0 MMAs issued
        else if (unit == worker + n_workers) B200_TR(7); // tile 1 MMAs issued
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const unsigned int ew = warp - 2;                 // 0 .. EPI_WARPS-1
    const unsigned int quarter = warp & 3u;           // TMEM lanes this warp may read
#if B200_CLUSTER_K > 1
    const unsigned int row_group = k_rank * B200_X_GROUPS + ew % B200_X_GROUPS;   // the 32 rows of the tile this warp finishes
    const unsigned int col_part = ew / B200_X_GROUPS;                             // and which part of its columns
    const bool b200_idle = col_part * B200_WARP_COLS >= B200_BN;
#else
    const unsigned int row_group = quarter;
    const unsigned int col_part = ew >> 2;
    constexpr bool b200_idle = false;
#endif
    constexpr unsigned int cols_per_warp = B200_WARP_COLS;
    // this warp's 4 KB staging tile (transposes a chunk so that stores cover whole row segments)
    uint4* b200_stage = (uint4*)(smem_gen + B200_STAGES * B200_STAGE_BYTES + ew * (unsigned int)(B200_STAGING_TILES * B200_STAGING_BYTES));
    b200_epi_state b200_es;
    b200_es.tma = shape.tma_out != 0u;
    b200_es.nst = 0u;
    // the tile and barrier of a row operand that arrives by TMA (B200_LOAD_TILE_BYTES is 0 without one)
    b200_es.ltile = (uint4*)(smem_gen + B200_STAGES * B200_STAGE_BYTES + B200_EPI_WARPS * B200_STAGING_TILES * B200_STAGING_BYTES +
                             ew * (unsigned int)B200_LOAD_TILE_BYTES);
    b200_es.lbar = bar_load + 8u * ew;
    b200_es.lph = 0u;
    b200_es.abort_flag = abort_flag;
    b200_es.status = status;
    b200_es.part = 0.0f;
    B200_EPI_PROLOGUE
    asm volatile("griddepcontrol.wait;" ::: "memory");
    unsigned int acc = 0, acc_phase = 0;
    // (batch, row, first column) of the part of a unit's tile that this thread works on
    auto b200_coords = [&](unsigned int u, unsigned int& tile, unsigned int& b0, unsigned int& b1, unsigned int& mt, unsigned int& nt) {
      tile = u % total_tiles;
      const unsigned int bidx = tile / tiles_per_batch;
      const unsigned int t = tile - bidx * tiles_per_batch;
      const unsigned int group = t / (B200_RASTER * B200_TILES_N);
      const unsigned int first_m = group * B200_RASTER;
      const unsigned int rows = min((unsigned int)B200_RASTER, B200_TILES_M - first_m);
      const unsigned int r = t - group * B200_RASTER * B200_TILES_N;
      mt = first_m + r % rows;
      nt = r / rows;
      b0 = bidx / B200_B1;
      b1 = bidx - b0 * B200_B1;
    };
    // operand tiles of the epilogue (bias, mask, residual rows ...): loaded for a tile's first chunk
    // before its accumulator is waited for -- by the previous tile's last chunk when there was one
    b200_in_tiles b200_tiles;
    bool b200_prefetched = false;
    for (unsigned int unit = worker; unit < total_units; unit += n_workers) {
      unsigned int tile, b200_b0, b200_b1, mt, nt;
      b200_coords(unit, tile, b200_b0, b200_b1, mt, nt);
      const unsigned int b200_m = mt * B200_BM + cta_rank * B200_CTA_M + row_group * 32u + lane;
      // one scratch slot per epilogue warp of the grid for epilogues that end in a grid-wide sum (whose tiles are one
      // chunk wide: of a cluster's warps, those of the first column part)
#if B200_CLUSTER_K > 1
      const unsigned int b200_slot = B200_BLOCK * B200_X_GROUPS + ew % B200_X_GROUPS, b200_nslots = B200_GRID * B200_X_GROUPS;
#else
      const unsigned int b200_slot = B200_BLOCK * B200_EPI_WARPS + ew, b200_nslots = B200_GRID * B200_EPI_WARPS;
#endif
      // this warp's share of the next tile, for the prefetch at the end of this one
      bool b200_nx_ok = false;
      unsigned int b200_nx_b0 = 0, b200_nx_b1 = 0, b200_nx_m = 0, b200_nx_n0 = 0;
      if (unit + n_workers < total_units) {
        unsigned int ntile, nmt, nnt;
        b200_coords(unit + n_workers, ntile, b200_nx_b0, b200_nx_b1, nmt, nnt);
        b200_nx_m = nmt * B200_BM + cta_rank * B200_CTA_M + row_group * 32u + lane;
        b200_nx_n0 = nnt * B200_BN + col_part * cols_per_warp;
        b200_nx_ok = b200_nx_n0 < B200_N;
      }
      B200_EPILOGUE_ROWS
      if (!b200_prefetched) {
        const unsigned int b200_pn0 = nt * B200_BN + col_part * cols_per_warp;
        if (!b200_idle && b200_pn0 < B200_N) { B200_EPILOGUE_LOAD }
      }
      b200_prefetched = b200_nx_ok && (nt * B200_BN + col_part * cols_per_warp < B200_N);
#if B200_FLUSH
      constexpr int kCols = (B200_WARP_COLS + B200_EPI_CHUNK - 1) / B200_EPI_CHUNK * B200_EPI_CHUNK;
      const unsigned int col0 = col_part * cols_per_warp;
      float b200_sum[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) b200_sum[j] = 0.0f;
      {
        const unsigned int split = unit / total_tiles;
        const unsigned int kb0 = split * k_blocks / B200_SPLITK, kb1 = (split + 1u) * k_blocks / B200_SPLITK;
        bool got = true;
        for (unsigned int kbf = kb0; kbf < kb1; kbf += B200_FLUSH) {
          got = b200_wait(bar_acc_full + 8u * acc, acc_phase, abort_flag, status, 4u);
          if (!got) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned int taddr = tmem_base + acc * B200_BN + ((quarter * 32u) << 16) + col0;
          unsigned int part[kCols];
#pragma unroll
          for (int c = 0; c < kCols; c += B200_EPI_CHUNK) b200_tmem_ld_chunk(taddr + c, part + c);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < kCols; ++j) b200_sum[j] += __uint_as_float(part[j]);
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) b200_mbar_arrive_relaxed(bar_acc_empty + 8u * acc);
          if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
        }
        if (!got) break;
      }
#pragma unroll
      for (int c = 0; c < kCols; c += B200_EPI_CHUNK) {
        const unsigned int b200_n0 = nt * B200_BN + col0 + c;
        if (b200_n0 >= B200_N) break;  // warp-uniform
        unsigned int b200_r[B200_EPI_CHUNK];
#pragma unroll
        for (int j = 0; j < B200_EPI_CHUNK; ++j) b200_r[j] = __float_as_uint(b200_sum[c + j]);
        const bool b200_has_next = (c + B200_EPI_CHUNK < cols_per_warp) && (b200_n0 + B200_EPI_CHUNK < B200_N);
        const unsigned int b200_next_taddr = tmem_base;   // (a load that nothing reads)
        B200_EPILOGUE_ROW
      }
#elif B200_CLUSTER_K > 1
      const bool got_acc = b200_wait(bar_acc_full, 0u, abort_flag, status, 4u);
      if (got_acc) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned int taddr = tmem_base + ((quarter * 32u) << 16);
        // partials lie as [slice][row group][columns / 4][row]
        const unsigned int owner = quarter / B200_X_GROUPS, bar = b200_map_to_rank(bar_x, owner);
        const unsigned int to = b200_map_to_rank(smem_base + x_offset + ((k_rank * B200_X_GROUPS + quarter % B200_X_GROUPS) * (B200_BN / 4) * 32u + lane) * 16u, owner);
        constexpr int step = B200_BN >= 32 ? 32 : 16;
#pragma unroll
        for (int c = 0; c < B200_BN; c += step) {
          unsigned int part[step];
          if constexpr (step == 32) b200_tmem_ld32(taddr + c, part); else b200_tmem_ld16(taddr + c, part);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int g = 0; g < step / 4; ++g) b200_st_async(to + (c / 4 + g) * 512u, bar, part[4 * g], part[4 * g + 1], part[4 * g + 2], part[4 * g + 3]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      }
      b200_cluster_arrive_relaxed();   // nothing more goes to the other CTAs' shared memory
      if (!got_acc || !b200_wait(bar_x, 0u, abort_flag, status, 6u)) break;
      if (b200_idle) break;   // (a cluster takes one tile)
      const uint4* const from = (const uint4*)(smem_gen + x_offset) + (ew % B200_X_GROUPS) * (B200_BN / 4) * 32u + lane;
#pragma unroll 1
      for (unsigned int c = 0; c < cols_per_warp; c += B200_EPI_CHUNK) {
        const unsigned int col = col_part * cols_per_warp + c;
        const unsigned int b200_n0 = nt * B200_BN + col;
        if (b200_n0 >= B200_N) break;  // warp-uniform
        unsigned int b200_r[B200_EPI_CHUNK];
#pragma unroll
        for (int g = 0; g < B200_EPI_CHUNK / 4; ++g) {
          float4 v = *(const float4*)(from + (col / 4 + g) * 32u);
#pragma unroll
          for (int r = 1; r < B200_CLUSTER_K; ++r) {
            const float4 w = *(const float4*)(from + (r * B200_X_GROUPS * (B200_BN / 4) + col / 4 + g) * 32u);
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
          }
          b200_r[4 * g] = __float_as_uint(v.x); b200_r[4 * g + 1] = __float_as_uint(v.y);
          b200_r[4 * g + 2] = __float_as_uint(v.z); b200_r[4 * g + 3] = __float_as_uint(v.w);
        }
        const bool b200_has_next = (c + B200_EPI_CHUNK < cols_per_warp) && (b200_n0 + B200_EPI_CHUNK < B200_N);
        const unsigned int b200_next_taddr = tmem_base;   // (a load that nothing reads)
        B200_EPILOGUE_ROW
      }
#else
      if (!b200_wait(bar_acc_full + 8u * acc, acc_phase, abort_flag, status, 4u)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (warp == 2 && lane == 0) { if (unit == worker) B200_TR(8); else if (unit == worker + n_workers) B200_TR(10); }
#ifdef B200_TRACE
      B200_TRE(3);   // waiting for the accumulator (and the operand prefetch before it)
#endif
      const unsigned int taddr = tmem_base + acc * B200_BN + ((quarter * 32u) << 16);
      // One register buffer: the epilogue issues the TMEM load of the next chunk as soon as it
      // has consumed the current one, so the load overlaps the epilogue's stores.  (The loop is
      // deliberately not unrolled: the generated epilogue can be thousands of instructions.)
      unsigned int b200_r[B200_EPI_CHUNK];
      const unsigned int col0 = col_part * cols_per_warp;
      if (nt * B200_BN + col0 < B200_N) b200_tmem_ld_chunk(taddr + col0, b200_r);
#pragma unroll 1
      for (unsigned int c = 0; c < cols_per_warp; c += B200_EPI_CHUNK) {
        const unsigned int col = col0 + c;
        const unsigned int b200_n0 = nt * B200_BN + col;
        if (b200_n0 >= B200_N) break;  // warp-uniform
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#ifdef B200_TRACE
        B200_TRE(4);
#endif
        const bool b200_has_next = (c + B200_EPI_CHUNK < cols_per_warp) && (b200_n0 + B200_EPI_CHUNK < B200_N);
        const unsigned int b200_next_taddr = taddr + col + B200_EPI_CHUNK;
        // every lane takes part: rows beyond M compute nothing but help move the chunk
        B200_EPILOGUE_ROW
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
#if B200_CTA_PAIR
      if (lane == 0) b200_mbar_arrive_cluster_relaxed(b200_map_to_cta(bar_acc_empty + 8u * acc, 0u));
#else
      if (lane == 0) b200_mbar_arrive_relaxed(bar_acc_empty + 8u * acc);
#endif
      if (warp == 2 && lane == 0) { if (unit == worker) B200_TR(9); else if (unit == worker + n_workers) B200_TR(11); }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
#endif
#ifdef B200_TRACE
      B200_TRE(5);   // release of the accumulator buffer
#endif
    }
    // the copy engine has read this warp's staging tiles before the CTA gives its shared memory back
    if (lane == 0) b200_tma_store_read_wait<0>();
#ifdef B200_TRACE
    b200_tre(0, true, status);
#endif
  }

  // ---------------------------------------------------------------------- teardown
  __syncwarp();
#if B200_CLUSTER_K > 1
  if (warp < 2) b200_cluster_arrive_relaxed();   // (the epilogue's warps have arrived after their last copies)
#endif
  if (*abort_flag) {
    // let copies and MMAs already in flight land before the tensor memory is released
    const unsigned long long t0 = b200_now_ns();
    while (b200_now_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // no CTA of a cluster leaves while another may still read or write its memory or signal its barriers
#if B200_CLUSTER_K > 1
  b200_cluster_wait();
#else
  b200_cluster_sync();
#endif
  if (threadIdx.x == 0) B200_TR(12);  // all roles done
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc." B200_CG ".sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((unsigned int)B200_TMEM_COLS)
                 : "memory");
  }
}

#endif  // B200_GEMM_SM100_CUH
