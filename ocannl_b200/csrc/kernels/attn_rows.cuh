// Fused attention stage for short rows: the chain of attn_sm100.cuh (scores, softmax, weights . values) for
// any number of keys up to 256 and any head dimension that is a multiple of 16.
//
// A warp takes 16 queries of one (batch, head), in the accumulator layout of mma.m16n8k16: thread (g, c) =
// (lane / 4, lane % 4) holds columns 8 n + 2 c and + 1 of rows g and g + 8 for every key tile n.  Scores, then
// exponentials, lie in shared memory, four per thread and tile, each read back by the thread that wrote it (no
// barrier); row maximum and sum are two shuffles within four lanes; the weights, rounded to the node's 16-bit
// format, are at once the A fragments of the second product, whose B fragments come transposed out of shared
// memory (ldmatrix.trans).  Keys and values of the (batch, head) lie in shared memory too, rows padded by 16
// bytes so that the eight rows of an ldmatrix fall into different banks.
// What bounds it: latency, of the loads and of three short loops per warp (scores; exponentials; weights and
// their product); neither a tensor-memory round trip nor a block-wide barrier stands between them, and a
// sequence of 100 positions is 7 warps' work where the tile kernels pad it to 128 x 128.  The loops run over 16
// keys at a time and are not unrolled further than twice: score rows held in registers instead meant straight
// code of up to 150 KB, which was fetched from memory more slowly than it ran (66 heads of 192 queries and keys: 23 us,
// now 17 us, 6 of it the launch).
//
// 16 keys for which no query of the warp has a mask bit set are not multiplied, and their scores are one
// constant per row: exponential and weight are evaluated once for all of them, and when that weight is zero
// (it is, unless a row is masked throughout) they add nothing to the output either.  A causal mask halves the
// work this way.
//
// The translation unit defines B200_AR_NAME, B200_T, B200_E, B200_HALF (1: half, 0: bfloat16), B200_WARPS, B200_KS,
// B200_OUT_T (storage type of the output), B200_NCOND, B200_MASKED (1: the score is a constant where mask 0 is
// zero), B200_KEEP_SCORES / _EXP / _W, B200_ATTN_PARAMS / B200_ATTN_ARGS, and the generated functions below.
#ifndef B200_ATTN_ROWS_CUH
#define B200_ATTN_ROWS_CUH

struct b200_ar_shape {
  unsigned int S, B0, B1, tiles;           // queries; batch extents, outer and inner; query tiles per (batch, head)
  long long q_row, q_b0, q_b1, k_row, k_b0, k_b1, v_row, v_b0, v_b1;   // element strides
};
struct b200_attn_row {
  unsigned int b0, b1, s;
  bool ok;
};
struct b200_ar_ptrs {   // addresses of this row in the nodes the routine keeps (0: not written)
  unsigned long long scores, mx, exps, sum, w, out;
};

#define B200_NT ((B200_T + 15) / 16 * 2)          // key tiles of 8, an even number
#define B200_TP (B200_NT * 8)
#define B200_LD (B200_E + 8)                      // elements per padded row in shared memory
#define B200_NP (B200_NT / 2)                     // the loops' steps, 16 keys each
// B200_KS warps share 16 queries (1, 2 or 4 of a block's B200_WARPS): each takes every B200_KS'th step of 16 keys, and
// row maxima, sums and outputs meet in shared memory.  With few heads most SMs hold a warp or two, and a warp's
// three loops are one chain of latencies, as long as the row.
#define B200_QT (B200_WARPS / B200_KS)            // groups of 16 queries in a block

__device__ __forceinline__ float b200_ar_score(const b200_attn_row& row, unsigned int b200_t, float b200_acc, unsigned int cb0, unsigned int cb1 B200_ATTN_PARAMS);
__device__ __forceinline__ float b200_ar_masked_score();
__device__ __forceinline__ float b200_ar_max_init();
__device__ __forceinline__ float b200_ar_row_max(const b200_attn_row& row, float reduced B200_ATTN_PARAMS);
__device__ __forceinline__ float b200_ar_exp(const b200_attn_row& row, unsigned int b200_t, float x, float mx B200_ATTN_PARAMS);
__device__ __forceinline__ float b200_ar_row_sum(const b200_attn_row& row, float reduced B200_ATTN_PARAMS);
__device__ __forceinline__ float b200_ar_divisor(const b200_attn_row& row, float sum B200_ATTN_PARAMS);
template <bool FAST>
__device__ __forceinline__ float b200_ar_weight(const b200_attn_row& row, unsigned int b200_t, float e, float sum, const b200_divisor& b200_dv B200_ATTN_PARAMS);
__device__ __forceinline__ B200_OUT_T b200_ar_out(const b200_attn_row& row, unsigned int b200_e, float b200_acc B200_ATTN_PARAMS);
__device__ __forceinline__ void b200_ar_rows(const b200_attn_row& row, b200_ar_ptrs& p B200_ATTN_PARAMS);
__device__ __forceinline__ void b200_ar_cond_rows(const b200_attn_row& row, const unsigned int** p B200_ATTN_PARAMS);

__device__ __forceinline__ void b200_ar_mma(float* d, const unsigned int* a, unsigned int b0, unsigned int b1) {
#if B200_HALF
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
#else
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
#endif
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void b200_ldsm4(unsigned int* r, unsigned int addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void b200_ldsm4t(unsigned int* r, unsigned int addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ unsigned int b200_ar_pack(float lo, float hi) {
#if B200_HALF
  return b200_pack_hf(lo, hi);
#else
  return b200_pack_bf(lo, hi);
#endif
}
// columns t and t + 1 of a row (t even): one 8- or 4-byte store where the row's address allows it
__device__ __forceinline__ void b200_ar_put(unsigned long long p, unsigned int t, float x, float y) {
  if (!p) return;
  float* d = (float*)p + t;
  if (B200_T % 2 == 0 && (p & 7ull) == 0ull) {
    if (t < B200_T) *(b200_f2*)d = b200_f2{x, y};
  } else {
    if (t < B200_T) d[0] = x;
    if (t + 1u < B200_T) d[1] = y;
  }
}
__device__ __forceinline__ void b200_ar_put16(unsigned long long p, unsigned int t, unsigned int w) {
  if (!p) return;
  unsigned short* d = (unsigned short*)p + t;
  if (B200_T % 2 == 0 && (p & 3ull) == 0ull) {
    if (t < B200_T) *(unsigned int*)d = w;
  } else {
    if (t < B200_T) d[0] = (unsigned short)w;
    if (t + 1u < B200_T) d[1] = (unsigned short)(w >> 16);
  }
}

// the rows of one (batch, head) on their way into shared memory, one group of copies
__device__ __forceinline__ void b200_ar_fetch(unsigned short* to, const unsigned short* from, long long row) {
  constexpr unsigned int P = B200_E / 8;   // 16-byte pieces per row
  const unsigned int at = (unsigned int)__cvta_generic_to_shared(to);
  for (unsigned int i = threadIdx.x; i < B200_TP * P; i += 32u * B200_WARPS) {
    const unsigned int t = i / P, piece = i % P;
    const bool in = t < B200_T;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 :: "r"(at + 2u * (t * B200_LD + 8u * piece)), "l"(__cvta_generic_to_global(from + (in ? (long long)t * row + 8u * piece : 0ll))), "r"(in ? 16u : 0u) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
// the warps that share 16 queries
__device__ __forceinline__ void b200_ar_meet(unsigned int qt) {
  if (B200_KS > 1) asm volatile("bar.sync %0, %1;" ::"r"(1u + qt), "n"(32 * B200_KS) : "memory");
}
// all of the block's warps, wherever they are in the kernel
__device__ __forceinline__ void b200_ar_barrier() { asm volatile("bar.sync 0;" ::: "memory"); }

// the weights of one key tile of the thread's two rows, as rounded pairs
template <bool FAST>
__device__ __forceinline__ void b200_ar_weight4(const b200_attn_row* row, unsigned int t, const float4& x, const float* sum, const b200_divisor* dv,
                                                unsigned int* w B200_ATTN_PARAMS) {
  const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float a = t < B200_T ? b200_ar_weight<FAST>(row[r], t, v[2 * r], sum[r], dv[r] B200_ATTN_ARGS) : 0.0f;
    const float b = t + 1u < B200_T ? b200_ar_weight<FAST>(row[r], t + 1u, v[2 * r + 1], sum[r], dv[r] B200_ATTN_ARGS) : 0.0f;
    w[r] = b200_ar_pack(a, b);
  }
}

extern "C" __global__ void __launch_bounds__(32 * B200_WARPS)
B200_AR_NAME(const unsigned short* __restrict__ b200_qp, const unsigned short* __restrict__ b200_kp, const unsigned short* __restrict__ b200_vp,
             const b200_ar_shape shape B200_ATTN_PARAMS) {
  extern __shared__ __align__(16) unsigned char b200_dyn_smem[];
  unsigned short* const ks = (unsigned short*)b200_dyn_smem;
  unsigned short* const vs = ks + B200_TP * B200_LD;
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, c = lane & 3u;
  // (last tiles first: under a causal mask they look at the most keys)
  const unsigned int heads = shape.B0 * shape.B1;
  const unsigned int tile = shape.tiles - 1u - blockIdx.x / heads, bh = blockIdx.x % heads;
  const unsigned int b0 = bh / shape.B1, b1 = bh - b0 * shape.B1;

  // keys and values into shared memory, 16 bytes at a time, all of them under way at once (through registers
  // they came in several round trips to memory, a third of the kernel's time with few warps); rows beyond T zero
  b200_ar_fetch(ks, b200_kp + (long long)b0 * shape.k_b0 + (long long)b1 * shape.k_b1, shape.k_row);
  b200_ar_fetch(vs, b200_vp + (long long)b0 * shape.v_b0 + (long long)b1 * shape.v_b1, shape.v_row);
  const unsigned int qt = warp / B200_KS, part = warp % B200_KS;   // the queries and the share of the keys this warp looks at
  const unsigned int s0 = (tile * B200_QT + qt) * 16u;
  b200_attn_row row[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    row[r].b0 = b0;
    row[r].b1 = b1;
    row[r].s = s0 + g + 8u * r;
    row[r].ok = row[r].s < shape.S;
  }
  // query fragments straight from global memory (rows beyond S: zero)
  unsigned int qa[B200_E / 16][4];
  {
    const unsigned short* const qb = b200_qp + (long long)b0 * shape.q_b0 + (long long)b1 * shape.q_b1;
#pragma unroll
    for (unsigned int k = 0; k < B200_E / 16; ++k)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const unsigned short* const qr = qb + (long long)row[r].s * shape.q_row + 16u * k + 2u * c;
        qa[k][r] = row[r].ok ? *(const unsigned int*)qr : 0u;
        qa[k][2 + r] = row[r].ok ? *(const unsigned int*)(qr + 8) : 0u;
      }
  }
  // mask bits: word k of a row covers keys 32 k .. 32 k + 31
  const unsigned int* cp[2][B200_NCOND > 0 ? B200_NCOND : 1];
#if B200_NCOND > 0
  b200_ar_cond_rows(row[0], cp[0] B200_ATTN_ARGS);
  b200_ar_cond_rows(row[1], cp[1] B200_ATTN_ARGS);
#endif
  // bit j: no row of the warp has a mask bit among keys 16 j .. 16 j + 15
  unsigned int skip = 0u;
#if B200_MASKED
  {
    unsigned int any = 0u;
#pragma unroll
    for (unsigned int k = 0; k < (B200_NP + 1) / 2; ++k) {
      const unsigned int m = (cp[0][0] ? cp[0][0][k] : 0u) | (cp[1][0] ? cp[1][0][k] : 0u);
      any |= (m & 0xFFFFu ? 1u << (2u * k) : 0u) | (m >> 16 ? 2u << (2u * k) : 0u);
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) any |= __shfl_xor_sync(0xffffffffu, any, o);
    skip = ~any & ((1u << B200_NP) - 1u);
  }
#endif
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  b200_ar_barrier();
  if (s0 >= shape.S) {   // no queries for this warp: it only brought its part of the keys and values
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    b200_ar_barrier();
    return;
  }
  b200_ar_ptrs p[2];
  b200_ar_rows(row[0], p[0] B200_ATTN_ARGS);
  b200_ar_rows(row[1], p[1] B200_ATTN_ARGS);

  // this thread's scores: float4 n * 32 holds key tile n of rows g (x, y) and g + 8 (z, w)
  float4* const xs = (float4*)(vs + B200_TP * B200_LD) + qt * (B200_NT * 32u) + lane;
  // where the warps that share queries meet: row maxima and sums, partial outputs
  float* const meet = (float*)(vs + B200_TP * B200_LD) + (B200_QT * B200_NT * 128u + qt * (B200_KS * (32u + 16u * B200_E)));
  (void)meet;

  // ---- scores and row maximum
  float mx[2] = {b200_ar_max_init(), b200_ar_max_init()};
  const unsigned int k_at = (unsigned int)__cvta_generic_to_shared(ks), v_at = (unsigned int)__cvta_generic_to_shared(vs);
#pragma unroll 2
  for (unsigned int j = part; j < B200_NP; j += B200_KS) {
    if (B200_MASKED && ((skip >> j) & 1u)) {
#if B200_KEEP_SCORES
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < 2; ++r) b200_ar_put(p[r].scores, 16u * j + 8u * h + 2u * c, b200_ar_masked_score(), b200_ar_masked_score());
#endif
      continue;
    }
    unsigned int cw[2][2] = {{0u, 0u}, {0u, 0u}};
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int i = 0; i < B200_NCOND; ++i) cw[r][i] = cp[r][i] ? cp[r][i][j >> 1] >> (16u * (j & 1u)) : 0u;
    float d[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
    // an x4 load: eight keys, head dimensions 32 k2 .. 32 k2 + 31 (two k steps); an odd last step loads 16 twice
#pragma unroll
    for (unsigned int k2 = 0; k2 < (B200_E + 31) / 32; ++k2)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        unsigned int b[4];
        const unsigned int col = 32u * k2 + 8u * (lane >> 3);
        b200_ldsm4(b, k_at + 2u * ((16u * j + 8u * h + (lane & 7u)) * B200_LD + (col < B200_E ? col : col - 16u)));
        b200_ar_mma(d[h], qa[2 * k2], b[0], b[1]);
        if (2 * k2 + 1 < B200_E / 16) b200_ar_mma(d[h], qa[2 * k2 + 1 < B200_E / 16 ? 2 * k2 + 1 : 0], b[2], b[3]);
      }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = i >> 1;
        const unsigned int in = 8u * h + 2u * c + (i & 1), t = 16u * j + in;
        x[i] = t < B200_T ? b200_ar_score(row[r], t, d[h][i], (cw[r][0] >> in) & 1u, (cw[r][1] >> in) & 1u B200_ATTN_ARGS) : b200_ar_max_init();
        mx[r] = fmaxf(mx[r], x[i]);
      }
      xs[32u * (2u * j + h)] = make_float4(x[0], x[1], x[2], x[3]);
#if B200_KEEP_SCORES
      b200_ar_put(p[0].scores, 16u * j + 8u * h + 2u * c, x[0], x[1]);
      b200_ar_put(p[1].scores, 16u * j + 8u * h + 2u * c, x[2], x[3]);
#endif
    }
  }
  float sum[2] = {0.0f, 0.0f}, em[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    if (B200_MASKED && skip) mx[r] = fmaxf(mx[r], b200_ar_masked_score());
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
    if (B200_KS > 1 && c == 0u) meet[32u * part + g + 8u * r] = mx[r];
  }
  b200_ar_meet(qt);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
#pragma unroll
    for (unsigned int i = 0; i < B200_KS && B200_KS > 1; ++i) mx[r] = fmaxf(mx[r], meet[32u * i + g + 8u * r]);
    mx[r] = b200_ar_row_max(row[r], mx[r] B200_ATTN_ARGS);
    if (part == 0u && c == 0u && p[r].mx) *(float*)p[r].mx = mx[r];
    em[r] = B200_MASKED ? b200_ar_exp(row[r], 0u, b200_ar_masked_score(), mx[r] B200_ATTN_ARGS) : 0.0f;
  }
  // ---- exponentials and row sum
#pragma unroll 2
  for (unsigned int j = part; j < B200_NP; j += B200_KS) {
    const bool off = B200_MASKED && ((skip >> j) & 1u);
#if !B200_KEEP_EXP
    if (off && em[0] == 0.0f && em[1] == 0.0f) continue;
#endif
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned int t = 16u * j + 8u * h + 2u * c;
      float x[4] = {em[0], em[0], em[1], em[1]};
      if (!off) {
        const float4 v = xs[32u * (2u * j + h)];
        x[0] = b200_ar_exp(row[0], t, v.x, mx[0] B200_ATTN_ARGS);
        x[1] = b200_ar_exp(row[0], t + 1u, v.y, mx[0] B200_ATTN_ARGS);
        x[2] = b200_ar_exp(row[1], t, v.z, mx[1] B200_ATTN_ARGS);
        x[3] = b200_ar_exp(row[1], t + 1u, v.w, mx[1] B200_ATTN_ARGS);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (t + (i & 1) >= B200_T) x[i] = 0.0f;
        sum[i >> 1] += x[i];
      }
      if (!off) xs[32u * (2u * j + h)] = make_float4(x[0], x[1], x[2], x[3]);
#if B200_KEEP_EXP
      b200_ar_put(p[0].exps, t, x[0], x[1]);
      b200_ar_put(p[1].exps, t, x[2], x[3]);
#endif
    }
  }
  b200_divisor dv[2];
  unsigned int wm[2];
  float wz[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
    if (B200_KS > 1 && c == 0u) meet[32u * part + 16u + g + 8u * r] = sum[r];
  }
  b200_ar_meet(qt);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    if (B200_KS > 1) sum[r] = meet[16u + g + 8u * r];
#pragma unroll
    for (unsigned int i = 1; i < B200_KS; ++i) sum[r] += meet[32u * i + 16u + g + 8u * r];
    sum[r] = b200_ar_row_sum(row[r], sum[r] B200_ATTN_ARGS);
    if (part == 0u && c == 0u && p[r].sum) *(float*)p[r].sum = sum[r];
    dv[r] = b200_divisor_of(b200_ar_divisor(row[r], sum[r] B200_ATTN_ARGS));
    wz[r] = B200_MASKED ? b200_ar_weight<false>(row[r], 0u, em[r], sum[r], dv[r] B200_ATTN_ARGS) : 0.0f;
    wm[r] = b200_ar_pack(wz[r], wz[r]);
  }
  // ---- weights, the A fragments of the second product, and the product; masked keys that weigh nothing in any
  // row of the warp are left out of it
  const bool fast = __all_sync(0xffffffffu, dv[0].fast && dv[1].fast);
  const bool leave = !__any_sync(0xffffffffu, wz[0] != 0.0f || wz[1] != 0.0f);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  b200_ar_barrier();
  float o[B200_E / 8][4];
#pragma unroll
  for (unsigned int e = 0; e < B200_E / 8; ++e)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[e][i] = 0.0f;
#pragma unroll 2
  for (unsigned int j = part; j < B200_NP; j += B200_KS) {
    const bool off = B200_MASKED && ((skip >> j) & 1u);
#if !B200_KEEP_W
    if (off && leave) continue;
#endif
    // (masked keys that end beyond the row: the values beyond T are zero rows, so the weights there do not matter)
    unsigned int a[4] = {wm[0], wm[1], wm[0], wm[1]};
    if (!off) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const unsigned int t = 16u * j + 8u * h + 2u * c;
        const float4 x = xs[32u * (2u * j + h)];
        if (fast) b200_ar_weight4<true>(row, t, x, sum, dv, a + 2 * h B200_ATTN_ARGS);
        else b200_ar_weight4<false>(row, t, x, sum, dv, a + 2 * h B200_ATTN_ARGS);
      }
    }
#if B200_KEEP_W
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int r = 0; r < 2; ++r) b200_ar_put16(p[r].w, 16u * j + 8u * h + 2u * c, a[2 * h + r]);
    if (off && leave) continue;
#endif
#pragma unroll
    for (unsigned int e = 0; e < B200_E / 8; e += 2) {
      // keys 16 j .. 16 j + 15, head dimensions 8 e .. 8 e + 15
      unsigned int b[4];
      b200_ldsm4t(b, v_at + 2u * ((16u * j + (lane & 15u)) * B200_LD + 8u * e + 8u * (lane >> 4)));
      b200_ar_mma(o[e], a, b[0], b[1]);
      b200_ar_mma(o[e + 1], a, b[2], b[3]);
    }
  }
  // the warps' partial outputs, as [part][tile of 8 columns][value][lane]; each warp finishes some of the tiles
  if (B200_KS > 1) {
    float* const mine = meet + 32u * B200_KS + part * (16u * B200_E) + lane;
#pragma unroll
    for (unsigned int e = 0; e < B200_E / 8; ++e)
#pragma unroll
      for (int i = 0; i < 4; ++i) mine[(4u * e + i) * 32u] = o[e][i];
    b200_ar_meet(qt);
  }
#pragma unroll
  for (unsigned int e0 = 0; e0 < B200_E / 8; e0 += B200_KS) {
    const unsigned int e = e0 + part;
    if (e >= B200_E / 8) break;
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (B200_KS > 1) {
        const float* const at = meet + 32u * B200_KS + (4u * e + i) * 32u + lane;
        v[i] = at[0];
#pragma unroll
        for (unsigned int k = 1; k < B200_KS; ++k) v[i] += at[k * (16u * B200_E)];
      } else {
        v[i] = o[e0][i];
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (!p[r].out) continue;
      const unsigned int col = 8u * e + 2u * c;
      B200_OUT_T* const d = (B200_OUT_T*)p[r].out + col;
      const B200_OUT_T v0 = b200_ar_out(row[r], col, v[2 * r] B200_ATTN_ARGS), v1 = b200_ar_out(row[r], col + 1u, v[2 * r + 1] B200_ATTN_ARGS);
      if (sizeof(B200_OUT_T) == 2 && ((unsigned long long)d & 3ull) == 0ull) *(unsigned int*)d = (unsigned int)v0 | ((unsigned int)v1 << 16);
      else { d[0] = v0; d[1] = v1; }
    }
  }
}

#endif  // B200_ATTN_ROWS_CUH
