// Fused attention stage for short rows: the chain of attn_sm100.cuh (scores, softmax, weights . values) for
// any number of keys up to 256 and any head dimension that is a multiple of 16.
//
// A warp takes 16 queries of one (batch, head) and keeps their whole score rows in registers, in the
// accumulator layout of mma.m16n8k16: thread (g, c) = (lane / 4, lane % 4) holds columns 8 n + 2 c and + 1 of
// rows g and g + 8 for every key tile n.  Row maximum and sum are two shuffles within four lanes; the
// weights, rounded to the node's 16-bit format, are at once the A fragments of the second product, whose B
// fragments come transposed out of shared memory (ldmatrix.trans).  Keys and values of the (batch, head) lie
// in shared memory, rows padded by 16 bytes so that the eight rows of an ldmatrix fall into different banks.
// What bounds it: the softmax arithmetic, about 25 instructions per score; with 16 rows per warp there is
// neither a tensor-memory round trip nor a block-wide barrier between its passes, and a sequence of 100
// positions is 7 warps' work where the tile kernels pad it to 128 x 128.  (Before, such rows took four
// launches: scores, softmax, a gathered copy of the weights, weights . values.)
//
// Key tiles in which no query of the warp has a mask bit set are not multiplied, and their scores are one
// constant per row: exponential and weight are evaluated once for all of them, and when that weight is zero
// (it is, unless a row is masked throughout) the tile adds nothing to the output either.  A causal mask
// halves the work this way.
//
// The translation unit defines B200_AR_NAME, B200_T, B200_E, B200_HALF (1: half, 0: bfloat16), B200_WARPS,
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
#define B200_CW ((B200_T + 31) / 32)              // mask words per row

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

// softmax passes behind the row maximum, on the score fragments `x`; `skip`: bit n set when tile n is masked throughout
template <bool FAST>
__device__ __forceinline__ void b200_ar_weights(const b200_attn_row* row, const b200_ar_ptrs* p, unsigned int c, float (*x)[4], unsigned int skip,
                                                const float* sum, const b200_divisor* dv, const unsigned int* wm, unsigned int (*w)[2] B200_ATTN_PARAMS) {
#pragma unroll
  for (unsigned int n = 0; n < B200_NT; ++n) {
    const unsigned int t = 8u * n + 2u * c;
    if (B200_MASKED && ((skip >> n) & 1u)) {
      w[n][0] = wm[0];
      w[n][1] = wm[1];
    } else {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float a = t < B200_T ? b200_ar_weight<FAST>(row[r], t, x[n][2 * r], sum[r], dv[r] B200_ATTN_ARGS) : 0.0f;
        const float b = t + 1u < B200_T ? b200_ar_weight<FAST>(row[r], t + 1u, x[n][2 * r + 1], sum[r], dv[r] B200_ATTN_ARGS) : 0.0f;
        w[n][r] = b200_ar_pack(a, b);
      }
    }
    // (a masked tile that ends beyond the row keeps zeros there: the values beyond T are zero rows, so its weights do not matter)
#if B200_KEEP_W
    b200_ar_put16(p[0].w, t, w[n][0]);
    b200_ar_put16(p[1].w, t, w[n][1]);
#endif
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
  const unsigned int tile = blockIdx.x % shape.tiles, bh = blockIdx.x / shape.tiles;
  const unsigned int b0 = bh / shape.B1, b1 = bh - b0 * shape.B1;

  // keys and values into shared memory, 16 bytes at a time; rows beyond T are zero
  {
    const unsigned short* const kb = b200_kp + (long long)b0 * shape.k_b0 + (long long)b1 * shape.k_b1;
    const unsigned short* const vb = b200_vp + (long long)b0 * shape.v_b0 + (long long)b1 * shape.v_b1;
    constexpr unsigned int P = B200_E / 8;   // 16-byte pieces per row
#pragma unroll 4
    for (unsigned int i = threadIdx.x; i < B200_TP * P; i += 32u * B200_WARPS) {
      const unsigned int t = i / P, piece = i % P;
      uint4 kq = make_uint4(0u, 0u, 0u, 0u), vq = kq;
      if (t < B200_T) {
        kq = *(const uint4*)(kb + (long long)t * shape.k_row + 8u * piece);
        vq = *(const uint4*)(vb + (long long)t * shape.v_row + 8u * piece);
      }
      *(uint4*)(ks + t * B200_LD + 8u * piece) = kq;
      *(uint4*)(vs + t * B200_LD + 8u * piece) = vq;
    }
  }
  const unsigned int s0 = (tile * B200_WARPS + warp) * 16u;
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
  unsigned int cw[2][B200_NCOND > 0 ? B200_NCOND : 1][B200_CW];
#if B200_NCOND > 0
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const unsigned int* cp[B200_NCOND];
    b200_ar_cond_rows(row[r], cp B200_ATTN_ARGS);
#pragma unroll
    for (int i = 0; i < B200_NCOND; ++i)
#pragma unroll
      for (int k = 0; k < B200_CW; ++k) cw[r][i][k] = cp[i] ? cp[i][k] : 0u;
  }
#endif
  __syncthreads();
  if (s0 >= shape.S) return;   // (no barrier follows)
  b200_ar_ptrs p[2];
  b200_ar_rows(row[0], p[0] B200_ATTN_ARGS);
  b200_ar_rows(row[1], p[1] B200_ATTN_ARGS);

  // tiles without a mask bit in any of the warp's rows
  unsigned int skip = 0u;
#if B200_MASKED
  {
    unsigned int any = 0u;   // bit n: some row of this thread has a bit in tile n
#pragma unroll
    for (int k = 0; k < B200_CW; ++k) {
      const unsigned int m = cw[0][0][k] | cw[1][0][k];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (4 * k + q < B200_NT && ((m >> (8 * q)) & 0xFFu)) any |= 1u << (4 * k + q);
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) any |= __shfl_xor_sync(0xffffffffu, any, o);
    skip = ~any;
  }
#endif

  // ---- scores and row maximum
  float x[B200_NT][4];
  float mx[2] = {b200_ar_max_init(), b200_ar_max_init()};
  const unsigned int k_at = (unsigned int)__cvta_generic_to_shared(ks), v_at = (unsigned int)__cvta_generic_to_shared(vs);
#pragma unroll
  for (unsigned int n = 0; n < B200_NT; ++n) {
    const bool off = B200_MASKED && ((skip >> n) & 1u);
    if (!off) {
      float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      // an x4 load: keys 8 n .. 8 n + 7, head dimensions 32 k2 .. 32 k2 + 31 (two k steps); an odd last step loads 16 twice
#pragma unroll
      for (unsigned int k2 = 0; k2 < (B200_E + 31) / 32; ++k2) {
        unsigned int b[4];
        const unsigned int col = 32u * k2 + 8u * (lane >> 3);
        b200_ldsm4(b, k_at + 2u * ((8u * n + (lane & 7u)) * B200_LD + (col < B200_E ? col : col - 16u)));
        b200_ar_mma(d, qa[2 * k2], b[0], b[1]);
        if (2 * k2 + 1 < B200_E / 16) b200_ar_mma(d, qa[2 * k2 + 1 < B200_E / 16 ? 2 * k2 + 1 : 0], b[2], b[3]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = i >> 1;
        const unsigned int t = 8u * n + 2u * c + (i & 1);
        const unsigned int cb0 = B200_NCOND > 0 ? (cw[r][0][n / 4] >> (t & 31u)) & 1u : 0u;
        const unsigned int cb1 = B200_NCOND > 1 ? (cw[r][B200_NCOND > 1 ? 1 : 0][n / 4] >> (t & 31u)) & 1u : 0u;
        x[n][i] = t < B200_T ? b200_ar_score(row[r], t, d[i], cb0, cb1 B200_ATTN_ARGS) : b200_ar_max_init();
        mx[r] = fmaxf(mx[r], x[n][i]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) x[n][i] = b200_ar_masked_score();
      if (8u * n < B200_T) {
        mx[0] = fmaxf(mx[0], b200_ar_masked_score());
        mx[1] = fmaxf(mx[1], b200_ar_masked_score());
      }
    }
#if B200_KEEP_SCORES
    b200_ar_put(p[0].scores, 8u * n + 2u * c, x[n][0], x[n][1]);
    b200_ar_put(p[1].scores, 8u * n + 2u * c, x[n][2], x[n][3]);
#endif
  }
  float sum[2] = {0.0f, 0.0f}, em[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
    mx[r] = b200_ar_row_max(row[r], mx[r] B200_ATTN_ARGS);
    if (c == 0u && p[r].mx) *(float*)p[r].mx = mx[r];
    em[r] = B200_MASKED ? b200_ar_exp(row[r], 0u, b200_ar_masked_score(), mx[r] B200_ATTN_ARGS) : 0.0f;
  }
  // ---- exponentials and row sum
#pragma unroll
  for (unsigned int n = 0; n < B200_NT; ++n) {
    if (B200_MASKED && ((skip >> n) & 1u)) {
#pragma unroll
      for (int i = 0; i < 4; ++i) x[n][i] = em[i >> 1];
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) x[n][i] = b200_ar_exp(row[i >> 1], 8u * n + 2u * c + (i & 1), x[n][i], mx[i >> 1] B200_ATTN_ARGS);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (8u * n + 7u >= B200_T && 8u * n + 2u * c + (i & 1) >= B200_T) x[n][i] = 0.0f;
      sum[i >> 1] += x[n][i];
    }
#if B200_KEEP_EXP
    b200_ar_put(p[0].exps, 8u * n + 2u * c, x[n][0], x[n][1]);
    b200_ar_put(p[1].exps, 8u * n + 2u * c, x[n][2], x[n][3]);
#endif
  }
  b200_divisor dv[2];
  unsigned int wm[2];
  float wz[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
    sum[r] = b200_ar_row_sum(row[r], sum[r] B200_ATTN_ARGS);
    if (c == 0u && p[r].sum) *(float*)p[r].sum = sum[r];
    dv[r] = b200_divisor_of(b200_ar_divisor(row[r], sum[r] B200_ATTN_ARGS));
    wz[r] = B200_MASKED ? b200_ar_weight<false>(row[r], 0u, em[r], sum[r], dv[r] B200_ATTN_ARGS) : 0.0f;
    wm[r] = b200_ar_pack(wz[r], wz[r]);
  }
  // ---- weights: the A fragments of the second product
  unsigned int w[B200_NT][2];
  if (__all_sync(0xffffffffu, dv[0].fast && dv[1].fast)) b200_ar_weights<true>(row, p, c, x, skip, sum, dv, wm, w B200_ATTN_ARGS);
  else b200_ar_weights<false>(row, p, c, x, skip, sum, dv, wm, w B200_ATTN_ARGS);
  // masked tiles that weigh nothing in any row of the warp are left out of the product
  const unsigned int leave = __any_sync(0xffffffffu, wz[0] != 0.0f || wz[1] != 0.0f) ? 0u : skip;
  float o[B200_E / 8][4];
#pragma unroll
  for (unsigned int e = 0; e < B200_E / 8; ++e)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[e][i] = 0.0f;
#pragma unroll
  for (unsigned int k = 0; k < B200_NT / 2; ++k) {
    if (((leave >> (2u * k)) & 3u) == 3u) continue;
    const unsigned int a[4] = {w[2 * k][0], w[2 * k][1], w[2 * k + 1][0], w[2 * k + 1][1]};
#pragma unroll
    for (unsigned int e = 0; e < B200_E / 8; e += 2) {
      // keys 16 k .. 16 k + 15, head dimensions 8 e .. 8 e + 15
      unsigned int b[4];
      b200_ldsm4t(b, v_at + 2u * ((16u * k + (lane & 15u)) * B200_LD + 8u * e + 8u * (lane >> 4)));
      b200_ar_mma(o[e], a, b[0], b[1]);
      b200_ar_mma(o[e + 1], a, b[2], b[3]);
    }
  }
#pragma unroll
  for (unsigned int e = 0; e < B200_E / 8; ++e)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (!p[r].out) continue;
      const unsigned int col = 8u * e + 2u * c;
      B200_OUT_T* const d = (B200_OUT_T*)p[r].out + col;
      const B200_OUT_T v0 = b200_ar_out(row[r], col, o[e][2 * r] B200_ATTN_ARGS), v1 = b200_ar_out(row[r], col + 1u, o[e][2 * r + 1] B200_ATTN_ARGS);
      if (sizeof(B200_OUT_T) == 2 && ((unsigned long long)d & 3ull) == 0ull) *(unsigned int*)d = (unsigned int)v0 | ((unsigned int)v1 << 16);
      else { d[0] = v0; d[1] = v1; }
    }
}

#endif  // B200_ATTN_ROWS_CUH
