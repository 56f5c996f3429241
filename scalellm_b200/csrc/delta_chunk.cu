// delta_chunk.cu — the gated delta rule of delta_rule.cu over prompt portions, 16 tokens at a time on the tensor cores
// (key and value sizes 128).  With d the decays and, inside a chunk, D(s, t] = prod_{s < r <= t} diag(d_r):
//
//     u_t = b_t (v_t - (D(0, t] k_t)^T S - sum_{s < t} A[t, s] u_s)         A[t, s] = k_t^T D(s, t] k_s
//     o_t = (D(0, t] q_t)^T S + sum_{s <= t} B[t, s] u_s                     B[t, s] = q_t^T D(s, t] k_s
//     S  <- D(0, 16] S + sum_s (D(s, 16] k_s) u_s^T
//
// so  U = T (V - Kbar S),  O = Qbar S + B U,  S <- D S + Khat^T U  with  T = (I + diag(b) A)^{-1} diag(b).
//
//   chunks : every chunk and head in parallel: the products of decays as they are (never a quotient: no decay is too strong),
//            A, B and T in fp32; leaves Kbar, Qbar, Khat, T, B as two bf16 terms each, laid out as the scan reads them
//   scan   : per (sequence, head, 16 x NW value columns) a CTA of NW warps walks the chunks.  A warp keeps S^T of its 16
//            columns in accumulators — their layout is the A operand's in S^T Kbar^T, so the state never goes through
//            memory — and a producer warp streams the chunks' 27 KB by bulk copies, three in flight.
//
// Every product takes three terms (high x high, high x low, low x high): 16 bits of both factors, fp32 sums.
// Bound by the chain of a chunk (state -> U -> state), 3.2 us for 16 tokens at eight warps an SM.  8 prompts of up to 1 024
// tokens, 16 heads: chunks 85 us, scan 207 us, norm and gate 22 us (the token-by-token walk: 1 613 us and 36 us); 64 x 32
// tokens, whole layer: 223 us against 348; 1 x 16 tokens 40 us against 57.
#include "common.cuh"
#include "guard.cuh"

namespace b200 {
namespace {

constexpr int DC_T = 16, DC_D = 128;
constexpr int DC_MAT = DC_T * DC_D * 2;                 // one [16 x 128] bf16 term, rows of 256 bytes, 16-byte pieces swizzled
constexpr int DC_KB = 0, DC_QB = 2 * DC_MAT, DC_KH = 4 * DC_MAT, DC_TT = 6 * DC_MAT, DC_BB = DC_TT + 1024,
              DC_DEC = DC_BB + 1024, DC_UNIT = DC_DEC + DC_D * 4;                                // (low terms follow the high)
constexpr int DC_STAGES = 3;

__device__ __forceinline__ uint32_t dc_mat_off(int row, int piece) { return row * 256 + ((piece ^ (row & 7)) << 4); }
__device__ __forceinline__ void dc_split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = Num<__nv_bfloat16>::pack(x, y);
  const float2 h = Num<__nv_bfloat16>::unpack(hi);
  lo = Num<__nv_bfloat16>::pack(x - h.x, y - h.y);
}
// first chunk of a sequence in the step's list (every sequence's chunks fit before the next one's first)
__device__ __forceinline__ int64_t dc_first(int seq_row0, int seq) { return seq_row0 / DC_T + seq; }

// One unit = (chunk, head): two warps, two channels a lane.
__global__ void __launch_bounds__(64)
delta_chunks_kernel(uint8_t* __restrict__ units, const float* __restrict__ q, const float* __restrict__ k,
                    const float* __restrict__ decay, const float* __restrict__ beta, const int* __restrict__ q_cu, int H,
                    int G) {
  __shared__ float red[2][256];
  __shared__ float Am[DC_T][DC_T + 1], Bm[DC_T][DC_T + 1];
  const int h = blockIdx.x, seq = blockIdx.z, c = blockIdx.y;
  const int row0 = q_cu[seq], len = q_cu[seq + 1] - row0;
  if (c * DC_T >= len) return;
  const int n = min(DC_T, len - c * DC_T), t0 = row0 + c * DC_T;
  uint8_t* unit = units + ((dc_first(row0, seq) + c) * H + h) * DC_UNIT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ch = warp * 64 + 2 * lane, g = h / (H / G);
  float2 kk[DC_T], qq[DC_T], dd[DC_T];
#pragma unroll
  for (int t = 0; t < DC_T; ++t) {
    kk[t] = qq[t] = make_float2(0.0f, 0.0f);
    dd[t] = make_float2(1.0f, 1.0f);
    if (t < n) {
      kk[t] = *reinterpret_cast<const float2*>(k + ((int64_t)(t0 + t) * G + g) * DC_D + ch);
      qq[t] = *reinterpret_cast<const float2*>(q + ((int64_t)(t0 + t) * G + g) * DC_D + ch);
      dd[t] = *reinterpret_cast<const float2*>(decay + ((int64_t)(t0 + t) * H + h) * DC_D + ch);
    }
  }
  // A below the diagonal and B up to it: 256 sums over the channels, 32 at a time; after five halving exchanges lane l
  // holds sum l of the group
  {
    float buf[32];
    int idx = 0, group = 0;
    auto push = [&](float v) {
      buf[idx & 31] = v;
      if ((++idx & 31) == 0) {
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
          const bool up = (lane & w) != 0;
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (i < w) {
              const float give = up ? buf[i] : buf[i + w], keep = up ? buf[i + w] : buf[i];
              buf[i] = keep + __shfl_xor_sync(0xffffffffu, give, w);
            }
        }
        red[warp][group * 32 + lane] = buf[0];
        ++group;
      }
    };
#pragma unroll
    for (int s = 0; s < DC_T; ++s) {
      float2 p = kk[s];
      push(p.x * qq[s].x + p.y * qq[s].y);                                   // B[s, s]
#pragma unroll
      for (int t = s + 1; t < DC_T; ++t) {
        p.x *= dd[t].x;
        p.y *= dd[t].y;
        push(p.x * kk[t].x + p.y * kk[t].y);                                 // A[t, s]
        push(p.x * qq[t].x + p.y * qq[t].y);                                 // B[t, s]
      }
    }
  }
  // scaled keys and queries, as two terms
  {
    const int piece = ch >> 3, in = (lane & 3) * 4;
    float2 p = make_float2(1.0f, 1.0f);
#pragma unroll
    for (int t = 0; t < DC_T; ++t) {
      p.x *= dd[t].x;
      p.y *= dd[t].y;
      uint32_t hi, lo;
      const uint32_t o = dc_mat_off(t, piece) + in;
      dc_split2(p.x * kk[t].x, p.y * kk[t].y, hi, lo);
      *reinterpret_cast<uint32_t*>(unit + DC_KB + o) = hi;
      *reinterpret_cast<uint32_t*>(unit + DC_KB + DC_MAT + o) = lo;
      dc_split2(p.x * qq[t].x, p.y * qq[t].y, hi, lo);
      *reinterpret_cast<uint32_t*>(unit + DC_QB + o) = hi;
      *reinterpret_cast<uint32_t*>(unit + DC_QB + DC_MAT + o) = lo;
    }
    *reinterpret_cast<float2*>(unit + DC_DEC + ch * 4) = p;
    p = make_float2(1.0f, 1.0f);
#pragma unroll
    for (int t = DC_T - 1; t >= 0; --t) {
      uint32_t hi, lo;
      const uint32_t o = dc_mat_off(t, piece) + in;
      dc_split2(p.x * kk[t].x, p.y * kk[t].y, hi, lo);
      *reinterpret_cast<uint32_t*>(unit + DC_KH + o) = hi;
      *reinterpret_cast<uint32_t*>(unit + DC_KH + DC_MAT + o) = lo;
      p.x *= dd[t].x;
      p.y *= dd[t].y;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += 64) {
    // sum i belongs to column s = the run of 31 - 2 s sums it lies in: [B(s, s), A(s + 1, s), B(s + 1, s), ...]
    int s = 0, rest = i;
    while (rest >= 31 - 2 * s) {
      rest -= 31 - 2 * s;
      ++s;
    }
    const float v = red[0][i] + red[1][i];
    const int t = s + (rest + 1) / 2;
    if (rest & 1) Am[t][s] = v;
    else Bm[t][s] = v;
  }
  __syncthreads();
  // T by columns, forward; B's upper part is zero
  if (threadIdx.x < DC_T) {
    const int col = threadIdx.x;
    float x[DC_T];
#pragma unroll
    for (int t = 0; t < DC_T; ++t) {
      const float b = t < n ? beta[(int64_t)(t0 + t) * H + h] : 0.0f;
      float acc = t == col ? 1.0f : 0.0f;
#pragma unroll
      for (int s = 0; s < t; ++s) acc -= Am[t][s] * x[s];
      x[t] = b * acc;
    }
    __nv_bfloat16* th = reinterpret_cast<__nv_bfloat16*>(unit + DC_TT);
#pragma unroll
    for (int t = 0; t < DC_T; ++t) {
      const __nv_bfloat16 hi = __float2bfloat16_rn(x[t]);
      th[t * DC_T + col] = hi;
      th[256 + t * DC_T + col] = __float2bfloat16_rn(x[t] - __bfloat162float(hi));
    }
  } else if (threadIdx.x >= 32 && threadIdx.x < 32 + DC_T) {
    const int col = threadIdx.x - 32;
    __nv_bfloat16* bh = reinterpret_cast<__nv_bfloat16*>(unit + DC_BB);
#pragma unroll
    for (int t = 0; t < DC_T; ++t) {
      const float v = t >= col ? Bm[t][col] : 0.0f;
      const __nv_bfloat16 hi = __float2bfloat16_rn(v);
      bh[t * DC_T + col] = hi;
      bh[256 + t * DC_T + col] = __float2bfloat16_rn(v - __bfloat162float(hi));
    }
  }
}

__device__ __forceinline__ void dc_ldsm(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void dc_ldsm_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void dc_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two 8-column accumulator tiles -> the A operand of a 16-deep step, as two terms
__device__ __forceinline__ void dc_operand(const float (&x)[4], const float (&y)[4], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
  dc_split2(x[0], x[1], hi[0], lo[0]);
  dc_split2(x[2], x[3], hi[1], lo[1]);
  dc_split2(y[0], y[1], hi[2], lo[2]);
  dc_split2(y[2], y[3], hi[3], lo[3]);
}

template <int NW>
__global__ void __launch_bounds__((NW + 1) * 32)
delta_chunk_scan_kernel(float* __restrict__ raw, const uint8_t* __restrict__ units, const float* __restrict__ v,
                        float* __restrict__ state, const int* __restrict__ q_cu, const int* __restrict__ positions,
                        const int* __restrict__ state_slots, int H) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t full[DC_STAGES], empty[DC_STAGES];
  __shared__ uint32_t dead_word;
  volatile uint32_t* dead = &dead_word;
  const int h = blockIdx.x, seq = blockIdx.y;
  const int row0 = q_cu[seq], len = q_cu[seq + 1] - row0;
  if (len <= 0) return;
  const int chunks = (len + DC_T - 1) / DC_T;
  const uint8_t* src = units + (dc_first(row0, seq) * H + h) * DC_UNIT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < DC_STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], NW);
    }
    *dead = 0u;
    fence_mbar_init();
  }
  __syncthreads();
  if (warp == NW) {
    if (lane == 0)
      for (int c = 0; c < chunks; ++c) {
        const int s = c % DC_STAGES;
        guard_wait(&empty[s], ((c / DC_STAGES) & 1) ^ 1, dead);
        mbar_arrive_expect_tx(&full[s], DC_UNIT);
        bulk_load_1d(smem + s * DC_UNIT, src + (int64_t)c * H * DC_UNIT, DC_UNIT, &full[s]);
      }
  } else {
    const int g = lane >> 2, t2 = (lane & 3) * 2;
    const int col = (blockIdx.z * NW + warp) * 16 + g;      // this lane's value columns: col, col + 8
    const int64_t nv = (int64_t)H * DC_D;
    float* Sg = state + ((int64_t)state_slots[seq] * H + h) * DC_D * DC_D;                     // [key][value]
    float S[16][4];                                         // S^T: rows col, col + 8; tile n: keys 8 n + t2, + 1
    const bool fresh = positions[row0] == 0;
#pragma unroll
    for (int n = 0; n < 16; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        S[n][e] = fresh ? 0.0f : Sg[(int64_t)(n * 8 + t2 + (e & 1)) * DC_D + col + (e >> 1) * 8];
    const float* vc = v + (int64_t)row0 * nv + (int64_t)h * DC_D + col;
    float* oc = raw + (int64_t)row0 * nv + (int64_t)h * DC_D + col;
    float vn[2][4];                                         // V^T of the next chunk, as an accumulator holds it
    auto load_v = [&](int c) {
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = c * DC_T + n * 8 + t2 + (e & 1);
          vn[n][e] = t < len ? vc[(int64_t)t * nv + (e >> 1) * 8] : 0.0f;
        }
    };
    load_v(0);
    // operand rows of this lane for ldmatrix: tokens as n (plain) and as k (transposed)
    const int rn = (lane & 7) + ((lane >> 4) & 1) * 8, pn = (lane >> 3) & 1;
    const int rk = (lane & 7) + ((lane >> 3) & 1) * 8, pk = lane >> 4;
    for (int c = 0; c < chunks; ++c) {
      const int s = c % DC_STAGES;
      const uint32_t base = smem_u32(smem + s * DC_UNIT);
      float w[2][4], wx[2][4], o[2][4], ox[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          w[n][e] = vn[n][e];
          wx[n][e] = o[n][e] = ox[n][e] = 0.0f;
        }
      if (c + 1 < chunks) load_v(c + 1);
      guard_wait(&full[s], (c / DC_STAGES) & 1, dead);
      // (the sign of Kbar S: the operands of U take V - Kbar S, so its sums start from -V and change sign after)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) w[n][e] = -w[n][e];
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        uint32_t ah[4], al[4], kh[4], kl[4], qh[4], ql[4];
        dc_operand(S[2 * kk], S[2 * kk + 1], ah, al);
        const uint32_t off = dc_mat_off(rn, kk * 2 + pn);
        dc_ldsm(kh, base + DC_KB + off);
        dc_ldsm(kl, base + DC_KB + DC_MAT + off);
        dc_ldsm(qh, base + DC_QB + off);
        dc_ldsm(ql, base + DC_QB + DC_MAT + off);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          dc_mma(w[n], ah, kh[2 * n], kh[2 * n + 1]);
          dc_mma(o[n], ah, qh[2 * n], qh[2 * n + 1]);
          dc_mma(wx[n], ah, kl[2 * n], kl[2 * n + 1]);
          dc_mma(ox[n], ah, ql[2 * n], ql[2 * n + 1]);
          dc_mma(wx[n], al, kh[2 * n], kh[2 * n + 1]);
          dc_mma(ox[n], al, qh[2 * n], qh[2 * n + 1]);
        }
      }
      float u[2][4], ux[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          w[n][e] = -(w[n][e] + wx[n][e]);
          u[n][e] = ux[n][e] = 0.0f;
        }
      {
        uint32_t xh[4], xl[4], th[4], tl[4];
        dc_operand(w[0], w[1], xh, xl);
        const uint32_t off = rn * 32 + pn * 16;
        dc_ldsm(th, base + DC_TT + off);
        dc_ldsm(tl, base + DC_TT + 512 + off);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          dc_mma(u[n], xh, th[2 * n], th[2 * n + 1]);
          dc_mma(ux[n], xh, tl[2 * n], tl[2 * n + 1]);
          dc_mma(ux[n], xl, th[2 * n], th[2 * n + 1]);
        }
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) u[n][e] += ux[n][e];
      uint32_t uh[4], ul[4];
      dc_operand(u[0], u[1], uh, ul);
      {
        uint32_t bh[4], bl[4];
        const uint32_t off = rn * 32 + pn * 16;
        dc_ldsm(bh, base + DC_BB + off);
        dc_ldsm(bl, base + DC_BB + 512 + off);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          dc_mma(o[n], uh, bh[2 * n], bh[2 * n + 1]);
          dc_mma(ox[n], uh, bl[2 * n], bl[2 * n + 1]);
          dc_mma(ox[n], ul, bh[2 * n], bh[2 * n + 1]);
        }
      }
#pragma unroll
      for (int np = 0; np < 8; ++np) {
        uint32_t kh[4], kl[4];
        const uint32_t off = dc_mat_off(rk, np * 2 + pk);
        dc_ldsm_t(kh, base + DC_KH + off);
        dc_ldsm_t(kl, base + DC_KH + DC_MAT + off);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float (&a)[4] = S[np * 2 + j];
          const float2 d = *reinterpret_cast<const float2*>(smem + s * DC_UNIT + DC_DEC + ((np * 2 + j) * 8 + t2) * 4);
          a[0] *= d.x; a[1] *= d.y; a[2] *= d.x; a[3] *= d.y;
          dc_mma(a, uh, kh[2 * j], kh[2 * j + 1]);
          dc_mma(a, uh, kl[2 * j], kl[2 * j + 1]);
          dc_mma(a, ul, kh[2 * j], kh[2 * j + 1]);
        }
      }
      const bool lost = *dead != 0u;
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = c * DC_T + n * 8 + t2 + (e & 1);
          if (t < len) oc[(int64_t)t * nv + (e >> 1) * 8] = lost ? NAN : o[n][e] + ox[n][e];
        }
    }
    const bool lost = *dead != 0u;
#pragma unroll
    for (int n = 0; n < 16; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        Sg[(int64_t)(n * 8 + t2 + (e & 1)) * DC_D + col + (e >> 1) * 8] = lost ? NAN : S[n][e];
  }
  if (threadIdx.x == NW * 32 && *dead) guard_drain();
  __syncthreads();
}

// out = raw / rms(raw) * nw * sigmoid(gate) per head of 128: a warp per (row, head), 16 bytes a lane
__global__ void __launch_bounds__(256)
delta_norm_gate_kernel(__nv_bfloat16* __restrict__ out, int64_t ldo, const float* __restrict__ raw,
                       const __nv_bfloat16* __restrict__ gate, int64_t ld_gate, const float* __restrict__ nw, int64_t n_units,
                       int H, float eps) {
  const int64_t u = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (u >= n_units) return;
  const int64_t row = u / H;
  const int h = (int)(u - row * H);
  float r[4], w[4], gv[4];
  load4<float>(raw + u * DC_D + lane * 4, r);
  const __nv_bfloat16* gp = gate + row * ld_gate + (int64_t)h * DC_D + lane * 4;
  load4<__nv_bfloat16>(gp, gv);
  load4<float>(nw + lane * 4, w);
  const float ss = warp_sum((r[0] * r[0] + r[1] * r[1]) + (r[2] * r[2] + r[3] * r[3]));
  const float inv = rsqrtf(ss / (float)DC_D + eps);
  uint2 o;
#pragma unroll
  for (int i = 0; i < 4; ++i) r[i] = r[i] * inv * w[i] * (1.0f / (1.0f + expf(-gv[i])));
  o.x = Num<__nv_bfloat16>::pack(r[0], r[1]);
  o.y = Num<__nv_bfloat16>::pack(r[2], r[3]);
  *reinterpret_cast<uint2*>(out + row * ldo + (int64_t)h * DC_D + lane * 4) = o;
}

template <int NW>
int launch_scan(float* raw, const uint8_t* units, const float* v, float* state, const int* q_cu, const int* positions,
                const int* slots, int n_seq, int H, cudaStream_t st) {
  auto kern = delta_chunk_scan_kernel<NW>;
  B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, DC_STAGES * DC_UNIT));
  kern<<<dim3((unsigned)H, (unsigned)n_seq, 8 / NW), (NW + 1) * 32, DC_STAGES * DC_UNIT, st>>>(raw, units, v, state, q_cu,
                                                                                               positions, slots, H);
  B200_LAUNCH_OK("delta_chunk_scan_kernel");
  return B200_OK;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

int64_t b200_gated_delta_chunked_workspace_bytes(int64_t rows, int64_t n_seq, int64_t H) {
  return (rows / DC_T + n_seq) * H * DC_UNIT + rows * H * DC_D * (int64_t)sizeof(float);
}

int b200_gated_delta_chunked(void* out, int64_t ldo, const void* gate_logits, int64_t ld_gate, const float* norm_weight,
                             float eps, const float* q, const float* k, const float* v, const float* decay,
                             const float* beta, float* state, const int32_t* q_cu_lens, const int32_t* positions,
                             const int32_t* state_slots, int64_t n_seq, int64_t rows, int64_t q_max, int64_t H, int64_t G,
                             void* workspace, int64_t workspace_bytes, b200_stream_t stream) {
  if (n_seq == 0 || rows == 0) return B200_OK;
  B200_CHECK_ARG(out && gate_logits && norm_weight && q && k && v && decay && beta && state && q_cu_lens && positions && state_slots && workspace,
                 "gated_delta_chunked: null pointer");
  const int64_t chunks = (q_max + DC_T - 1) / DC_T;
  B200_CHECK_ARG(n_seq > 0 && n_seq <= 65535 && rows > 0 && q_max > 0 && chunks <= 65535 && H > 0 && G > 0 && H % G == 0 &&
                     ldo >= H * DC_D && ldo % 4 == 0 && is_aligned(out, 8) && ld_gate >= H * DC_D && ld_gate % 4 == 0 &&
                     is_aligned(gate_logits, 8) && is_aligned(norm_weight, 16) && is_aligned(q, 8) && is_aligned(k, 8) && is_aligned(decay, 8) && is_aligned(workspace, 16) &&
                     workspace_bytes >= b200_gated_delta_chunked_workspace_bytes(rows, n_seq, H),
                 "gated_delta_chunked: bad shape or workspace");
  auto st = static_cast<cudaStream_t>(stream);
  float* raw = static_cast<float*>(workspace);             // read-outs, then the chunks' operands
  uint8_t* units = reinterpret_cast<uint8_t*>(raw + rows * H * DC_D);
  delta_chunks_kernel<<<dim3((unsigned)H, (unsigned)chunks, (unsigned)n_seq), 64, 0, st>>>(units, q, k, decay, beta,
                                                                                            q_cu_lens, (int)H, (int)G);
  B200_LAUNCH_OK("delta_chunks_kernel");
  // a CTA per SM or more: fewer sequences and heads than that share a state's columns out over up to four CTAs
  const int64_t pairs = n_seq * H, sms = sm_count();
  int rc;
#define DC_GO(NW) launch_scan<NW>(raw, units, v, state, q_cu_lens, positions, state_slots, (int)n_seq, (int)H, st)
  if (pairs * 2 > sms) rc = DC_GO(8);
  else if (pairs * 4 > sms) rc = DC_GO(4);
  else rc = DC_GO(2);
#undef DC_GO
  if (rc != B200_OK) return rc;
  const int64_t n_units = rows * H;
  delta_norm_gate_kernel<<<(unsigned)((n_units + 7) / 8), 256, 0, st>>>(
      static_cast<__nv_bfloat16*>(out), ldo, raw, static_cast<const __nv_bfloat16*>(gate_logits), ld_gate, norm_weight, n_units,
      (int)H, eps);
  B200_LAUNCH_OK("delta_norm_gate_kernel");
  return B200_OK;
}

}  // extern "C"
