// nrgpu_mlp.cu -- the learned warm start of the puncture multigrid (sm_100a).
// No counterpart in the reference: a coordinate MLP conditioned on the
// puncture parameters predicts the conformal-factor correction u that
// PunctureData otherwise obtains from u = 0 by multigrid.
//
// Network: 32 input features -> 4 hidden layers of 128 (SiLU) -> 1 output.
// Every hidden-layer product runs on the tensor cores as BF16 x BF16 with
// FP32 accumulation (mma.sync m16n8k16); the master weights, the Adam state,
// biases and the output layer are FP32, the loss is summed in 64 bits (its error
// against a 64-bit network, 2e-5 to 4e-4 after 16 steps, is the BF16 products').
// Training is the plain reverse-mode chain with the same BF16 operands as the forward pass.
//
// Kernels:
//   mlp_features_kernel     feature rows (double math, rounded to BF16)
//   mlp_rows_kernel         forward, loss and backward of 128 rows per block
//   mlp_weight_grad_kernel  dW = A^T dZ, split over row chunks with FP32 atomics
//   adam_kernel             Adam step on the FP32 master copy + BF16 refresh
#include <cuda_bf16.h>
#include <stdint.h>
#include <string.h>
#include "nrgpu_common.cuh"
#include "nrgpu_tma.cuh"

static constexpr int IN = NRGPU_MLP_IN;
static constexpr int HID = NRGPU_MLP_HIDDEN;

namespace {

// flat FP32 parameter layout: W1 [IN][HID], b1, W2 [HID][HID], b2, W3, b3,
// W4, b4, w5 [HID], b5
__host__ __device__ constexpr int off_w(int l) { return l == 0 ? 0 : IN * HID + HID + (l - 1) * (HID * HID + HID); }
constexpr int kOffW5 = IN * HID + HID + 3 * (HID * HID + HID);
constexpr int kNParams = kOffW5 + HID + 1;
__host__ __device__ constexpr int off_b(int l) { return off_w(l) + (l == 0 ? IN : HID) * HID; }
__host__ __device__ constexpr int fan_in(int l) { return l == 0 ? IN : HID; }

// ---- features ----------------------------------------------------------------
// conditioning vector of one binary: m1 m2 | pos 6 | mom 6 | spin 6
struct Feat {
  int m;
  double dx;
};

__device__ __forceinline__ __nv_bfloat16 to_bf16(double v) { return __float2bfloat16_rn((float)v); }

__global__ void mlp_features_kernel(const double *__restrict__ cond, const int *__restrict__ set,
                                    const int *__restrict__ pt, long first, int n, Feat F, __nv_bfloat16 *X) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const long p = pt ? (long)pt[r] : first + r;
  const double *c = cond + 20 * (set ? set[r] : 0);
  const int m = F.m;
  const double h0 = -0.5 * (m - 1) * F.dx;
  const int i = (int)(p % m), j = (int)((p / m) % m), k = (int)(p / ((long)m * m));
  const double x[3] = {h0 + i * F.dx, h0 + j * F.dx, h0 + k * F.dx};
  const double s = 1.0 / 8.0;
  __nv_bfloat16 *f = X + (long)r * IN;
  f[0] = to_bf16(x[0] * s);
  f[1] = to_bf16(x[1] * s);
  f[2] = to_bf16(x[2] * s);
  for (int q = 0; q < 2; ++q) {
    const double mq = c[q];
    const double d0 = x[0] - c[2 + 3 * q], d1 = x[1] - c[3 + 3 * q], d2 = x[2] - c[4 + 3 * q];
    const double rr = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
    __nv_bfloat16 *g = f + 3 + 12 * q;
    g[0] = to_bf16(d0 * s);
    g[1] = to_bf16(d1 * s);
    g[2] = to_bf16(d2 * s);
    g[3] = to_bf16(rr * s);
    g[4] = to_bf16(mq / (rr + mq));
    g[5] = to_bf16(2.0 * mq);
    for (int a = 0; a < 3; ++a) {
      g[6 + a] = to_bf16(5.0 * c[8 + 3 * q + a]);
      g[9 + a] = to_bf16(5.0 * c[14 + 3 * q + a]);
    }
  }
  for (int q = 27; q < IN; ++q) f[q] = __float2bfloat16_rn(0.0f);
}

// ---- forward and backward of 128 rows on the tensor cores -------------------------
// One kernel runs the whole network over a block's 128 rows: the BF16 weights
// of all layers lie in shared memory, two warps share 16 rows, each with half
// of the columns of every layer, and pass their halves of the next operand
// through shared memory (a barrier of the pair per layer); the backward pass
// follows in the same way.  Training writes what the weight gradients need,
// the BF16 activations and pre-activation gradients of every layer, and keeps
// silu'(z) in FP32 (Z) between the passes.  With a kernel per product and per
// elementwise step the same work took 32 launches and eleven passes over
// 8 MB arrays: 380 us per step of 16384 rows.  What bounds it now is latency:
// a step has rows for one block per SM, so 16 warps (with whole rows per
// warp, 8 warps, this kernel took 100 us).
constexpr int kWPitch = HID + 8;             // BF16 per weight row: ldmatrix meets no bank twice
constexpr int kWRows = IN + 3 * HID;
constexpr int kRowsSmem = (kWRows + 2 * 128) * kWPitch * 2;

__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + expf(-z)); }

__device__ __forceinline__ void mma16816(float d[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t r[4], const __nv_bfloat16 *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm4t(uint32_t r[4], const __nv_bfloat16 *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void cp16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ float2 unpack2(uint32_t v) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&v));
}

struct RowsArgs {
  const __nv_bfloat16 *X, *Wb;  // features, weights of W1..W4
  const float *P, *y;
  float *out;                   // network output per row
  float *Z[4];                  // silu'(z) (training)
  __nv_bfloat16 *A[4], *dZ[4];  // activations, pre-activation gradients (training)
  float *grad;
  double *loss;
  int n;
};

// sum over the rows of a warp's 16 x 8 tiles: v[0], v[1] = this thread's
// columns 2 tg, 2 tg + 1; the lanes of row 0 add the result
__device__ __forceinline__ void add_columns(float *dst, float v0, float v1, int lane) {
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    v0 += __shfl_xor_sync(0xffffffffu, v0, o);
    v1 += __shfl_xor_sync(0xffffffffu, v1, o);
  }
  if (lane < 4) {
    atomicAdd(dst + 2 * lane, v0);
    atomicAdd(dst + 2 * lane + 1, v1);
  }
}

constexpr int kRowsThreads = 512;
__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

template <bool TRAIN>
__global__ void __launch_bounds__(kRowsThreads) mlp_rows_kernel(const RowsArgs a) {
  extern __shared__ __align__(16) __nv_bfloat16 wsm[];
  __nv_bfloat16 *xsm = wsm + kWRows * kWPitch;  // two buffers of 128 rows, the operands between layers
  __shared__ float sums[5 * HID + 1];  // db of the four layers, dw5, db5
  __shared__ double squares[kRowsThreads / 64];  // loss of each pair of warps, in 64 bits
  __shared__ float outs[2][128];       // the two halves of the output sums
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, tg = lane & 3;
  const int pair = warp >> 1, c0 = (warp & 1) * (HID / 2);  // 16 rows, 64 columns
  for (int q = t; q < kWRows * HID / 8; q += kRowsThreads)
    cp16(wsm + (q / (HID / 8)) * kWPitch + (q % (HID / 8)) * 8, a.Wb + (long)q * 8);
  if (TRAIN) {
    for (int q = t; q < 5 * HID + 1; q += kRowsThreads) sums[q] = 0.0f;
    if (t < kRowsThreads / 64) squares[t] = 0.0;
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int r0 = blockIdx.x * 128 + pair * 16;
  if (r0 < a.n) {
    // this lane's row of an ldmatrix: matrix lane / 8, row lane % 8
    const int mi = lane >> 3, ri = lane & 7;
    uint32_t af[8][4];  // the layer's operand: 16 rows, all columns
    const long ra = (long)(r0 + g), rb = ra + 8;
    // the pair's rows of the operand buffers: where this lane writes and reads
    __nv_bfloat16 *put = xsm + (pair * 16 + g) * kWPitch + 2 * tg + c0;
    const __nv_bfloat16 *get = xsm + (pair * 16 + (mi & 1) * 8 + ri) * kWPitch + (mi >> 1) * 8;
    constexpr int kBuf = 128 * kWPitch;
#pragma unroll
    for (int ks = 0; ks < IN / 16; ++ks) {
      const __nv_bfloat16 *p = a.X + ra * IN + ks * 16 + 2 * tg, *q = a.X + rb * IN + ks * 16 + 2 * tg;
      af[ks][0] = *(const uint32_t *)p;
      af[ks][1] = *(const uint32_t *)q;
      af[ks][2] = *(const uint32_t *)(p + 8);
      af[ks][3] = *(const uint32_t *)(q + 8);
    }
    float acc[8][4];
    uint32_t last[8][2];  // the last layer's activations
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const int wr = l == 0 ? 0 : IN + (l - 1) * HID;  // first weight row of the layer
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[nt][e] = 0.0f;
#pragma unroll
      for (int ks = 0; ks < (l == 0 ? IN : HID) / 16; ++ks)
#pragma unroll
        for (int nt = 0; nt < 8; nt += 2) {
          uint32_t bf[4];
          ldsm4t(bf, wsm + (wr + ks * 16 + (mi & 1) * 8 + ri) * kWPitch + c0 + nt * 8 + (mi >> 1) * 8);
          mma16816(acc[nt], af[ks], bf[0], bf[1]);
          mma16816(acc[nt + 1], af[ks], bf[2], bf[3]);
        }
      const float *bias = a.P + off_b(l);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const int c = c0 + nt * 8 + 2 * tg;
        const float2 bc = *(const float2 *)(bias + c);
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float z = acc[nt][e] + (e & 1 ? bc.y : bc.x), s = sigm(z);
          y[e] = z * s;
          if (TRAIN) acc[nt][e] = s * (1.0f + z * (1.0f - s));
        }
        const uint32_t ya = pack2(y[0], y[1]), yb = pack2(y[2], y[3]);
        if (l < 3) {
          *(uint32_t *)(put + (l & 1) * kBuf + nt * 8) = ya;
          *(uint32_t *)(put + (l & 1) * kBuf + 8 * kWPitch + nt * 8) = yb;
        }
        last[nt][0] = ya;
        last[nt][1] = yb;
        if (TRAIN && l < 3) {
          *(uint32_t *)(a.A[l] + ra * HID + c) = ya;
          *(uint32_t *)(a.A[l] + rb * HID + c) = yb;
          *(float2 *)(a.Z[l] + ra * HID + c) = make_float2(acc[nt][0], acc[nt][1]);
          *(float2 *)(a.Z[l] + rb * HID + c) = make_float2(acc[nt][2], acc[nt][3]);
        }
      }
      if (l < 3) {
        pair_sync(1 + pair);
#pragma unroll
        for (int ks = 0; ks < HID / 16; ++ks) ldsm4(af[ks], get + (l & 1) * kBuf + ks * 16);
      }
    }
    // out = A4 w5 + b5
    const float *w5 = a.P + kOffW5;
    float oa = 0.0f, ob = 0.0f;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const float2 w = *(const float2 *)(w5 + c0 + nt * 8 + 2 * tg);
      const float2 u = unpack2(last[nt][0]), v = unpack2(last[nt][1]);
      oa = fmaf(u.x, w.x, fmaf(u.y, w.y, oa));
      ob = fmaf(v.x, w.x, fmaf(v.y, w.y, ob));
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      oa += __shfl_xor_sync(0xffffffffu, oa, o);
      ob += __shfl_xor_sync(0xffffffffu, ob, o);
    }
    if (tg == 0) {
      outs[warp & 1][pair * 16 + g] = oa;
      outs[warp & 1][pair * 16 + g + 8] = ob;
    }
    pair_sync(1 + pair);
    oa = outs[0][pair * 16 + g] + outs[1][pair * 16 + g] + w5[HID];
    ob = outs[0][pair * 16 + g + 8] + outs[1][pair * 16 + g + 8] + w5[HID];
    if (tg == 0 && c0 == 0) {
      a.out[ra] = oa;
      a.out[rb] = ob;
    }
    if (TRAIN) {
      const float ea = oa - a.y[ra], eb = ob - a.y[rb];
      const float da = 2.0f * ea / (float)a.n, db = 2.0f * eb / (float)a.n;
      if (tg == 0 && c0 == 0) {
        atomicAdd(sums + 5 * HID, da + db);
      }
      if (c0 == 0) {
        double q = (double)ea * ea + (double)eb * eb;
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        if (lane == 0) squares[pair] = q;
      }
#pragma unroll
      for (int l = 3; l >= 0; --l) {
        // acc: silu' of layer 3, or dA of layer l; dZ_l out and into the next operand
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
          const int c = c0 + nt * 8 + 2 * tg;
          uint32_t fa, fb;
          if (l == 3) {
            const float2 u = unpack2(last[nt][0]), v = unpack2(last[nt][1]), w = *(const float2 *)(w5 + c);
            add_columns(sums + 4 * HID + c0 + nt * 8, da * u.x + db * v.x, da * u.y + db * v.y, lane);
            fa = pack2(da * w.x * acc[nt][0], da * w.y * acc[nt][1]);
            fb = pack2(db * w.x * acc[nt][2], db * w.y * acc[nt][3]);
          } else {
            const float2 u = *(const float2 *)(a.Z[l] + ra * HID + c), v = *(const float2 *)(a.Z[l] + rb * HID + c);
            fa = pack2(acc[nt][0] * u.x, acc[nt][1] * u.y);
            fb = pack2(acc[nt][2] * v.x, acc[nt][3] * v.y);
          }
          if (l > 0) {
            *(uint32_t *)(put + (l & 1) * kBuf + nt * 8) = fa;
            *(uint32_t *)(put + (l & 1) * kBuf + 8 * kWPitch + nt * 8) = fb;
          }
          *(uint32_t *)(a.dZ[l] + ra * HID + c) = fa;
          *(uint32_t *)(a.dZ[l] + rb * HID + c) = fb;
          const float2 u = unpack2(fa), v = unpack2(fb);
          add_columns(sums + l * HID + c0 + nt * 8, u.x + v.x, u.y + v.y, lane);
        }
        if (l == 0) break;
        pair_sync(1 + pair);
#pragma unroll
        for (int ks = 0; ks < HID / 16; ++ks) ldsm4(af[ks], get + (l & 1) * kBuf + ks * 16);
        const int wr = IN + (l - 1) * HID;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[nt][e] = 0.0f;
#pragma unroll
        for (int ks = 0; ks < HID / 16; ++ks)
#pragma unroll
          for (int nt = 0; nt < 8; nt += 2) {
            uint32_t bf[4];  // columns of W_l^T: rows of W_l
            ldsm4(bf, wsm + (wr + c0 + nt * 8 + (mi >> 1) * 8 + ri) * kWPitch + ks * 16 + (mi & 1) * 8);
            mma16816(acc[nt], af[ks], bf[0], bf[1]);
            mma16816(acc[nt + 1], af[ks], bf[2], bf[3]);
          }
      }
    }
  }
  if (TRAIN) {
    __syncthreads();
    for (int q = t; q < 5 * HID; q += kRowsThreads)
      atomicAdd(a.grad + (q < 4 * HID ? off_b(q / HID) + q % HID : kOffW5 + q % HID), sums[q]);
    if (t == 0) {
      atomicAdd(a.grad + kOffW5 + HID, sums[5 * HID]);
      double q = 0.0;
      for (int w = 0; w < kRowsThreads / 64; ++w) q += squares[w];
      atomicAdd(a.loss, q / a.n);
    }
  }
}

// ---- weight gradients ---------------------------------------------------------------
// dW_l += A_{l-1}^T dZ_l of rows [z chunk, (z + 1) chunk) for layer blockIdx.x:
// the whole fan_in x 128 product in one block's registers (16 rows of dW per
// warp), 64 rows of both operands at a time through shared memory, fetched
// ahead by cp.async; the partial sums of the row chunks meet in FP32 atomics.
constexpr int kGradRows = 64;
constexpr int kGradSmem = 2 * 2 * kGradRows * kWPitch * 2;

__global__ void __launch_bounds__(256) mlp_weight_grad_kernel(const RowsArgs a, int chunk) {
  extern __shared__ __align__(16) __nv_bfloat16 gsm[];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, tg = lane & 3;
  const int l = blockIdx.x, fi = l == 0 ? IN : HID;
  const __nv_bfloat16 *A = l == 0 ? a.X : a.A[l - 1], *D = a.dZ[l];
  const int r0 = blockIdx.y * chunk, r1 = min(a.n, r0 + chunk);
  auto fetch = [&](int buf, int r) {  // rows r .. r + 63 (a multiple of 64 rows in all)
    __nv_bfloat16 *sa = gsm + buf * 2 * kGradRows * kWPitch, *sd = sa + kGradRows * kWPitch;
    for (int q = t; q < kGradRows * fi / 8; q += 256) cp16(sa + (q / (fi / 8)) * kWPitch + (q % (fi / 8)) * 8, A + (long)r * fi + (long)q * 8);
    for (int q = t; q < kGradRows * HID / 8; q += 256) cp16(sd + (q / (HID / 8)) * kWPitch + (q % (HID / 8)) * 8, D + (long)r * HID + (long)q * 8);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[16][4];
#pragma unroll
  for (int nt = 0; nt < 16; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[nt][e] = 0.0f;
  const int mi = lane >> 3, ri = lane & 7;
  if (r0 < r1) fetch(0, r0);
  int buf = 0;
  for (int r = r0; r < r1; r += kGradRows, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (r + kGradRows < r1) fetch(buf ^ 1, r + kGradRows);
    const __nv_bfloat16 *sa = gsm + buf * 2 * kGradRows * kWPitch, *sd = sa + kGradRows * kWPitch;
    if (warp * 16 < fi) {
#pragma unroll
      for (int ks = 0; ks < kGradRows / 16; ++ks) {
        uint32_t af[4];
        ldsm4t(af, sa + (ks * 16 + (mi >> 1) * 8 + ri) * kWPitch + warp * 16 + (mi & 1) * 8);
#pragma unroll
        for (int nt = 0; nt < 16; nt += 2) {
          uint32_t bf[4];
          ldsm4t(bf, sd + (ks * 16 + (mi & 1) * 8 + ri) * kWPitch + nt * 8 + (mi >> 1) * 8);
          mma16816(acc[nt], af, bf[0], bf[1]);
          mma16816(acc[nt + 1], af, bf[2], bf[3]);
        }
      }
    }
    __syncthreads();
  }
  if (warp * 16 >= fi || r0 >= r1) return;
  float *G = a.grad + off_w(l) + (long)(warp * 16 + g) * HID + 2 * tg;
#pragma unroll
  for (int nt = 0; nt < 16; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(G + h * 8 * HID + nt * 8), "f"(acc[nt][2 * h]),
                   "f"(acc[nt][2 * h + 1])
                   : "memory");
}

struct AdamArgs {
  float lr, b1, b2, eps, c1, c2;  // c1 = 1/(1-b1^t), c2 = 1/(1-b2^t)
};

// the BF16 copy of weight i of the flat layout, -1 for biases and w5
__device__ __forceinline__ int wb_index(int i) {
#pragma unroll
  for (int l = 0; l < 4; ++l)
    if (i >= off_w(l) && i < off_b(l)) return (l == 0 ? 0 : IN * HID + (l - 1) * HID * HID) + i - off_w(l);
  return -1;
}

// Adam step and the refreshed BF16 copy
__global__ void adam_kernel(float *P, const float *__restrict__ G, float *Mo, float *Vo, __nv_bfloat16 *Wb, AdamArgs a,
                            int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float g = G[i];
  const float m = a.b1 * Mo[i] + (1.0f - a.b1) * g;
  const float v = a.b2 * Vo[i] + (1.0f - a.b2) * g * g;
  Mo[i] = m;
  Vo[i] = v;
  const float p = P[i] - a.lr * (m * a.c1) / (sqrtf(v * a.c2) + a.eps);
  P[i] = p;
  const int w = wb_index(i);
  if (w >= 0) Wb[w] = __float2bfloat16_rn(p);
}

// BF16 copies of W1..W4 in the [K][N] layout of the forward products
__global__ void refresh_bf16_kernel(const float *__restrict__ P, __nv_bfloat16 *Wb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n1 = IN * HID, nh = HID * HID;
  if (i >= n1 + 3 * nh) return;
  int l, q;
  if (i < n1) { l = 0; q = i; }
  else { l = 1 + (i - n1) / nh; q = (i - n1) % nh; }
  Wb[i] = __float2bfloat16_rn(P[off_w(l) + q]);
}

// ---- FP32 inference (CUDA cores) ------------------------------------------------
// The whole forward pass for 128 grid points per block, in FP32 from the FP32
// master weights: features rounded to FP32 only (not BF16), hidden products
// as a 128 x 128 x K register-tiled product (thread: 8 rows x 8 columns),
// bias + SiLU, the output layer by a warp reduction; u = s out.
// Used to evaluate the trained network without the BF16 rounding of the
// training path (whose grid-scale noise the undamped Jacobi smoother of the
// multigrid does not remove).
// Bound by the FP32 units.  The activations stay in shared memory with the
// rows of one feature side by side, the weights pass through it in chunks of
// 16 features fetched ahead by cp.async: 4 16-byte loads per 64 FMAs and
// thread.  Two blocks per SM, so that one's SiLU runs beside the other's FMAs.
constexpr int kFR = 128;          // rows (grid points) per block
constexpr int kFP = kFR + 4;      // row pitch: 8 lanes' 16-byte stores at stride kFP meet no bank twice
constexpr int kFK = 16;           // features per weight chunk
constexpr int kFSmem = (HID * kFP + 2 * kFK * HID) * (int)sizeof(float);

// chunk c of a layer's weights into buf: column cg + 16 q of a feature at
// (q / 4) 64 + 4 cg + q % 4, i.e. a thread's 8 columns as two 16-byte words
__device__ __forceinline__ void weights_ahead(float *buf, const float *__restrict__ W, int c, int t) {
#pragma unroll
  for (int e = t; e < kFK * HID; e += 256) {
    const int k = e / HID, j = e % HID, q = j / 16;
    const unsigned d = (unsigned)__cvta_generic_to_shared(buf + k * HID + (q / 4) * 64 + (j % 16) * 4 + q % 4);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(W + (long)c * kFK * HID + e) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

__global__ void __launch_bounds__(256, 2) mlp_forward_fp32_kernel(const double *__restrict__ cond, int m, double dx,
                                                                  const float *__restrict__ P, double s, double *u,
                                                                  long np) {
  extern __shared__ __align__(16) float fsm[];
  float *act = fsm, *wb = fsm + HID * kFP;  // act[feature][row], two weight chunks
  const int t = threadIdx.x;
  const long first = (long)blockIdx.x * kFR;
  weights_ahead(wb, P + off_w(0), 0, t);
  // features of the block's rows (the formulas of mlp_features_kernel)
  if (t < kFR) {
    float *f = act + t;
    const long p = min(first + t, np - 1);
    const double h0 = -0.5 * (m - 1) * dx;
    const int i = (int)(p % m), j = (int)((p / m) % m), k = (int)(p / ((long)m * m));
    const double x[3] = {h0 + i * dx, h0 + j * dx, h0 + k * dx};
    const double sc = 1.0 / 8.0;
    f[0] = (float)(x[0] * sc);
    f[kFP] = (float)(x[1] * sc);
    f[2 * kFP] = (float)(x[2] * sc);
    for (int q = 0; q < 2; ++q) {
      const double mq = cond[q];
      const double d0 = x[0] - cond[2 + 3 * q], d1 = x[1] - cond[3 + 3 * q], d2 = x[2] - cond[4 + 3 * q];
      const double rr = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
      float *g = f + (3 + 12 * q) * kFP;
      g[0] = (float)(d0 * sc);
      g[kFP] = (float)(d1 * sc);
      g[2 * kFP] = (float)(d2 * sc);
      g[3 * kFP] = (float)(rr * sc);
      g[4 * kFP] = (float)(mq / (rr + mq));
      g[5 * kFP] = (float)(2.0 * mq);
      for (int a = 0; a < 3; ++a) {
        g[(6 + a) * kFP] = (float)(5.0 * cond[8 + 3 * q + a]);
        g[(9 + a) * kFP] = (float)(5.0 * cond[14 + 3 * q + a]);
      }
    }
    for (int q = 27; q < IN; ++q) f[q * kFP] = 0.0f;
  }
  const int cg = t % 16, rg = t / 16;  // columns cg + 16 q, rows 4 rg .. 4 rg + 3 and 64 further
  int buf = 0;
  for (int l = 0; l < 4; ++l) {
    const int nc = fan_in(l) / kFK;
    const float *W = P + off_w(l), *bias = P + off_b(l);
    float acc[8][8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[r][q] = 0.0f;
    for (int c = 0; c < nc; ++c) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // the chunk, and the layer's activations, are there; the other buffer is free
      if (c + 1 < nc) weights_ahead(wb + (buf ^ 1) * kFK * HID, W, c + 1, t);
      else if (l < 3) weights_ahead(wb + (buf ^ 1) * kFK * HID, P + off_w(l + 1), 0, t);
      const float *wk = wb + buf * kFK * HID + 4 * cg, *ak = act + c * kFK * kFP + 4 * rg;
#pragma unroll
      for (int k = 0; k < kFK; ++k) {
        float a[8], w[8];
        *(float4 *)a = *(const float4 *)(ak + k * kFP);
        *(float4 *)(a + 4) = *(const float4 *)(ak + k * kFP + 64);
        *(float4 *)w = *(const float4 *)(wk + k * HID);
        *(float4 *)(w + 4) = *(const float4 *)(wk + k * HID + 64);
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[r][q] = fmaf(a[r], w[q], acc[r][q]);
      }
      buf ^= 1;
    }
    __syncthreads();  // every thread has read the layer's input
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int col = cg + 16 * q;
      const float bq = __ldg(bias + col);
      float y[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float z = acc[r][q] + bq;
        y[r] = z * sigm(z);
      }
      *(float4 *)(act + col * kFP + 4 * rg) = *(float4 *)y;
      *(float4 *)(act + col * kFP + 64 + 4 * rg) = *(float4 *)(y + 4);
    }
  }
  __syncthreads();
  // out = A4 w5 + b5: warp w reduces rows 16 w .. 16 w + 15
  const int w = t >> 5, lane = t & 31;
  const float *w5 = P + kOffW5;
  for (int r = 16 * w; r < 16 * w + 16; ++r) {
    float v = 0.0f;
    for (int k = lane; k < HID; k += 32) v = fmaf(act[k * kFP + r], __ldg(w5 + k), v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0 && first + r < np) u[first + r] = s * (double)(v + __ldg(w5 + HID));
  }
}

__global__ void scale_to_u_kernel(const float *__restrict__ o, double s, double *u, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) u[i] = s * (double)o[i];
}

// ---- the forward pass on the 5th-generation tensor cores (tcgen05) ---------------
// One CTA of 512 threads per SM, two teams of 8 warps; each team walks its
// own tiles of 128 grid points with its own 128 columns of tensor memory,
// so the tensor core runs one team's layer while the other forms its
// activations.  W1..W4 sit in shared memory for the whole walk, as BF16 in
// the K-major layout without swizzle that the MMA reads through matrix
// descriptors: an operand of R rows and K columns is stored as K/8 chunks of
// R x 8 elements, each chunk row by row (16 B per row), so the 8-row core
// matrices are 128 B apart (stride byte offset) and the two 8-column chunks
// of one K = 16 step are 16 R bytes apart (leading byte offset).  Per tile:
// the features of the 128 points go into X; per layer one thread of the
// team issues the tcgen05.mma chain D[128 x 128] (FP32, tensor memory) =
// X or A (128 x K) * W^T and commits it to the team's mbarrier; thread
// (row, half) of the team then reads columns 64 half .. 64 half + 63 of its
// row of D (tcgen05.ld: warp w reaches lanes 32 (w mod 4) ..), adds the
// bias, applies SiLU, rounds to BF16 and writes the next layer's A (after
// layer 4 the two halves form out = A4 w5 + b5).  Operands BF16,
// accumulation FP32: the arithmetic of the training path.  SiLU is
// z sigm(z) = z/2 (1 + tanh(z/2)) with the hardware tanh (tanh.approx.f32,
// relative error about 2^-11, below the BF16 rounding that follows).
namespace tc {
constexpr int kRows = 128;
constexpr int kThreads = 512;                    // two teams of 256
constexpr int kChunk = kRows * 16;               // bytes of one 8-column chunk of a 128-row operand
constexpr int kOffW0 = 0;                        // W1^T: 128 x 32, 4 chunks
constexpr int kOffW = kOffW0 + 4 * kChunk;       // W2^T, W3^T, W4^T: 128 x 128, 16 chunks each
constexpr int kOffX = kOffW + 3 * 16 * kChunk;   // features, per team: 128 x 32
constexpr int kOffA = kOffX + 2 * 4 * kChunk;    // activations, per team: 128 x 128
constexpr int kOffP = kOffA + 2 * 16 * kChunk;   // b1..b4 [4][128], w5 [128], b5 (FP32)
constexpr int kOffRed = kOffP + ((4 * HID + HID + 1) * 4 + 15) / 16 * 16;   // per team: 128 partial outputs
constexpr int kOffBar = kOffRed + 2 * kRows * 4; // 2 mbarriers
constexpr int kOffTmem = kOffBar + 16;           // the tensor-memory base address; 2 timeout flags
constexpr int kSmem = kOffTmem + 16 + 128;       // + room to align the base to 128 B
static_assert(kSmem <= 227 * 1024, "shared memory of the tensor-core forward");
// the instruction descriptor of kind::f16: FP32 accumulator, A and B BF16,
// both K-major, N = 128 (bits 17-22: N/8), M = 128 (bits 24-28: M/16)
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

// byte offset of element (row, k) in a chunked K-major operand
__device__ __forceinline__ int off(int row, int k) { return (k >> 3) * kChunk + row * 16 + (k & 7) * 2; }

// shared-memory matrix descriptor (sm_100): start address >> 4 (bits 0-13),
// leading byte offset >> 4 (bits 16-29: between the two K chunks of one
// MMA), stride byte offset >> 4 (bits 32-45: between 8-row core matrices),
// version 1 (bits 46-47), base offset 0, no swizzle (bits 61-63 zero)
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((kChunk >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((128 >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void mma(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      ::"r"(dtmem), "l"(a), "l"(b), "r"(kIdesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   tma::smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// barrier of one team (named barriers 1 and 2)
__device__ __forceinline__ void team_sync(int team) { asm volatile("bar.sync %0, 256;" ::"r"(team + 1) : "memory"); }

__device__ __forceinline__ float silu(float z) {
  float th;
  const float h = 0.5f * z;
  asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(h));
  return fmaf(h, th, h);
}
// two FP32 values rounded to nearest even BF16, packed (lower column low)
template <int CVT>
__device__ __forceinline__ uint32_t pack_bf16(float x0, float x1) {
  if (CVT == 0) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x0, x1);
    return *reinterpret_cast<const uint32_t *>(&v);
  }
  // round to nearest even on the bits (finite values): add 0x7FFF plus the
  // lowest kept bit, keep the upper 16 bits
  uint32_t u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
  u0 += 0x7FFFu + ((u0 >> 16) & 1u);
  u1 += 0x7FFFu + ((u1 >> 16) & 1u);
  return __byte_perm(u0, u1, 0x7632);
}

// 32 consecutive FP32 columns of this thread's row (warp-collective); the
// caller waits (tcgen05.wait::ld) before using them
__device__ __forceinline__ void ld32(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
}  // namespace tc

template <int CVT>
__global__ void __launch_bounds__(tc::kThreads, 1) mlp_forward_tc_kernel(const double *__restrict__ cond, int m,
                                                                        double dx, const float *__restrict__ P,
                                                                        double uscale, double *u, long np,
                                                                        int *status) {
  using namespace tc;
  extern __shared__ __align__(128) unsigned char tc_raw[];
  unsigned char *sm = tc_raw + ((128 - (tma::smem_addr(tc_raw) & 127)) & 127);
  const int t = threadIdx.x, warp = t >> 5, team = t >> 8, tr = t & 255, r = tr & 127, half = tr >> 7;
  const uint32_t sbase = tma::smem_addr(sm);
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm + kOffBar) + team;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + kOffTmem);
  volatile int *failed = reinterpret_cast<volatile int *>(sm + kOffTmem + 4);
  float *par = reinterpret_cast<float *>(sm + kOffP);
  float *red = reinterpret_cast<float *>(sm + kOffRed) + team * kRows;
  // the weights, transposed to [n][k] in the chunked layout, and the biases
  for (int idx = t; idx < IN * HID; idx += kThreads) {
    const int k = idx / HID, n = idx % HID;
    *reinterpret_cast<__nv_bfloat16 *>(sm + kOffW0 + off(n, k)) = __float2bfloat16_rn(P[off_w(0) + idx]);
  }
  for (int l = 1; l < 4; ++l)
    for (int idx = t; idx < HID * HID; idx += kThreads) {
      const int k = idx / HID, n = idx % HID;
      *reinterpret_cast<__nv_bfloat16 *>(sm + kOffW + (l - 1) * 16 * kChunk + off(n, k)) =
          __float2bfloat16_rn(P[off_w(l) + idx]);
    }
  for (int idx = t; idx < 4 * HID; idx += kThreads) par[idx] = P[off_b(idx / HID) + idx % HID];
  for (int idx = t; idx <= HID; idx += kThreads) par[4 * HID + idx] = P[kOffW5 + idx];
  // 256 columns of tensor memory: the FP32 accumulators (128 x 128) of the
  // two teams
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tma::smem_addr(tslot)),
                 "r"(256u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t < 2) {
    tma::mbar_init(reinterpret_cast<uint64_t *>(sm + kOffBar) + t, 1);
    failed[t] = 0;
  }
  if (t == 0) tma::mbar_fence_init();
  fence_async_smem();
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t dcol = tmem + 128u * team;                                          // the team's accumulator
  const uint32_t trow = dcol + ((uint32_t)(32 * (warp & 3)) << 16) + 64u * half;     // this thread's lanes/half
  unsigned char *X = sm + kOffX + team * 4 * kChunk;
  unsigned char *A = sm + kOffA + team * 16 * kChunk;
  const float *w5 = par + 4 * HID;
  uint32_t phase = 0;
  const long ntiles = (np + kRows - 1) / kRows;
  for (long tile = 2L * blockIdx.x + team; tile < ntiles; tile += 2L * gridDim.x) {
    const long row = tile * kRows + r;
    {
      // features of this thread's point (mlp_features_kernel's formulas):
      // half 0 forms columns 0-15 (the coordinates, the first puncture's
      // twelve, the second's x offset), half 1 columns 16-31
      const long pp = row < np ? row : np - 1;
      int i, j, k;
      if (np <= 0x7FFFFFFFL) {
        const unsigned q = (unsigned)pp, um = (unsigned)m, qm = q / um;
        i = (int)(q - qm * um);
        j = (int)(qm % um);
        k = (int)(qm / um);
      } else {
        i = (int)(pp % m);
        j = (int)((pp / m) % m);
        k = (int)(pp / ((long)m * m));
      }
      const double h0 = -0.5 * (m - 1) * dx;
      const double x[3] = {h0 + i * dx, h0 + j * dx, h0 + k * dx};
      const double sc = 1.0 / 8.0;
      __align__(16) __nv_bfloat16 f[16];
      const int q = half;
      const double mq = cond[q];
      const double d0 = x[0] - cond[2 + 3 * q], d1 = x[1] - cond[3 + 3 * q], d2 = x[2] - cond[4 + 3 * q];
      const double rr = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
      const double g[12] = {d0 * sc, d1 * sc, d2 * sc, rr * sc, mq / (rr + mq), 2.0 * mq,
                            5.0 * cond[8 + 3 * q], 5.0 * cond[9 + 3 * q], 5.0 * cond[10 + 3 * q],
                            5.0 * cond[14 + 3 * q], 5.0 * cond[15 + 3 * q], 5.0 * cond[16 + 3 * q]};
      if (half == 0) {
        f[0] = to_bf16(x[0] * sc);
        f[1] = to_bf16(x[1] * sc);
        f[2] = to_bf16(x[2] * sc);
#pragma unroll
        for (int c = 0; c < 12; ++c) f[3 + c] = to_bf16(g[c]);
        f[15] = to_bf16((x[0] - cond[5]) * sc);
      } else {
#pragma unroll
        for (int c = 1; c < 12; ++c) f[c - 1] = to_bf16(g[c]);
#pragma unroll
        for (int c = 11; c < 16; ++c) f[c] = __float2bfloat16_rn(0.0f);
      }
#pragma unroll
      for (int c = 0; c < 2; ++c)
        *reinterpret_cast<uint4 *>(X + off(r, 16 * half + 8 * c)) = *reinterpret_cast<const uint4 *>(f + 8 * c);
    }
    float out = 0.0f;
    for (int l = 0; l < 4; ++l) {
      // the operand was written by the threads: make it visible to the
      // tensor core, then one thread issues the layer's MMA chain
      fence_async_smem();
      fence_before();
      team_sync(team);
      fence_after();
      if (failed[team]) break;   // read after the barrier: the same in every thread of the team
      if (tr == 0) {
        const uint32_t a0 = sbase + (uint32_t)((l == 0 ? X : A) - sm);
        const uint32_t b0 = sbase + (uint32_t)(l == 0 ? kOffW0 : kOffW + (l - 1) * 16 * kChunk);
        const int ks = fan_in(l) / 16;
        for (int s = 0; s < ks; ++s)
          mma(dcol, sdesc(a0 + s * 2 * kChunk), sdesc(b0 + s * 2 * kChunk), s > 0 ? 1u : 0u);
        commit(bar);
      }
      __syncwarp();
      // a warp whose wait ran out skips the (warp-collective) tensor-memory
      // reads; the team leaves the walk at its next barrier
      if (!__all_sync(0xffffffffu, tma::mbar_wait(bar, phase))) {
        failed[team] = 1;
        continue;
      }
      phase ^= 1u;
      fence_after();
      uint32_t acc[64];
      ld32(trow, acc);
      ld32(trow + 32, acc + 32);
      ld_wait();
      const float4 *bias = reinterpret_cast<const float4 *>(par + l * HID + 64 * half);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        // the bias (and w5) as 16-byte broadcast reads of shared memory
        const float4 b0 = bias[2 * c], b1 = bias[2 * c + 1];
        const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = silu(__uint_as_float(acc[8 * c + q]) + bb[q]);
        uint4 pk;
        pk.x = pack_bf16<CVT>(v[0], v[1]);
        pk.y = pack_bf16<CVT>(v[2], v[3]);
        pk.z = pack_bf16<CVT>(v[4], v[5]);
        pk.w = pack_bf16<CVT>(v[6], v[7]);
        if (l < 3) {
          *reinterpret_cast<uint4 *>(A + off(r, 64 * half + 8 * c)) = pk;
        } else {
          const uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
          const float4 *w5v = reinterpret_cast<const float4 *>(w5 + 64 * half + 8 * c);
          const float4 c0 = w5v[0], c1 = w5v[1];
          const float cc[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            out = fmaf(__uint_as_float(w[q] << 16), cc[2 * q], out);
            out = fmaf(__uint_as_float(w[q] & 0xFFFF0000u), cc[2 * q + 1], out);
          }
        }
      }
    }
    // out = A4 w5 + b5 from the two halves of the row
    if (half == 1) red[r] = out;
    team_sync(team);
    if (failed[team]) break;
    if (half == 0 && row < np) u[row] = uscale * (double)(out + red[r] + w5[HID]);
    // this tile's tensor-memory reads are done before the next tile's first
    // MMA overwrites the accumulator (the barrier at the next layer start)
    fence_before();
  }
  if (failed[team] && tr == 0) {
    // an MMA chain still in flight is waited for (bounded) before the
    // tensor memory is freed
    atomicOr(status, 1);
    tma::mbar_wait(bar, phase);
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
}


}  // namespace

struct nrgpu_mlp {
  int device;
  int max_batch;
  float *P, *G, *Mo, *Vo;  // master params, gradients, Adam moments
  __nv_bfloat16 *Wb;       // BF16 W1..W4
  __nv_bfloat16 *X;        // [max_batch][IN]
  float *Z[4];             // [max_batch][HID] silu' of the pre-activations (1 to 3)
  __nv_bfloat16 *Ab[4];    // [max_batch][HID] activations (1 to 3)
  __nv_bfloat16 *dZ[4];    // [max_batch][HID] pre-activation gradients
  float *out;
  double *loss;            // right after G, on the next 8 bytes
  double *cond;            // the conditioning table
  int ncond;
  int *d_tcstatus;         // a wait of the tensor-core forward ran out
  long adam_t;
};

namespace {

inline int nb(long n, int t = 256) { return (int)((n + t - 1) / t); }

RowsArgs rows_args(nrgpu_mlp *M, int n, const float *y, float *out) {
  RowsArgs a = {M->X, M->Wb, M->P, y, out, {}, {}, {}, M->G, M->loss, n};
  for (int l = 0; l < 4; ++l) {
    a.Z[l] = M->Z[l];
    a.A[l] = M->Ab[l];
    a.dZ[l] = M->dZ[l];
  }
  return a;
}

// network output of n rows already featurised in M->X
int forward(nrgpu_mlp *M, int n, float *out, cudaStream_t st) {
  NRGPU_CUDA_TRY(cudaFuncSetAttribute(mlp_rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsSmem));
  mlp_rows_kernel<false><<<nb(n, 128), kRowsThreads, kRowsSmem, st>>>(rows_args(M, n, nullptr, out));
  NRGPU_CUDA_TRY(cudaGetLastError());
  return NRGPU_OK;
}

int set_cond(nrgpu_mlp *M, const double *host_cond, int nsets) {
  if (nsets > M->ncond) {
    cudaFree(M->cond);
    if (cudaMalloc(&M->cond, sizeof(double) * 20 * nsets) != cudaSuccess) {
      M->cond = nullptr;
      M->ncond = 0;
      cudaGetLastError();
      return nrgpu_set_error(NRGPU_ERR_NOMEM, "conditioning table");
    }
    M->ncond = nsets;
  }
  NRGPU_CUDA_TRY(cudaMemcpy(M->cond, host_cond, sizeof(double) * 20 * nsets, cudaMemcpyHostToDevice));
  return NRGPU_OK;
}

}  // namespace

extern "C" int nrgpu_mlp_nparams(void) { return kNParams; }

extern "C" int nrgpu_mlp_create(int max_batch, nrgpu_mlp **out) {
  if (!out || max_batch < 64 || max_batch % 64) return nrgpu_set_error(NRGPU_ERR_ARG, "max_batch: a multiple of 64");
  nrgpu_mlp *M = (nrgpu_mlp *)calloc(1, sizeof(nrgpu_mlp));
  if (!M) return nrgpu_set_error(NRGPU_ERR_NOMEM, "host allocation");
  cudaGetDevice(&M->device);
  M->max_batch = max_batch;
  const size_t nh = (size_t)max_batch * HID;
  bool ok = cudaMalloc(&M->P, sizeof(float) * kNParams) == cudaSuccess &&
            cudaMalloc(&M->G, sizeof(float) * (kNParams + 3)) == cudaSuccess &&
            cudaMalloc(&M->Mo, sizeof(float) * kNParams) == cudaSuccess &&
            cudaMalloc(&M->Vo, sizeof(float) * kNParams) == cudaSuccess &&
            cudaMalloc(&M->Wb, sizeof(__nv_bfloat16) * (IN * HID + 3 * HID * HID)) == cudaSuccess &&
            cudaMalloc(&M->X, sizeof(__nv_bfloat16) * (size_t)max_batch * IN) == cudaSuccess &&
            cudaMalloc(&M->out, sizeof(float) * max_batch) == cudaSuccess &&
            cudaMalloc(&M->d_tcstatus, sizeof(int)) == cudaSuccess &&
            cudaMemset(M->d_tcstatus, 0, sizeof(int)) == cudaSuccess;
  for (int l = 0; l < 4 && ok; ++l)
    ok = (l == 3 || cudaMalloc(&M->Z[l], sizeof(float) * nh) == cudaSuccess) &&
         (l == 3 || cudaMalloc(&M->Ab[l], sizeof(__nv_bfloat16) * nh) == cudaSuccess) &&
         cudaMalloc(&M->dZ[l], sizeof(__nv_bfloat16) * nh) == cudaSuccess;
  M->loss = (double *)(M->G + (kNParams + 1) / 2 * 2);
  if (ok)
    ok = cudaMemset(M->P, 0, sizeof(float) * kNParams) == cudaSuccess &&
         cudaMemset(M->G, 0, sizeof(float) * (kNParams + 3)) == cudaSuccess &&
         cudaMemset(M->Mo, 0, sizeof(float) * kNParams) == cudaSuccess &&
         cudaMemset(M->Vo, 0, sizeof(float) * kNParams) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    nrgpu_mlp_destroy(M);
    return nrgpu_set_error(NRGPU_ERR_NOMEM, "device allocation of the network (batch %d)", max_batch);
  }
  *out = M;
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_destroy(nrgpu_mlp *M) {
  if (!M) return NRGPU_OK;
  cudaFree(M->P); cudaFree(M->G); cudaFree(M->Mo); cudaFree(M->Vo); cudaFree(M->Wb); cudaFree(M->X);
  cudaFree(M->out); cudaFree(M->cond);
  cudaFree(M->d_tcstatus);
  for (int l = 0; l < 4; ++l) {
    cudaFree(M->Z[l]);
    cudaFree(M->Ab[l]);
    cudaFree(M->dZ[l]);
  }
  free(M);
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_set_params(nrgpu_mlp *M, const float *host, int n) {
  if (!M || !host || n != kNParams) return nrgpu_set_error(NRGPU_ERR_ARG, "parameter count %d != %d", n, kNParams);
  NRGPU_CUDA_TRY(cudaMemcpy(M->P, host, sizeof(float) * kNParams, cudaMemcpyHostToDevice));
  NRGPU_CUDA_TRY(cudaMemset(M->Mo, 0, sizeof(float) * kNParams));
  NRGPU_CUDA_TRY(cudaMemset(M->Vo, 0, sizeof(float) * kNParams));
  M->adam_t = 0;
  refresh_bf16_kernel<<<nb(IN * HID + 3 * HID * HID), 256>>>(M->P, M->Wb);
  NRGPU_CUDA_TRY(cudaGetLastError());
  NRGPU_CUDA_TRY(cudaDeviceSynchronize());
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_get_params(nrgpu_mlp *M, float *host, int n) {
  if (!M || !host || n != kNParams) return nrgpu_set_error(NRGPU_ERR_ARG, "parameter count %d != %d", n, kNParams);
  NRGPU_CUDA_TRY(cudaDeviceSynchronize());
  NRGPU_CUDA_TRY(cudaMemcpy(host, M->P, sizeof(float) * kNParams, cudaMemcpyDeviceToHost));
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_set_conditions(nrgpu_mlp *M, const double *host_cond, int nsets) {
  if (!M || !host_cond || nsets < 1) return nrgpu_set_error(NRGPU_ERR_ARG, "bad conditioning table");
  return set_cond(M, host_cond, nsets);
}

extern "C" int nrgpu_mlp_features(nrgpu_mlp *M, const int *d_set, const int *d_pt, int n, int m, double dx,
                                  void *stream) {
  if (!M || !d_set || !d_pt || n < 1 || n > M->max_batch || m < 2 || !M->cond)
    return nrgpu_set_error(NRGPU_ERR_ARG, "bad feature arguments (conditioning table set?)");
  mlp_features_kernel<<<nb(n), 256, 0, (cudaStream_t)stream>>>(M->cond, d_set, d_pt, 0, n, Feat{m, dx}, M->X);
  NRGPU_CUDA_TRY(cudaGetLastError());
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_copy_features(nrgpu_mlp *M, int n, uint16_t *host) {
  if (!M || !host || n < 1 || n > M->max_batch) return nrgpu_set_error(NRGPU_ERR_ARG, "bad feature copy");
  NRGPU_CUDA_TRY(cudaDeviceSynchronize());
  NRGPU_CUDA_TRY(cudaMemcpy(host, M->X, sizeof(uint16_t) * (size_t)n * IN, cudaMemcpyDeviceToHost));
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_train_step(nrgpu_mlp *M, const float *d_y, int n, float lr, int update, float *loss,
                                    void *stream) {
  if (!M || !d_y || n < 64 || n % 64 || n > M->max_batch)
    return nrgpu_set_error(NRGPU_ERR_ARG, "batch %d: a multiple of 64 up to %d", n, M ? M->max_batch : 0);
  const cudaStream_t st = (cudaStream_t)stream;
  NRGPU_CUDA_TRY(cudaMemsetAsync(M->G, 0, sizeof(float) * (kNParams + 3), st));  // the gradients and the loss
  NRGPU_CUDA_TRY(cudaFuncSetAttribute(mlp_rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsSmem));
  NRGPU_CUDA_TRY(cudaFuncSetAttribute(mlp_weight_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmem));
  const RowsArgs a = rows_args(M, n, d_y, M->out);
  mlp_rows_kernel<true><<<nb(n, 128), kRowsThreads, kRowsSmem, st>>>(a);
  // row chunks: enough blocks (four layers each) for the SMs, at least 128
  // rows each so that the atomics of a block's 128 x 128 sums stay few
  const int chunk = max(128, (n + 36 * kGradRows - 1) / (36 * kGradRows) * kGradRows);
  mlp_weight_grad_kernel<<<dim3(4, nb(n, chunk)), 256, kGradSmem, st>>>(a, chunk);
  NRGPU_CUDA_TRY(cudaGetLastError());
  if (update) {
    M->adam_t++;
    AdamArgs q;
    q.lr = lr; q.b1 = 0.9f; q.b2 = 0.999f; q.eps = 1e-8f;
    q.c1 = (float)(1.0 / (1.0 - pow(0.9, (double)M->adam_t)));
    q.c2 = (float)(1.0 / (1.0 - pow(0.999, (double)M->adam_t)));
    adam_kernel<<<nb(kNParams), 256, 0, st>>>(M->P, M->G, M->Mo, M->Vo, M->Wb, q, kNParams);
    NRGPU_CUDA_TRY(cudaGetLastError());
  }
  if (loss) {
    double l;
    NRGPU_CUDA_TRY(cudaMemcpyAsync(&l, M->loss, sizeof l, cudaMemcpyDeviceToHost, st));
    NRGPU_CUDA_TRY(cudaStreamSynchronize(st));
    *loss = (float)l;
  }
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_gradients(nrgpu_mlp *M, float *host_grad, int n_params) {
  if (!M || !host_grad || n_params != kNParams) return nrgpu_set_error(NRGPU_ERR_ARG, "gradient buffer");
  NRGPU_CUDA_TRY(cudaDeviceSynchronize());
  NRGPU_CUDA_TRY(cudaMemcpy(host_grad, M->G, sizeof(float) * kNParams, cudaMemcpyDeviceToHost));
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_forward(nrgpu_mlp *M, int n, float *d_out, void *stream) {
  if (!M || !d_out || n < 16 || n % 16 || n > M->max_batch)
    return nrgpu_set_error(NRGPU_ERR_ARG, "rows %d: a multiple of 16 up to %d", n, M ? M->max_batch : 0);
  return forward(M, n, d_out, (cudaStream_t)stream);
}

extern "C" int nrgpu_mlp_predict_u(nrgpu_mlp *M, const double *host_cond, int m, double dx, double uscale, double *u,
                                   void *stream) {
  if (!M || !host_cond || !u || m < 2) return nrgpu_set_error(NRGPU_ERR_ARG, "bad prediction arguments");
  const cudaStream_t st = (cudaStream_t)stream;
  NRGPU_CUDA_TRY(cudaStreamSynchronize(st));  // the table is replaced below
  int e = set_cond(M, host_cond, 1);
  if (e) return e;
  const long np = (long)m * m * m;
  for (long first = 0; first < np; first += M->max_batch) {
    const int n = (int)min((long)M->max_batch, np - first);
    const int n16 = (n + 15) / 16 * 16;  // rows past np are computed and dropped
    mlp_features_kernel<<<nb(n16), 256, 0, st>>>(M->cond, nullptr, nullptr, first, n16, Feat{m, dx}, M->X);
    NRGPU_CUDA_TRY(cudaGetLastError());
    if ((e = forward(M, n16, M->out, st))) return e;
    scale_to_u_kernel<<<nb(n), 256, 0, st>>>(M->out, uscale, u + first, n);
    NRGPU_CUDA_TRY(cudaGetLastError());
  }
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_predict_u_fp32(nrgpu_mlp *M, const double *host_cond, int m, double dx, double uscale,
                                        double *u, void *stream) {
  if (!M || !host_cond || !u || m < 2) return nrgpu_set_error(NRGPU_ERR_ARG, "bad prediction arguments");
  const cudaStream_t st = (cudaStream_t)stream;
  NRGPU_CUDA_TRY(cudaStreamSynchronize(st));  // the table is replaced below
  int e = set_cond(M, host_cond, 1);
  if (e) return e;
  const long np = (long)m * m * m;
  NRGPU_CUDA_TRY(cudaFuncSetAttribute(mlp_forward_fp32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFSmem));
  mlp_forward_fp32_kernel<<<(unsigned)((np + kFR - 1) / kFR), 256, kFSmem, st>>>(M->cond, m, dx, M->P, uscale, u, np);
  NRGPU_CUDA_TRY(cudaGetLastError());
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_predict_u_tc(nrgpu_mlp *M, const double *host_cond, int m, double dx, double uscale,
                                      double *u, void *stream) {
  if (!M || !host_cond || !u || m < 2) return nrgpu_set_error(NRGPU_ERR_ARG, "bad prediction arguments");
  const cudaStream_t st = (cudaStream_t)stream;
  NRGPU_CUDA_TRY(cudaStreamSynchronize(st));  // the table is replaced below
  int e = set_cond(M, host_cond, 1);
  if (e) return e;
  static bool attr_set[64] = {};
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm < 1) {
    cudaGetLastError();
    nsm = 148;
  }
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    NRGPU_CUDA_TRY(cudaFuncSetAttribute(mlp_forward_tc_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::kSmem));
    attr_set[dev] = true;
  }
  const long np = (long)m * m * m;
  const long pairs = ((np + tc::kRows - 1) / tc::kRows + 1) / 2;
  const unsigned grid = (unsigned)(pairs < nsm ? pairs : nsm);
  NRGPU_CUDA_TRY(cudaMemsetAsync(M->d_tcstatus, 0, sizeof(int), st));
  mlp_forward_tc_kernel<0><<<grid, tc::kThreads, tc::kSmem, st>>>(M->cond, m, dx, M->P, uscale, u, np, M->d_tcstatus);
  NRGPU_CUDA_TRY(cudaGetLastError());
  return NRGPU_OK;
}

extern "C" int nrgpu_mlp_tc_status(nrgpu_mlp *M, int *timed_out) {
  if (!M || !timed_out) return nrgpu_set_error(NRGPU_ERR_ARG, "bad status arguments");
  NRGPU_CUDA_TRY(cudaDeviceSynchronize());
  NRGPU_CUDA_TRY(cudaMemcpy(timed_out, M->d_tcstatus, sizeof(int), cudaMemcpyDeviceToHost));
  return *timed_out ? nrgpu_set_error(NRGPU_ERR_TIMEOUT, "a wait of the tensor-core forward ran out") : NRGPU_OK;
}
