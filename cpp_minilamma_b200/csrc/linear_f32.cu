// y[M, N] = x[M, K] . W[N, K]^T in true float32 for the few rows of a decode step: a weight-streaming kernel.
//
// Bound: reading W once from HBM (1B shape, 4 rows, in a CUDA graph, us, this kernel / the library / the bytes at the copy
// peak: q/k/v 7.0 / 39.7 / 3.9, o 5.3 / 24.3 / 2.6, gate/up 25.0 / 68.6 / 20.6, down 13.6 / 63.0 / 10.3, head 156 / 302 / 161;
// 8 rows: 9.8 / 36.1, 6.6 / 23.6, 35.4 / 69.0, 17.7 / 63.6, 228 / 313).  Up to about 20 rows the multiplications fit under that (M FMAs a weight of 4 bytes),
// so the kernel is laid out for bytes in flight: a warp owns 4 weight rows and a slice of K, a lane 16 contiguous bytes of
// each 512-byte run, and U runs of all four rows are asked for before the first is used.  The activations come through
// the L1 cache, where the warps of a block find the same lines.  Products of two neighbouring k are formed by one
// fma.rn.f32x2, whose halves are added at the end; a lane's sums are then added over the lanes and, in slice order, over
// the warps that share the rows, so a result does not depend on the run.  Long sums fall apart into 64 parts and more
// that way: the error against 64 bits is smaller than that of a chain over K.
//
// The reference calls cublasSgemm with rows = 1 for every linear (src/cuda_matmul.cc:181-186).
#include "common.cuh"

namespace mll {

enum : int { FEPI_F32 = 1, FEPI_SWIGLU = 2, FEPI_GEGLU = 4 };  // numbered as the bfloat16 kernels' epilogues
constexpr int F_WARPS = 8, F_ROWS = 4;
constexpr int F_MAX_M = 16;

struct LinearF32Args {
  const float* x;     // [M, K]
  const float* w;     // [N, K]
  const float* bias;  // optional [N]
  float* out;         // [M, N] (gated epilogues: [M, N / 2])
  int M, N, K, epilogue;
  int slices_log2;    // warps of a block that share weight rows, each with a slice of K
  int slice;          // k elements of a slice, a multiple of 128
};

__device__ __forceinline__ unsigned long long f_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ ulonglong2 f_stream(const float* p) {
  ulonglong2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ ulonglong2 f_keep(const float* p) {
  ulonglong2 v;
  asm volatile("ld.global.nc.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
  return v;
}

// Sums N values a lane over the lanes of a warp: at every step a lane gives one half of its values away and adds the other
// lane's share of the rest.  v[0 .. N / 32 - 1] (one at least) are left; the index of the first among the N is returned.
template <int N, int OFF>
__device__ __forceinline__ int f_lane_sums(float* v, int lane) {
  if constexpr (OFF == 0) {
    return 0;
  } else if constexpr (N > 1) {
    const bool upper = lane & OFF;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      const float give = upper ? v[i] : v[i + N / 2], keep = upper ? v[i + N / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, OFF);
    }
    return (upper ? N / 2 : 0) + f_lane_sums<N / 2, OFF / 2>(v, lane);
  } else {
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], OFF);
    return f_lane_sums<1, OFF / 2>(v, lane);
  }
}

// MT: batch rows a warp works on (rows beyond M repeat the last one and are not stored); U: 128-element runs in flight;
// OCC: blocks a multiprocessor that the register allocation aims at.  From 5 rows on the sums alone take 64 registers and
// more, and what sets the pace is the activations' way through the L1 cache (as many bytes a row as a weight row has):
// fewer warps with more loads in flight each are the better use of the registers there (gate/up of the 1B shape, 8 rows:
// 35.4 us against 37.7 with two blocks a multiprocessor).
template <int MT, int U, int OCC>
__global__ void __launch_bounds__(F_WARPS * 32, OCC) linear_f32_kernel(LinearF32Args a) {
  constexpr int NV = F_ROWS * MT;
  __shared__ float red[F_WARPS][NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slices = 1 << a.slices_log2, groups = F_WARPS >> a.slices_log2;
  const int group = warp >> a.slices_log2, slice = warp & (slices - 1);
  const bool gated = a.epilogue != FEPI_F32;
  // a warp's weight rows: four neighbours, or gate rows j, j + 1 and their up rows, 8 further (blocks of 8 interleaved)
  auto row_of = [&](int unit, int r) {
    if (!gated) return unit * F_ROWS + r;
    const int pair = unit * (F_ROWS / 2) + r % (F_ROWS / 2);
    return (pair >> 3) * 16 + (pair & 7) + r / (F_ROWS / 2) * 8;
  };
  const int unit = blockIdx.x * groups + group;
  const int begin = slice * a.slice, end = min(a.K, begin + a.slice);

  const float* wr[F_ROWS];
#pragma unroll
  for (int r = 0; r < F_ROWS; ++r) wr[r] = a.w + (size_t)min(row_of(unit, r), a.N - 1) * a.K + lane * 4;
  const float* x0 = a.x + lane * 4;  // at most 16 rows: 32-bit offsets
  unsigned long long acc[F_ROWS][MT];
#pragma unroll
  for (int r = 0; r < F_ROWS; ++r)
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[r][m] = 0ull;

  int k = begin;
  for (; k + U * 128 <= end; k += U * 128) {
    ulonglong2 w[U][F_ROWS];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < F_ROWS; ++r) w[u][r] = f_stream(wr[r] + k + u * 128);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const ulonglong2 x = f_keep(x0 + min(m, a.M - 1) * a.K + k + u * 128);
#pragma unroll
        for (int r = 0; r < F_ROWS; ++r) acc[r][m] = f_fma2(w[u][r].y, x.y, f_fma2(w[u][r].x, x.x, acc[r][m]));
      }
  }
  for (; k < end; k += 128) {
    const bool in = k + lane * 4 < end;  // K is a multiple of 4
    ulonglong2 w[F_ROWS];
#pragma unroll
    for (int r = 0; r < F_ROWS; ++r) w[r] = in ? f_stream(wr[r] + k) : make_ulonglong2(0ull, 0ull);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const ulonglong2 x = in ? f_keep(x0 + min(m, a.M - 1) * a.K + k) : make_ulonglong2(0ull, 0ull);
#pragma unroll
      for (int r = 0; r < F_ROWS; ++r) acc[r][m] = f_fma2(w[r].y, x.y, f_fma2(w[r].x, x.x, acc[r][m]));
    }
  }

  float v[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const unsigned long long s = acc[i / MT][i % MT];
    v[i] = __uint_as_float((unsigned)s) + __uint_as_float((unsigned)(s >> 32));
  }
  const int at = f_lane_sums<NV, 16>(v, lane);  // index of this lane's first value
  constexpr int LEFT = NV > 32 ? NV / 32 : 1;
#pragma unroll
  for (int i = 0; i < LEFT; ++i) red[warp][at + i] = v[i];  // lanes that hold the same value write the same word
  __syncthreads();

  // over the slices, in their order; neighbouring threads take neighbouring columns
  const int per_unit = gated ? F_ROWS / 2 : F_ROWS, columns = groups * per_unit;
  const int half = a.N >> 1;
  for (int i = threadIdx.x; i < columns * a.M; i += F_WARPS * 32) {
    const int m = i / columns, g = (i % columns) / per_unit, r = i % per_unit;
    const int u = blockIdx.x * groups + g;
    float s = 0.f, s2 = 0.f;
    for (int j = 0; j < slices; ++j) {
      s += red[(g << a.slices_log2) + j][r * MT + m];
      if (gated) s2 += red[(g << a.slices_log2) + j][(r + F_ROWS / 2) * MT + m];
    }
    if (gated) {
      const int col = u * (F_ROWS / 2) + r;
      if (col < half)
        a.out[(size_t)m * half + col] = gate_act_mul<false>(a.epilogue == FEPI_GEGLU ? GATE_ACT_GELU_TANH : GATE_ACT_SILU, s, s2);
    } else {
      const int col = u * F_ROWS + r;
      if (col < a.N) a.out[(size_t)m * a.N + col] = a.bias ? s + a.bias[col] : s;
    }
  }
}

template <int MT, int U, int OCC>
int launch_linear_f32(LinearF32Args a, int slices, cudaStream_t stream) {
  const int units = (a.N + F_ROWS - 1) / F_ROWS;
  if (slices <= 0) {
    // As many slices as still let all blocks be resident at once (o of the 1B shape, 4 rows: 8.7 us unsplit, 5.3 in four,
    // 6.1 in eight; 256 x 192, 9 rows: 4.3 unsplit, 3.1 in four).  A matrix that takes several waves anyway: slices of 1,024, four
    // at most, where two blocks share a multiprocessor (its 128,256-row head: 164 us unsplit, 156 in two, 168 in four; 131,072 x
    // 512, one row: 39 unsplit, 62 in two), else none.
    const int resident = mll_sm_count() * OCC;
    slices = 1;
    if ((units + F_WARPS - 1) / F_WARPS <= resident) {
      while (slices < F_WARPS && (units * slices * 2 + F_WARPS - 1) / F_WARPS <= resident && a.K / (slices * 2) >= 32) slices *= 2;
    } else if (OCC > 1) {
      while (slices < 4 && a.K / (slices * 2) >= 1024) slices *= 2;
    }
  }
  MLL_REQUIRE(slices == 1 || slices == 2 || slices == 4 || slices == 8, "linear_f32: %d slices", slices);
  while ((1 << a.slices_log2) < slices) ++a.slices_log2;
  const int runs = (a.K + 127) / 128;
  a.slice = (runs + slices - 1) / slices * 128;
  const int groups = F_WARPS / slices, blocks = (units + groups - 1) / groups;
  MLL_LAUNCH((linear_f32_kernel<MT, U, OCC>), dim3((unsigned)blocks), F_WARPS * 32, 0, stream, a);
  MLL_LAUNCH_CHECK();
  return 0;
}

}  // namespace mll

// Whether mll_linear_f32 takes this problem: at most 16 rows, rows of W and x that start on 16-byte boundaries.  From 9
// rows on the multiplications and the activations' loads set the pace, and tall matrices are left to the library (16
// rows, us, this kernel / the library: 1B q/k/v 18.3 / 33.4, o 10.9 / 24.2, gate/up 65 / 69, head 433 / 373; 8B gate/up,
// 28,672 rows, 208 / 202).
MLL_API int mll_linear_f32_supported(int M, int N, int K, int epilogue) {
  if (M < 1 || M > mll::F_MAX_M || N < 1 || K < 4 || K % 4 != 0 || (M > 8 && N > 16384)) return 0;
  if (epilogue == mll::FEPI_F32) return 1;
  return (epilogue == mll::FEPI_SWIGLU || epilogue == mll::FEPI_GEGLU) && N % 16 == 0;
}

// Whether it takes this problem and is the faster way for a product without an epilogue (us, the library / here): short rows of a tall matrix are not what
// the kernel is laid out for (8 rows, 16,384 x 64 5.1 / 7.5; 6,144 x 256 9.3 / 5.4), from 9 rows on no short rows are (16 rows, 64 x
// 64 2.6 / 3.3; 1,024 x 128 4.7 / 3.0) and the tallest matrices need long ones (16 rows, 12,288 x 512 19.6 / 17.8; 16,384 x 1,024
// 36.8 / 39.8; x 2,048 70 / 66).
MLL_API int mll_linear_f32_pays(int M, int N, int K) {
  if (!mll_linear_f32_supported(M, N, K, mll::FEPI_F32)) return 0;
  if (M <= 4) return 1;
  if (M <= 8) return K >= 256 || N <= 4096;
  return K >= (N <= 4096 ? 128 : 256) && (N <= 12288 || K >= 2048);
}

// x: float32 [M, K]; w: float32 [N, K]; bias: optional float32 [N]; out: float32 [M, N] (epilogue 1), or [M, N / 2] =
// silu(gate) * up with gate and up rows of w interleaved in blocks of 8 (2; 4: gelu in its tanh form), without a bias.
// slices: warps that share weight rows (1, 2, 4 or 8), 0 = choose.
MLL_API int mll_linear_f32(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int epilogue,
                           int slices, cudaStream_t stream) {
  MLL_REQUIRE(mll_linear_f32_supported(M, N, K, epilogue), "linear_f32: unsupported sizes M=%d N=%d K=%d epilogue %d", M, N, K,
              epilogue);
  MLL_REQUIRE(((uintptr_t)x | (uintptr_t)w) % 16 == 0, "linear_f32: operands must be 16-byte aligned");
  MLL_REQUIRE(epilogue == mll::FEPI_F32 || bias == nullptr, "linear_f32: the gated epilogues take no bias");
  mll::LinearF32Args a{x, w, bias, out, M, N, K, epilogue, 0, 0};
  if (M <= 1) return mll::launch_linear_f32<1, 4, 2>(a, slices, stream);
  if (M <= 2) return mll::launch_linear_f32<2, 4, 2>(a, slices, stream);
  if (M <= 4) return mll::launch_linear_f32<4, 4, 2>(a, slices, stream);
  if (M <= 8) return mll::launch_linear_f32<8, 4, 1>(a, slices, stream);
  return mll::launch_linear_f32<16, 1, 1>(a, slices, stream);
}
