// Dequantisation of frozen low-bit weights into bf16, layer by layer, just before the layer's GEMMs read them.
//
// The reference's `training_precision` "4bit" and "8bit" load the student's linear layers through bitsandbytes as
// NF4 (block-wise absmax over 64 values, the absmax values themselves quantised a second time) or row-wise int8
// weights, which are then FROZEN: only embeddings, norms and the LM head keep training (classes/student/model.py:
// 138-148, 194-201). Here the packed weights stay resident and a layer's matrices are expanded into a rotating bf16
// buffer by these kernels before its forward and again before its backward; the tensor-core GEMMs then run on bf16
// as everywhere else.
//
//   NF4   byte = (code of element 2i) << 4 | code of element 2i+1; value = nf4[code] * absmax(block of 64)
//         absmax(block) = int8 code * scale(group of 256 blocks) + offset      (second-level quantisation)
//   int8  value = code * scale(row)
#include "../common/ptx.cuh"
#include "../common/host.cuh"

namespace b200 {
namespace quant {

__constant__ float kNF4[16] = {-1.0f, -0.6961928009986877f, -0.5250730514526367f, -0.39491748809814453f,
                               -0.28444138169288635f, -0.18477343022823334f, -0.09105003625154495f, 0.0f,
                               0.07958029955625534f, 0.16093020141124725f, 0.24611230194568634f, 0.33791524171829224f,
                               0.44070982933044434f, 0.5626170039176941f, 0.7229568362236023f, 1.0f};

// One launch expands up to MAX_PARTS matrices (the four of a decoder layer): their blocks form one index space, so that the
// short ones fill the tail of the long one, where four launches would each have their own ramp and tail.
constexpr int MAX_PARTS = 4;
struct Nf4Part {
  const uint8_t* packed;
  const int8_t* absmax_code;
  const float* absmax_scale;
  __nv_bfloat16* out;
  float offset;
  long long units;      // groups of eight values
  int end;              // blocks of this part and those before it
};
struct Nf4Parts { Nf4Part part[MAX_PARTS]; int n; };
struct Int8Part {
  const int8_t* code;
  const float* row_scale;
  __nv_bfloat16* out;
  int units_per_row;    // groups of eight values
  long long units;
  int end;
};
struct Int8Parts { Int8Part part[MAX_PARTS]; int n; };

// Bound by HBM and L2: 2.5 bytes a value. A thread takes four groups of eight values (4 packed bytes, 16 bytes of output), a
// block apart, so that every access of a warp is one run, and all of its loads are under way before the first is used; the
// blocks cover each part in order and none straddles two. Issue slots come next (two thirds of them at 10 instructions a value),
// so the table is indexed in bytes and a block holds one second-level scale. A TinyLlama layer (44 M values) 21.1 us alone and
// 24.6 behind large GEMMs, 218 M values 86 (5.3 / 6.3 TB/s); groups of 16 in two stores 32 bytes apart, walked by a resident
// grid: 23.8, 33.4, 107.
constexpr int UNITS = 4;
__global__ void __launch_bounds__(256) dequant_nf4_kernel(const __grid_constant__ Nf4Parts ps) {
  pdl_wait();
  pdl_trigger();
  __shared__ float lut[16];
  if (threadIdx.x < 16) lut[threadIdx.x] = kNF4[threadIdx.x];
  int m = 0;
  while ((int)blockIdx.x >= ps.part[m].end) ++m;
  const Nf4Part& p = ps.part[m];
  const long long base = (long long)(blockIdx.x - (m ? ps.part[m - 1].end : 0)) * (256 * UNITS);
  const int left = (int)min(p.units - base, (long long)(256 * UNITS));
  const uint32_t* src = reinterpret_cast<const uint32_t*>(p.packed) + base;
  const int8_t* code = p.absmax_code + (base >> 3);      // 64-value blocks,
  const float scale = p.absmax_scale[base >> 11], offset = p.offset;               // 256 of them a scale
  uint4* out = reinterpret_cast<uint4*>(p.out) + base;
  uint32_t q[UNITS];
  float am[UNITS];
#pragma unroll
  for (int k = 0; k < UNITS; ++k) {
    const int u = threadIdx.x + k * 256;
    if (u >= left) continue;
    q[k] = src[u];
    am[k] = (float)code[u >> 3];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < UNITS; ++k) {
    const int u = threadIdx.x + k * 256;
    if (u >= left) continue;
    const float a = am[k] * scale + offset;
    auto value = [&](uint32_t byte_offset) { return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(lut) + byte_offset); };
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {                        // of byte j the high half first
      const uint32_t hi = (q[k] >> (8 * j + 2)) & 0x3cu, lo = (j ? q[k] >> (8 * j - 2) : q[k] << 2) & 0x3cu;
      w[j] = pack_bf16x2(value(hi) * a, value(lo) * a);
    }
    out[u] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// As above, from 8 codes to 16 bytes a group; the row of a group is found from the block's first one. 44 M values 28 us, 218 M 112
// (groups of 16 in a resident grid, a 64-bit division each: 42, 173).
__global__ void __launch_bounds__(256) dequant_int8_kernel(const __grid_constant__ Int8Parts ps) {
  pdl_wait();
  pdl_trigger();
  int m = 0;
  while ((int)blockIdx.x >= ps.part[m].end) ++m;
  const Int8Part& p = ps.part[m];
  const long long base = (long long)(blockIdx.x - (m ? ps.part[m - 1].end : 0)) * (256 * UNITS);
  const int left = (int)min(p.units - base, (long long)(256 * UNITS));
  const uint2* src = reinterpret_cast<const uint2*>(p.code) + base;
  uint4* out = reinterpret_cast<uint4*>(p.out) + base;
  const long long row = base / p.units_per_row;
  const uint32_t first = (uint32_t)(base - row * p.units_per_row), per_row = p.units_per_row;
  const float* scale = p.row_scale + row;
  uint2 q[UNITS];
  float sc[UNITS];
#pragma unroll
  for (int k = 0; k < UNITS; ++k) {
    const int u = threadIdx.x + k * 256;
    if (u >= left) continue;
    q[k] = src[u];
    sc[k] = scale[(first + u) / per_row];
  }
#pragma unroll
  for (int k = 0; k < UNITS; ++k) {
    const int u = threadIdx.x + k * 256;
    if (u >= left) continue;
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t two = (j < 2 ? q[k].x : q[k].y) >> (16 * (j & 1));
      w[j] = pack_bf16x2((float)(int8_t)(two & 0xffu) * sc[k], (float)(int8_t)((two >> 8) & 0xffu) * sc[k]);
    }
    out[u] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// blocks of a part and those before it; 0: beyond a grid
static int blocks_to(long long end, long long units) {
  end += (units + 256 * UNITS - 1) / (256 * UNITS);
  return end > 0x7fffffffll ? 0 : (int)end;
}

}  // namespace quant
}  // namespace b200

extern "C" {
using namespace b200;

// n_parts (1 .. 4) matrices at once; every array has n_parts entries. counts: values per matrix, multiples of 64.
int b200_dequant_nf4(const void* const* packed, const void* const* absmax_code, const float* const* absmax_scale,
                     const float* offset, void* const* out, const long long* counts, int n_parts, cudaStream_t st) {
  if (!packed || !absmax_code || !absmax_scale || !offset || !out || !counts || n_parts < 1 || n_parts > quant::MAX_PARTS)
    return B200_ERR_ARG;
  quant::Nf4Parts ps{};
  ps.n = n_parts;
  int end = 0;
  for (int i = 0; i < n_parts; ++i) {
    if (!packed[i] || !absmax_code[i] || !absmax_scale[i] || !out[i] || counts[i] <= 0 || (counts[i] & 63) ||
        (reinterpret_cast<uintptr_t>(packed[i]) & 7) || (reinterpret_cast<uintptr_t>(out[i]) & 15))
      return B200_ERR_ARG;
    if (!(end = quant::blocks_to(end, counts[i] >> 3))) return B200_ERR_ARG;
    ps.part[i] = quant::Nf4Part{(const uint8_t*)packed[i], (const int8_t*)absmax_code[i], absmax_scale[i],
                                (__nv_bfloat16*)out[i], offset[i], counts[i] >> 3, end};
  }
  launch_pdl(quant::dequant_nf4_kernel, end, 256, 0, st, ps);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

int b200_dequant_int8(const void* const* code, const float* const* row_scale, void* const* out, const long long* rows,
                      const int* cols, int n_parts, cudaStream_t st) {
  if (!code || !row_scale || !out || !rows || !cols || n_parts < 1 || n_parts > quant::MAX_PARTS) return B200_ERR_ARG;
  quant::Int8Parts ps{};
  ps.n = n_parts;
  int end = 0;
  for (int i = 0; i < n_parts; ++i) {
    if (!code[i] || !row_scale[i] || !out[i] || rows[i] <= 0 || cols[i] <= 0 || (cols[i] & 15) ||
        (reinterpret_cast<uintptr_t>(code[i]) & 15) || (reinterpret_cast<uintptr_t>(out[i]) & 15))
      return B200_ERR_ARG;
    const long long units = rows[i] * (cols[i] >> 3);
    if (!(end = quant::blocks_to(end, units))) return B200_ERR_ARG;
    ps.part[i] = quant::Int8Part{(const int8_t*)code[i], row_scale[i], (__nv_bfloat16*)out[i], cols[i] >> 3, units, end};
  }
  launch_pdl(quant::dequant_int8_kernel, end, 256, 0, st, ps);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}
}
