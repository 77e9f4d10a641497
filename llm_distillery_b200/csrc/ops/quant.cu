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

// One launch expands up to MAX_PARTS matrices (the four of a decoder layer): their 16-value groups form one index space,
// so that the short ones fill the tail of the long one. A TinyLlama layer (44 M values) took 34 us as four launches, each
// with its own ramp and tail; its bytes need 17.
constexpr int MAX_PARTS = 4;
struct Nf4Part {
  const uint8_t* packed;
  const int8_t* absmax_code;
  const float* absmax_scale;
  __nv_bfloat16* out;
  float offset;
  long long end;        // groups of this part and those before it
};
struct Nf4Parts { Nf4Part part[MAX_PARTS]; int n; };
struct Int8Part {
  const int8_t* code;
  const float* row_scale;
  __nv_bfloat16* out;
  int groups_per_row;
  long long end;
};
struct Int8Parts { Int8Part part[MAX_PARTS]; int n; };

// 16 values (8 packed bytes) per thread; sizes are multiples of 64, so a thread never straddles a block.
__global__ void __launch_bounds__(256) dequant_nf4_kernel(const __grid_constant__ Nf4Parts ps) {
  pdl_wait();
  pdl_trigger();
  __shared__ float lut[16];
  if (threadIdx.x < 16) lut[threadIdx.x] = kNF4[threadIdx.x];
  __syncthreads();
  const long long total = ps.part[ps.n - 1].end;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    int m = 0;
    while (i >= ps.part[m].end) ++m;
    const Nf4Part& p = ps.part[m];
    const long long g = m ? i - ps.part[m - 1].end : i;
    const long long blk = g >> 2;  // 64-value block
    const float am = (float)p.absmax_code[blk] * p.absmax_scale[blk >> 8] + p.offset;
    const uint2 q = reinterpret_cast<const uint2*>(p.packed)[g];
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t byte = ((j < 4 ? q.x : q.y) >> (8 * (j & 3))) & 0xffu;
      w[j] = pack_bf16x2(lut[byte >> 4] * am, lut[byte & 15u] * am);
    }
    uint4* o = reinterpret_cast<uint4*>(p.out + (g << 4));
    o[0] = make_uint4(w[0], w[1], w[2], w[3]);
    o[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// 16 values per thread; row lengths are multiples of 16.
__global__ void __launch_bounds__(256) dequant_int8_kernel(const __grid_constant__ Int8Parts ps) {
  pdl_wait();
  pdl_trigger();
  const long long total = ps.part[ps.n - 1].end;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    int m = 0;
    while (i >= ps.part[m].end) ++m;
    const Int8Part& p = ps.part[m];
    const long long g = m ? i - ps.part[m - 1].end : i;
    const float sc = p.row_scale[g / p.groups_per_row];
    const uint4 q = reinterpret_cast<const uint4*>(p.code)[g];
    const uint32_t words[4] = {q.x, q.y, q.z, q.w};
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t two = words[j >> 1] >> (16 * (j & 1));
      w[j] = pack_bf16x2((float)(int8_t)(two & 0xffu) * sc, (float)(int8_t)((two >> 8) & 0xffu) * sc);
    }
    uint4* o = reinterpret_cast<uint4*>(p.out + (g << 4));
    o[0] = make_uint4(w[0], w[1], w[2], w[3]);
    o[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

static int grid_for(long long items) {
  long long b = (items + 255) / 256;
  const long long cap = (long long)sm_count() * 8;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
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
  long long end = 0;
  for (int i = 0; i < n_parts; ++i) {
    if (!packed[i] || !absmax_code[i] || !absmax_scale[i] || !out[i] || counts[i] <= 0 || (counts[i] & 63) ||
        (reinterpret_cast<uintptr_t>(packed[i]) & 7) || (reinterpret_cast<uintptr_t>(out[i]) & 15))
      return B200_ERR_ARG;
    end += counts[i] >> 4;
    ps.part[i] = quant::Nf4Part{(const uint8_t*)packed[i], (const int8_t*)absmax_code[i], absmax_scale[i],
                                (__nv_bfloat16*)out[i], offset[i], end};
  }
  launch_pdl(quant::dequant_nf4_kernel, quant::grid_for(end), 256, 0, st, ps);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

int b200_dequant_int8(const void* const* code, const float* const* row_scale, void* const* out, const long long* rows,
                      const int* cols, int n_parts, cudaStream_t st) {
  if (!code || !row_scale || !out || !rows || !cols || n_parts < 1 || n_parts > quant::MAX_PARTS) return B200_ERR_ARG;
  quant::Int8Parts ps{};
  ps.n = n_parts;
  long long end = 0;
  for (int i = 0; i < n_parts; ++i) {
    if (!code[i] || !row_scale[i] || !out[i] || rows[i] <= 0 || cols[i] <= 0 || (cols[i] & 15) ||
        (reinterpret_cast<uintptr_t>(code[i]) & 15) || (reinterpret_cast<uintptr_t>(out[i]) & 15))
      return B200_ERR_ARG;
    end += rows[i] * (cols[i] >> 4);
    ps.part[i] = quant::Int8Part{(const int8_t*)code[i], row_scale[i], (__nv_bfloat16*)out[i], cols[i] >> 4, end};
  }
  launch_pdl(quant::dequant_int8_kernel, quant::grid_for(end), 256, 0, st, ps);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}
}
