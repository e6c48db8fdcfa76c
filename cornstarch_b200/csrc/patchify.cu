// Patches of an image as rows of a matrix: out[(b, gy, gx)][(c, y, x)] = in[b][c][gy * ph + y][gx * pw + x], the rest of a row zeros.
// What makes a convolution whose stride is its kernel size a GEMM.  A thread gathers the eight elements of one 16-byte store; a warp's
// stores are 512 consecutive bytes, its loads runs of pw elements (VEC2: in pairs, where every run starts on a 4-byte boundary).
// Latency bounds it at the sizes in use (729 patches of 588: 1.7 MB, 4 us), so eight loads per thread are in flight.
//
// Part of what replaces nn.Conv2d of the reference's vision encoders (HF SiglipVisionEmbeddings and its kin).
#include <cuda_bf16.h>

#include "host.h"

namespace csb {

struct PatchifyParams {
  const __nv_bfloat16* in;
  __nv_bfloat16* out;
  long sb, sc, sh;  // strides of image, channel and row, in elements
  int C, gh, gw, ph, pw, ld;
  long n8;  // 16-byte pieces of the output
};

template <bool VEC2>
__global__ void __launch_bounds__(256) patchify_kernel(const PatchifyParams p) {
  const int pieces = p.ld >> 3, plane = p.ph * p.pw, K = p.C * plane;
  for (long i = blockIdx.x * 256L + threadIdx.x; i < p.n8; i += gridDim.x * 256L) {
    const long row = i / pieces;
    const int k0 = static_cast<int>(i - row * pieces) * 8;
    const long b = row / (p.gh * p.gw);
    const int g = static_cast<int>(row - b * (p.gh * p.gw)), gy = g / p.gw, gx = g - gy * p.gw;
    const __nv_bfloat16* base = p.in + b * p.sb + static_cast<long>(gy) * p.ph * p.sh + static_cast<long>(gx) * p.pw;
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t pair = 0u;
      if constexpr (VEC2) {  // pw is even: the two elements of a pair are neighbours of one run, and K is even
        const int k = k0 + 2 * j;
        if (k < K) {
          const int c = k / plane, r = k - c * plane, y = r / p.pw, x = r - y * p.pw;
          pair = *reinterpret_cast<const uint32_t*>(base + c * p.sc + y * p.sh + x);
        }
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = k0 + 2 * j + h;
          if (k < K) {
            const int c = k / plane, r = k - c * plane, y = r / p.pw, x = r - y * p.pw;
            pair |= static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(base + c * p.sc + y * p.sh + x)) << (16 * h);
          }
        }
      }
      w[j] = pair;
    }
    reinterpret_cast<uint4*>(p.out)[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

}  // namespace csb

// in: B images of C channels with the given strides (elements; pixels of a row adjacent), at least gh * ph rows of gw * pw pixels;
// out: [B * gh * gw][ld], ld >= C * ph * pw a multiple of 8, 16-byte aligned.  vec2: base, strides and pw allow 4-byte loads.
CSB_API int csb_patchify(const void* in, void* out, long sb, long sc, long sh, int B, int C, int gh, int gw, int ph, int pw, int ld, int vec2,
                         void* stream) {
  using namespace csb;
  if (B < 1 || C < 1 || gh < 1 || gw < 1 || ph < 1 || pw < 1 || ld % 8 || ld < (long)C * ph * pw || (reinterpret_cast<uintptr_t>(out) & 15))
    return CSB_ERR_BAD_ARG;
  if (vec2 && ((reinterpret_cast<uintptr_t>(in) & 3) || (sb | sc | sh | pw) & 1)) return CSB_ERR_BAD_ARG;
  if ((long)gh * gw > 0x7fffffffL || (long)C * ph * pw > 0x7fffffffL) return CSB_ERR_TOO_LARGE;
  PatchifyParams p{reinterpret_cast<const __nv_bfloat16*>(in), reinterpret_cast<__nv_bfloat16*>(out), sb, sc, sh, C, gh, gw, ph, pw, ld,
                   (long)B * gh * gw * (ld / 8)};
  long blocks = (p.n8 + 255) / 256;
  if (blocks > (long)sm_count() * 8) blocks = (long)sm_count() * 8;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (vec2) patchify_kernel<true><<<(unsigned)blocks, 256, 0, s>>>(p);
  else patchify_kernel<false><<<(unsigned)blocks, 256, 0, s>>>(p);
  return launch_result();
}
