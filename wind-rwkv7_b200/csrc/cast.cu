// Several tensors converted between fp32 and bf16, or copied, in one launch: the time mixer's parameters (about thirty, from 64 to
// C*C elements) before its kernels, to bf16 and, those of the GroupNorm and the bonus, to one fp32 tensor.  (Weight gradients need none:
// they come out of their products in fp32.  bf16 -> fp32 is there for callers of the C ABI.)  A thread takes 8 elements (one
// 16-byte and one 32-byte access), a CTA a tile of 2048; the tiles of all tensors are numbered through.  Bound by DRAM: 18 MB
// at C = 768 take 5.4 us (torch's multi-tensor copy, which cuts tensors into tiles of 65536 elements for 46 CTAs: 18 us).
#include "expand_loras.h"
#include "mma_bf16.cuh"
#include "wkv7_kernels.h"

namespace wkv7 {

constexpr int CAST_TILE = 2048;

__global__ void __launch_bounds__(CAST_TILE / 8) cast_kernel(const __grid_constant__ CastParams p) {
    stream_order();
    long long tile = blockIdx.x;
    int t = 0;
    for (; t < p.count; ++t) {
        const long long n = (p.numel[t] + CAST_TILE - 1) / CAST_TILE;
        if (tile < n) break;
        tile -= n;
    }
    const long long at = tile * CAST_TILE + threadIdx.x * 8;
    if (at >= p.numel[t]) return;
    float f[8];
    if (p.kind[t] == 1) {
        unpack8(*reinterpret_cast<const uint4*>((const bf16*)p.src[t] + at), f);
    } else {
        const float4 a = *reinterpret_cast<const float4*>((const float*)p.src[t] + at), b = *reinterpret_cast<const float4*>((const float*)p.src[t] + at + 4);
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
    if (p.kind[t] == 0) {
        *reinterpret_cast<uint4*>((bf16*)p.dst[t] + at) = pack8(f);
    } else {
        *reinterpret_cast<float4*>((float*)p.dst[t] + at) = make_float4(f[0], f[1], f[2], f[3]);
        *reinterpret_cast<float4*>((float*)p.dst[t] + at + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
}

int launch_cast(const CastParams& p, cudaStream_t stream) {
    long long tiles = 0;
    for (int i = 0; i < p.count; ++i) tiles += (p.numel[i] + CAST_TILE - 1) / CAST_TILE;
    if (tiles > 0x7fffffffLL) return kTooLarge;
    return launch(cast_kernel, dim3((unsigned)tiles), CAST_TILE / 8, 0, stream, p) ? kOk : kLaunchFailed;
}

}  // namespace wkv7
