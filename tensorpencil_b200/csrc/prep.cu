// Plain ConvRot activation prep (x already in memory) and the int4 -> int8 weight
// expansion.  The kernel itself is in prep_common.cuh.
#include "prep_common.cuh"

using namespace tpb_prep;

namespace {

// 4 packed int4 bytes -> 8 int8 (element 2j in the low nibble, src/core/dtype.zig:146-149)
__device__ __forceinline__ uint2 w4_expand_word(uint32_t in) {
    // even nibbles -> bytes (n0,n2,n4,n6), odd -> (n1,n3,n5,n7); sign-extend
    // each nibble inside its byte: x | ((x & 8) * 30) sets bits 4..7.
    uint32_t e = in & 0x0f0f0f0fu;
    uint32_t o = (in >> 4) & 0x0f0f0f0fu;
    e |= (e & 0x08080808u) * 30u;
    o |= (o & 0x08080808u) * 30u;
    return make_uint2(__byte_perm(e, o, 0x5140), __byte_perm(e, o, 0x7362));   // n0 n1 n2 n3, n4 n5 n6 n7
}

// int4 -> int8 expansion of a packed weight: a thread takes BATCH pieces of 8 packed bytes with their loads in flight together, and
// writes 16 bytes beside its neighbours' (with 16 packed bytes a thread, every store touched half of its sectors).  Bound by HBM where the weight is
// large: 12288 x 3072 (56.6 MB, 8.7 us at 6.54 TB/s) 11.5 -> 9.7 us over weights and outputs that L2 does not hold (in a loop over one of them 7.4,
// its output then stays dirty in L2).  Four pieces where they still make five CTAs an SM, two below, where CTAs are too few and too coarse to share out
// evenly; us, 16 bytes a thread / four pieces / two: 12288 x 3072 11.5 / 9.7 / 9.8, 9216 x 2304 6.5 / 6.0 / 6.2; 2464 x 2816 3.4 / 3.7 / 3.0, 1872 x 4352
// 3.5 / 3.8 / 3.3, 1024 x 4096 3.0 / 3.3 / 2.3, 3728 x 512 2.1 / 2.4 / 1.8.
template <int BATCH>
__global__ void __launch_bounds__(256)
w4_expand_kernel(const uint2 *__restrict__ w4, uint4 *__restrict__ w8, size_t n_pieces) {
    tpb_grid_dep_launch();
    tpb_grid_dep_wait();
    const size_t first = (size_t)blockIdx.x * (256 * BATCH) + threadIdx.x;
    uint2 in[BATCH];
#pragma unroll
    for (int j = 0; j < BATCH; j++) {
        const size_t c = first + (size_t)(j * 256);
        in[j] = c < n_pieces ? __ldcg(w4 + c) : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int j = 0; j < BATCH; j++) {
        const size_t c = first + (size_t)(j * 256);
        if (c >= n_pieces) break;
        const uint2 lo = w4_expand_word(in[j].x), hi = w4_expand_word(in[j].y);
        w8[c] = make_uint4(lo.x, lo.y, hi.x, hi.y);
    }
}

template <typename T>
int launch_prep_t(tpb_handle_t h, cudaStream_t st, const T *x, int64_t m, int64_t k, int bits,
                  int8_t *q, float *act_scale, int32_t *act_sum) {
    PrepParams P = {};
    P.a = x;
    P.q = q;
    P.act_scale = act_scale;
    P.act_sum = act_sum;
    return launch_prep_op<T, OP_PLAIN, false>(h, st, P, m, k, bits);
}

}  // namespace

int tpb_launch_prep(tpb_handle_t h, cudaStream_t st, const void *x, int x_dtype, int64_t m,
                    int64_t k, int bits, int8_t *q, float *act_scale, int32_t *act_sum) {
    switch (x_dtype) {
        case TPB_F32:
            return launch_prep_t<float>(h, st, (const float *)x, m, k, bits, q, act_scale, act_sum);
        case TPB_F16:
            return launch_prep_t<__half>(h, st, (const __half *)x, m, k, bits, q, act_scale, act_sum);
        case TPB_BF16:
            return launch_prep_t<__nv_bfloat16>(h, st, (const __nv_bfloat16 *)x, m, k, bits, q,
                                                act_scale, act_sum);
    }
    return tpb_fail(h, TPB_ERR_INVALID_ARG, "prep: unsupported x_dtype %d", x_dtype);
}

int tpb_launch_w4_expand(tpb_handle_t h, cudaStream_t st, const void *w4, int64_t n, int64_t k,
                         int8_t *w8) {
    const size_t n_pieces = (size_t)n * (size_t)k / 16;  // 8 packed bytes each
    const int batch = n_pieces >= (size_t)5 * h->sm_count * (256 * 4) ? 4 : 2;
    const size_t grid = (n_pieces + 256 * batch - 1) / (256 * batch);
    if (grid > 0x7fffffffu) return tpb_fail(h, TPB_ERR_INVALID_ARG, "w4_expand: weight of %lld x %lld is too large", (long long)n, (long long)k);
    auto kern = batch == 4 ? w4_expand_kernel<4> : w4_expand_kernel<2>;
    TPB_CUDA(h, tpb_launch_pdl(kern, dim3((unsigned)grid), dim3(256), 0, st, (const uint2 *)w4, (uint4 *)w8, n_pieces));
    return TPB_OK;
}
