// Per-token glue of the Llama decode step around the matvec kernels: embedding row, RoPE + KV
// append, split-KV GQA attention, greedy argmax. All read the position / token from device memory
// so one captured CUDA graph serves every step. Arithmetic follows ALICE-LLM src/llama3.rs:
// apply_rope :5323-5333, KvCache::append :4773, gqa_attention :5431-5690 (scores q.k/sqrt(d),
// softmax, weighted V sum; evaluated here as an online softmax over KV splits, which reorders
// the f32 sums but not the math).
#include "common.cuh"
#include "glue.cuh"
#include "attn_body.cuh"

namespace alice {

// hidden[c] = d * q of row `token` of a Q8_0 table (dequantize_q8_0, src/gguf.rs:990-1004); the
// CPU model dequantizes the whole table at load (src/llama3.rs:12890) and copies a row per token.
__global__ void __launch_bounds__(256) embed_q8_0_kernel(const __grid_constant__ EmbedArgs a) {
    __shared__ double red[8];
    pdl_launch_dependents();   // the next kernel may become resident (and prefetch its weights) while this one waits
    pdl_wait();
    const uint32_t k = blockIdx.x;   // a CTA per token of the batch
    if (threadIdx.x < 64) rope_table_entry(a.rope_tab + (size_t)k * 128, threadIdx.x, (uint32_t)*a.pos + k, a.rope_freq);
    // one thread per 34-byte block (f16 scale + 32 int8): 17 independent 16-bit loads, so the row costs one memory
    // round trip instead of one per element
    const uint32_t nblk = a.cols / 32;
    uint32_t t = (uint32_t)a.tokens[k];
    if (t >= a.vocab) t = 0;
    for (uint32_t b = threadIdx.x; b < nblk; b += blockDim.x) {
        const unsigned short* src = reinterpret_cast<const unsigned short*>(a.table + (size_t)t * nblk * 34 + (size_t)b * 34);
        unsigned short h[17];
#pragma unroll
        for (int j = 0; j < 17; j++) h[j] = __ldg(src + j);
        const float d = f16_bits_to_f32(h[0]);
        float* out = a.hidden + (size_t)k * a.cols + (size_t)b * 32;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            out[2 * j] = __fmul_rn(d, (float)(int8_t)(h[1 + j] & 0xff));
            out[2 * j + 1] = __fmul_rn(d, (float)(int8_t)(h[1 + j] >> 8));
        }
    }
    if (a.pub.mode == PUB_VECTOR && (a.pub.dst.qs != nullptr || a.pub.dst.xn != nullptr)) {
        __threadfence();
        __syncthreads();
        publish_vector<8, 0>(a.pub, red, k);
    }
}

// RoPE (apply_rope / apply_rope_neox, src/llama3.rs:5323-5333, 5367-5378): pairs (i, i+1), or (i, i + d/2)
// for NeoX, freq = 1 / theta^(i_even / d), angle = pos * freq; a lane owns dims 4*lane .. 4*lane+3 of a
// head vector (head_dim = 128, so a NeoX partner sits in lane ^ 16).
template <int GROUP>
__global__ void __launch_bounds__(AD_WARPS * 32, 16 / AD_WARPS) attn_decode_kernel(const __grid_constant__ AttnArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    pdl_launch_dependents();   // the next kernel may become resident (and prefetch its weights) while this one waits
    pdl_wait();
    attn_decode_body<GROUP>(a, blockIdx.x, blockIdx.y, reinterpret_cast<AttnSmem<GROUP>*>(smem));
}

static void launch_cfg(cudaLaunchConfig_t& lc, cudaLaunchAttribute* at, dim3 grid, dim3 block, cudaStream_t st, bool pdl) {
    lc = {};
    lc.gridDim = grid; lc.blockDim = block; lc.dynamicSmemBytes = 0; lc.stream = st;
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = pdl ? 1 : 0;
}

cudaError_t launch_embed_q8_0(const EmbedArgs& a, cudaStream_t st, bool pdl) {
    cudaLaunchConfig_t lc; cudaLaunchAttribute at[1];
    launch_cfg(lc, at, dim3(a.batch), dim3(256), st, pdl);
    return cudaLaunchKernelEx(&lc, embed_q8_0_kernel, a);
}

template <int GROUP>
static cudaError_t launch_decode(const AttnArgs& a, cudaStream_t st, bool pdl) {
    static bool done[64] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev >= 64 || !done[dev]) {
        err = cudaFuncSetAttribute(attn_decode_kernel<GROUP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AttnSmem<GROUP>));
        if (err != cudaSuccess) return err;
        if (dev < 64) done[dev] = true;
    }
    cudaLaunchConfig_t lc; cudaLaunchAttribute at[1];
    launch_cfg(lc, at, dim3(a.shape.num_kv_heads, a.nsplit), dim3(AD_WARPS * 32), st, pdl);
    lc.dynamicSmemBytes = sizeof(AttnSmem<GROUP>);
    return cudaLaunchKernelEx(&lc, attn_decode_kernel<GROUP>, a);
}

cudaError_t launch_attention(const AttnArgs& a, cudaStream_t st, bool pdl) {
    const AttnShape& s = a.shape;
    if (s.head_dim != 128 || s.num_heads % s.num_kv_heads) return cudaErrorInvalidValue;
    const uint32_t group = s.num_heads / s.num_kv_heads;
    switch (group) {
        case 1: return launch_decode<1>(a, st, pdl);
        case 2: return launch_decode<2>(a, st, pdl);
        case 4: return launch_decode<4>(a, st, pdl);
        case 5: return launch_decode<5>(a, st, pdl);
        case 8: return launch_decode<8>(a, st, pdl);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace alice
