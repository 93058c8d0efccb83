// C entry points of the trainer's memory-bound kernels (libcoccl.so).
// All tensors are bf16 unless stated; statistics and gradients of parameters
// are fp32. `scratch` arguments are caller-provided device buffers whose
// required size is given next to each function. Return 0 or a cudaError_t;
// -1 = unsupported shape.
#pragma once
#include <cuda_runtime.h>
#ifdef __cplusplus
extern "C" {
#endif

// y = LayerNorm(x (+ res)); xOut (optional) = x + res. H % 8 == 0, H <= 16384.
int cocclkLayerNormFwd(const void* x, const void* res, const void* gamma, const void* beta, void* y, void* xOut,
                       float* mean, float* rstd, int M, int H, float eps, cudaStream_t s);
// Number of partial rows the backward uses; scratch = grid * 2 * H floats.
int cocclkLayerNormBwdGrid(int M);
// dx = dLN/dx (+ dres); dgamma/dbeta (fp32) are overwritten or accumulated into.
int cocclkLayerNormBwd(const void* dy, const void* x, const float* mean, const float* rstd, const void* gamma,
                       const void* dres, void* dx, float* dgamma, float* dbeta, int accumulate, float* scratch,
                       int M, int H, cudaStream_t s);
// The same two for RMSNorm (no mean, no beta); scratch = cocclkLayerNormBwdGrid(M) * H floats.
int cocclkRmsNormFwd(const void* x, const void* res, const void* gamma, void* y, void* xOut, float* rstd, int M, int H,
                     float eps, cudaStream_t s);
int cocclkRmsNormBwd(const void* dy, const void* x, const float* rstd, const void* gamma, const void* dres, void* dx,
                     float* dgamma, int accumulate, float* scratch, int M, int H, cudaStream_t s);
// llama_kernels.cu. qkv [tokens][(nh + 2 nkv) D] (q heads, k heads, v heads) -> q [tokens][nh][D], k and v [tokens][nkv][D]:
// queries and keys rotated by the position (token % seq), with qw / kw (both or neither) RMS-normalised per head before.
// cosT / sinT: fp32 [seq][D] whose second halves repeat the first. D = 32, 64, 128 or 256.
int cocclkRotateFwd(const void* qkv, void* q, void* k, void* v, const float* cosT, const float* sinT, const void* qw,
                    const void* kw, int tokens, int seq, int nh, int nkv, int D, float eps, cudaStream_t s);
// Backward; dqw / dkw (fp32 [D]) are overwritten or accumulated into. scratch = cocclkRotateBwdGrid(tokens) * 2 D floats,
// needed (like qkv) only with qw.
int cocclkRotateBwdGrid(int tokens);
int cocclkRotateBwd(const void* dq, const void* dk, const void* dv, const void* qkv, void* dqkv, const float* cosT,
                    const float* sinT, const void* qw, const void* kw, float* dqw, float* dkw, int accumulate, float* scratch,
                    int tokens, int seq, int nh, int nkv, int D, float eps, cudaStream_t s);
// embed_kernels.cu. Bwd: grad (fp32 [vocab][H]) row of every id += sum of its tokens' rows of dy (bf16 [T][H]), in a fixed order
// (the tokens are sorted by id with T^2 comparisons, meant for up to 16384 of them). scratch: cocclkEmbedScratchBytes(T, H),
// 16-byte aligned. PositionsBwd: grad (fp32 [seq][H]) += sum over the batch of dy [batch][seq][H]. H % 8 == 0.
long cocclkEmbedScratchBytes(int T, int H);
int cocclkEmbedBwd(const void* dy, const long* ids, void* scratch, float* grad, int T, int H, long vocab, cudaStream_t s);
int cocclkEmbedPositionsBwd(const void* dy, float* grad, int batch, int seq, int H, cudaStream_t s);
// z [M][2 F] = gate | up: y = silu(gate) * up, and its gradient. F % 8 == 0.
int cocclkSwigluFwd(const void* z, void* y, int M, int F, cudaStream_t s);
int cocclkSwigluBwd(const void* dy, const void* z, void* dz, int M, int F, cudaStream_t s);
// out[n] (+)= sum_m x[m][n]; scratch = cocclkColSumBlocks(M) * N floats.
int cocclkColSumBlocks(int M);
int cocclkColSum(const void* x, float* out, int accumulate, float* scratch, int M, int N, cudaStream_t s);
// y = gelu_tanh(z (+ bias[n % N])); zOut (optional) = z + bias.
int cocclkGeluFwd(const void* z, const void* bias, void* y, void* zOut, long n, int N, cudaStream_t s);
int cocclkGeluBwd(const void* dy, const void* z, void* dz, long n, cudaStream_t s);
// loss[m] = CE(logits[m], targets[m]); logits are overwritten by their gradient times gscale.
int cocclkCrossEntropy(void* logits, const long* targets, float* loss, int M, int V, long ld, float gscale,
                       cudaStream_t s);
// Vocabulary-parallel cross-entropy (the vocabulary is sharded over tensor-parallel ranks; this rank holds columns
// [vocabOffset, vocabOffset + V)). Stats writes 4 floats per row {local max, sum exp(logit - max), target logit or 0,
// target-in-shard flag}; the caller all-gathers them over the group into statsAll [tp][M][4]; Finish writes
// loss[m] (the same value on every rank) and overwrites the logits with (softmax - onehot) * gscale.
int cocclkCrossEntropyStats(const void* logits, const long* targets, float* stats, int M, int V, long ld, long vocabOffset,
                            cudaStream_t s);
int cocclkCrossEntropyFinish(void* logits, const long* targets, const float* statsAll, int tp, float* loss, int M, int V,
                             long ld, long vocabOffset, float gscale, cudaStream_t s);
// AdamW over a flat shard. grad is fp32 or bf16; param (optional) receives the bf16 copy.
int cocclkAdam(float* master, float* m, float* v, const void* grad, int gradIsBf16, void* param, long n, float lr,
               float b1, float b2, float eps, float wd, int step, const float* gradScale, cudaStream_t s);
// out[0] (+)= sum x^2; scratch = cocclkSumSqBlocks(n) floats.
int cocclkSumSqBlocks(long n);
int cocclkSumSq(const void* x, int isBf16, long n, float* out, int accumulate, float* scratch, cudaStream_t s);
int cocclkClipCoef(const float* sumsq, float maxNorm, float gradScaleIn, float* coef, float* normOut, cudaStream_t s);
// dst(fp32) (+)= src(bf16)
int cocclkAccumBf16(float* dst, const void* src, long n, int accumulate, cudaStream_t s);

#ifdef __cplusplus
}
#endif
