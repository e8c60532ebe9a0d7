// Routing of a mixture-of-experts layer behind the router's product (see moe_route.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

struct FlMoeRouteArgs {
  const void* logits;        // [tokens, experts] bf16
  const float* bias;         // [experts]
  int tokens, experts, topk; // experts <= 64, topk <= 8 and <= experts
  float* probs;              // [tokens, experts]: softmax(logits + bias)
  float* w;                  // [tokens, topk]: the chosen probabilities over their sum, largest first
  int* idx;                  // [tokens, topk]; equal probabilities: the lower expert first
  long long* idx64;          // the same
  float* part;               // scratch [fl_moe_route_blocks(tokens)][2][experts]
  float* share;              // [experts]: share of the tokens whose first choice is the expert
  float* aux;                // [1]: experts * sum(share * mean probability)
  // backward
  const float* dw;           // [tokens, topk] or null
  const float* daux;         // [1] or null
  void* dlogits;             // [tokens, experts] bf16
};

#ifdef __cplusplus
extern "C" {
#endif
int fl_moe_route_blocks(int tokens);
int fl_moe_route(const FlMoeRouteArgs* a, cudaStream_t stream);
int fl_moe_route_bwd(const FlMoeRouteArgs* a, cudaStream_t stream);
#ifdef __cplusplus
}
#endif
