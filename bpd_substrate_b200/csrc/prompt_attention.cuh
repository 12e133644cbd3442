// Attention of a prompt's tokens to cached positions on the tensor cores, for latent attention on expanded keys and values and for grouped attention.
#pragma once
#include "decoder_device.cuh"

namespace bpdq {

// Matrices are bf16, positions 0 .. *pos + T - 1 in rows 0 ..; a row's unit of 8 elements starts on 16 bytes.
struct PromptAttention {
    int T, context;                     // tokens; rows of keys and values, *pos + T
    const int* pos;                     // device: position of the first token
    int groups, share;                  // query heads per key head: head g * share + j reads keys and values of group g
    int dim, dim1, value_dim;           // of a query and key, of its part that `keys` holds (the rest: `rest`, one for all groups), of a value
    const bf16 *q, *keys, *rest, *values;
    long ld_q, ld_keys, ld_rest, ld_values;         // elements between tokens; heads of q and groups of keys and values lie side by side
    int chunk;                          // a position sees itself and what came before, with `chunk` only from the start of its chunk on
    float scale;                        // of a score q . k
    float cap;                          // 0: none; else cap tanh(score / cap), and a score of 0 without a value takes part in the softmax
    bf16* o;                            // [T][groups * share * value_dim]
};

// Whether the kernel below takes it.
bool prompt_attention_fits(const PromptAttention& p);
int prompt_attention(const PromptAttention& p, cudaStream_t s);

}  // namespace bpdq
