// Host interface of the whole-token kernel on integer tensor products (decode_token_mma.cu), which decode_token.cu hands the models it takes to.
#pragma once
#include "decode_token.h"

struct brasa_token_mma;

// For a model that brasa_token_program_supported accepts: whether this kernel runs it. *out stays null where its vectors leave no room.
bool brasa_token_mma_takes(const brasa_token_model &m);
int32_t brasa_token_mma_create(brasa_ctx *ctx, const brasa_token_model &m, brasa_token_mma **out);
void brasa_token_mma_free(brasa_token_mma *p);
int32_t brasa_token_mma_launch(brasa_cmd *cmd, brasa_token_mma *p);
