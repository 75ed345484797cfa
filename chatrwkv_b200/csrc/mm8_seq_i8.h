// mm8_seq on tcgen05 kind::i8 (mm8_seq_i8.cu): 1..4 matrices with the same rows of x count and in-features in one launch.
#pragma once
#include "seq_epi.cuh"

constexpr int kSeqI8MaxProblems = 4;
struct SeqI8Problem {
    const void* x; int64_t x_stride;
    const uint8_t* w; int64_t w_stride;
    const void* mx; const void* rx; const void* my; const void* ry;
    void* y; int64_t y_stride; int64_t M;
    SeqEpi epi;
    rwkv_mm8_seq_prologue pro;      // the same kind for all matrices of a launch
};
// Bytes for `rwkv_mm8_seq_i8` (0 where it does not apply); the first word of the workspace is its error word.
size_t rwkv_mm8_seq_i8_workspace_bytes(int nprob, int64_t T, int64_t N, const int64_t* M);
// fp16 operands; RWKV_ERR_UNSUPPORTED when a layout is not one TMA can fetch (the caller then takes another kernel).
int rwkv_mm8_seq_i8(int nprob, const SeqI8Problem* probs, int64_t T, int64_t N, void* workspace, size_t workspace_bytes, void* stream);
void rwkv_mm8_seq_i8_set_single_cta(bool single);       // never CTA pairs (same results)
