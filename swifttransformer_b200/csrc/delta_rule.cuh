// What the kernels of the gated delta rule share (delta_rule.cu: the mathematics and the walk token by token; delta_chunks.cu:
// long portions in chunks side by side).
#pragma once
#include "common.cuh"

struct DeltaShape {
    int H, G, dim, vd;            // value heads, query/key heads, key size, value size
    int q_off, k_off, v_off, b_off, a_off, g_off;   // columns of the projection
    int rank_a, rank_g;           // 0: no low-rank pair, the projection holds the logits themselves (see below)
    int gate_silu;                // the output gate: 0 sigmoid(z), 1 z * sigmoid(z)
    // columns of a prepared row
    __host__ __device__ int pq() const { return 0; }
    __host__ __device__ int pk() const { return G * dim; }
    __host__ __device__ int pv() const { return 2 * G * dim; }
    __host__ __device__ int pd() const { return 2 * G * dim + H * vd; }
    __host__ __device__ int pb() const { return 2 * G * dim + H * vd + H * dim; }
    __host__ __device__ int row() const { return 2 * G * dim + H * vd + H * dim + H; }
    int stride;                   // floats from one prepared row to the next (at least row())
};

// Long portions in chunks (delta_chunks.cu): floats of scratch beyond the prepared rows and the outputs for n_seqs requests in
// chunks, 0: the sizes do not fit; and the launch for the requests of at least `from` tokens, between delta_prepare and
// delta_output.
long long delta_chunks_floats(int n_tokens, int n_seqs, const DeltaShape& sh);
int delta_chunks_launch(const float* prep, const DeltaShape& sh, float* scratch, float* state, int write_state, float* o,
                        const int* positions, const int* q_start, const int* slots, int n_tokens, int n_seqs, int from, cudaStream_t s);
