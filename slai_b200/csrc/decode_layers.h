// The layers of a decode step as one launch (decode_layers.cuh), as the models describe them.
#pragma once
#include "common.cuh"

struct DecodeLayerPtrs {
    const uint8_t* w[7] = {};     // q, k, v, o, gate (or the only matrix of the feed-forward input), up, down
    const float* norm_w[2] = {};  // in front of q/k/v, of the feed-forward part
    const float* norm_b[2] = {};
    const float* bias[6] = {};    // q, k, v, o, feed-forward in, out (null: none)
};
struct DecodeLayers {
    int arch = 0;                 // 0: RmsNorm, gate / up with SiLU; 1: LayerNorm, one matrix with GELU
    int fmt = 0;                  // of every matrix
    bool kv_f16 = true;
    int n_layers = 0, dim = 0, q_dim = 0, kv_dim = 0, hidden = 0, head_size = 0, n_heads = 0, kv_mul = 1, seq_len = 0;
    float eps = 0.f;
    float *x = nullptr, *q = nullptr, *xb = nullptr, *hb = nullptr;
    const float* rope_cs = nullptr;  // (cos, sin) pairs of the position, adjacent pairs rotated (null: no rotation)
    const int* d_pos = nullptr;
    void *kcache = nullptr, *vcache = nullptr;  // [layer][head][position][head size]
    size_t layer_bytes = 0;
    bool whole_chip = false;      // not one cluster, see decode_layers_cluster_positions
};
bool decode_layers_supported(slai_ctx* ctx, const DecodeLayers& D);
int decode_layers_cluster_positions(const DecodeLayers& D);  // first position from which the whole chip is the quicker choice (INT_MAX: no choice)
size_t decode_layers_scratch_bytes(const DecodeLayers& D);
unsigned int* decode_layers_counter(void* scratch);  // the kernel's barrier counter: zero before every launch
constexpr int DECODE_LAYERS_NO_FIT = -1000;  // decode_layers_launch: the blocks cannot all run at once here; nothing was launched
int decode_layers_launch(slai_ctx* ctx, const DecodeLayers& D, const DecodeLayerPtrs* layers, void* scratch);
