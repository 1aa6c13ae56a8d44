// What the native launches of dense models (dense_step.cu, dense_decode.cu) are told about a layer.
#pragma once

// One schedule entry; weights and sizes, fixed when the model is bound (engine/native.py has the same order).
struct FdDenseLayer {
    const void *norm1, *norm2, *w_qkv, *b_qkv, *w_o, *w_gate_up, *w_down;
    long long norm1_f32, norm2_f32, bias_f32;      // whether these vectors are float32
    long long hidden, inter, n_q, n_kv, d, window, chunk, write_kv;
    long long group, index, position;              // cache group, layer in it, rotation tables
    double eps1, eps2, scale;
};
