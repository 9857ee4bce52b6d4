// What the products on CUDA cores, and the FP32 products on tensor cores, do with an output.
#pragma once
#include "device_utils.cuh"
#include "kernels.cuh"

// Every case is inlined for each output of a thread: a second GELU here made the code a fifth longer and small calls, which fetch it anew,
// 5 to 12 % slower (the reference architecture's gradients of 64 tokens 555 -> 631 us), so that Epilogue::Gelu is the tensor cores' alone.
template <class Out> struct EpilogueOps {
    // `value` is the FP32 accumulator; returns what is stored to C (already in storage rounding).
    __device__ static void apply(const GemmArgs &g, float value, int64_t c_index, int64_t r_index, int z) {
        Out *c = (Out *)g.c + z * g.c_batch;
        switch (g.epilogue) {
        case Epilogue::Store:
            c[c_index] = from_float<Out>(value);
            break;
        case Epilogue::Residual: {
            const Out *r = (const Out *)g.r + z * g.r_batch;
            c[c_index] = from_float<Out>(rounded<Out>(value) + to_float(r[r_index]));
            break;
        }
        case Epilogue::GeluDual: {
            float pre = rounded<Out>(value);
            c[c_index] = from_float<Out>(gelu_derivative(pre));
            ((Out *)g.c2 + z * g.c_batch)[c_index] = from_float<Out>(gelu(pre));
            break;
        }
        case Epilogue::GeluGrad: {
            const Out *r = (const Out *)g.r + z * g.r_batch;
            c[c_index] = from_float<Out>(rounded<Out>(value) * to_float(r[r_index]));
            break;
        }
        case Epilogue::Axpby: {
            const Out *r = (const Out *)g.r + z * g.r_batch;
            c[c_index] = from_float<Out>(g.alpha * value + g.beta * to_float(r[r_index]));
            break;
        }
        }
    }
};
