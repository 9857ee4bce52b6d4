// What tg_batch's results leave the GPU by while the backward pass runs: a stream of their own, and events that the kernel
// sequence records when the logits and when a piece of the gradients is complete.
#pragma once
#include "common.h"

struct BatchCopies {
    struct Piece { // of the gradient, from `begin` to the piece before it, or the end: complete after the backward pass of `layer`
        int layer;
        int64_t begin;
        cudaEvent_t ready = nullptr;
    };
    static constexpr int64_t LeastPiece = 1 << 19; // floats: two megabytes
    cudaStream_t stream = nullptr;
    cudaEvent_t forward_done = nullptr;
    std::vector<Piece> pieces;

    // All of it or nothing.  Without `in_pieces` the gradients have none and leave after the pass.
    void create(const Layout &layout, int depth, bool in_pieces) {
        BatchCopies made;
        try {
            auto event = [](cudaEvent_t &e) { CHECK_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)); };
            event(made.forward_done);
            int64_t end = layout.count;
            for (int l = depth - 1; l >= 0 && in_pieces; --l) {
                const int64_t begin = layout.layers[l].attention_norm;
                if (end - begin < LeastPiece)
                    continue;
                made.pieces.push_back({l, begin});
                event(made.pieces.back().ready);
                end = begin;
            }
            CHECK_CUDA(cudaStreamCreateWithFlags(&made.stream, cudaStreamNonBlocking));
        } catch (...) {
            made.destroy();
            throw;
        }
        destroy();
        *this = made;
    }
    void destroy() {
        if (stream) {
            cudaStreamSynchronize(stream);
            cudaStreamDestroy(stream);
        }
        if (forward_done)
            cudaEventDestroy(forward_done);
        for (const Piece &piece : pieces)
            if (piece.ready)
                cudaEventDestroy(piece.ready);
        *this = {};
    }
};
