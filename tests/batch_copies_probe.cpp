// Test probe (TEST INFRASTRUCTURE ONLY): csrc/batch_copies.h over a fake of the CUDA runtime whose n-th creation fails.
// For every n: nothing may be left behind, and the next creation is as the first.  Prints the pieces as "layer:begin".
#include "../turbogpt_b200/csrc/batch_copies.h"
#include <cstdio>
#include <set>

static int creations = 0, failing = 0, wrong = 0, handles = 0;
static std::set<void *> alive;
template <class T> static cudaError_t create(T *p) {
    if (++creations == failing)
        return cudaErrorMemoryAllocation;
    *p = reinterpret_cast<T>(uintptr_t(0x1000 + ++handles));
    alive.insert(*p);
    return cudaSuccess;
}
static cudaError_t destroy(void *p) {
    wrong += alive.erase(p) != 1; // not alive, or destroyed twice
    return cudaSuccess;
}
extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return create(e); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return create(s); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return destroy(e); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return destroy(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    wrong += !alive.count(s);
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "refused"; }
}

int main() {
    constexpr int Depth = 9;
    Layout layout{};
    for (int l = 0; l < Depth; ++l)
        layout.layers[l].attention_norm = 32768 + 197120 * l;
    layout.count = 32768 + 197120 * Depth + 256;
    BatchCopies copies;
    copies.create(layout, Depth, true);
    const int whole = creations;
    for (const BatchCopies::Piece &piece : copies.pieces)
        printf("%d:%lld ", piece.layer, (long long)piece.begin);
    for (int n = 1; n <= whole; ++n) {
        BatchCopies again;
        const size_t before = alive.size();
        creations = 0, failing = n;
        bool thrown = false;
        try {
            again.create(layout, Depth, true);
        } catch (const std::exception &) {
            thrown = true;
        }
        wrong += !thrown || alive.size() != before || again.stream || again.forward_done || !again.pieces.empty();
        failing = 0;
        again.create(layout, Depth, true);
        wrong += again.pieces.size() != copies.pieces.size() || alive.size() != before + whole;
        again.destroy();
        wrong += alive.size() != before;
    }
    copies.create(layout, Depth, false); // replaces what was there
    wrong += !copies.pieces.empty() || alive.size() != 2;
    copies.destroy();
    copies.destroy();
    printf("wrong %d alive %zu\n", wrong, alive.size());
    return 0;
}
