// The memory a context may keep for its mesh gradients, and what it holds. Test helper: compiled by
// tests/test_gpu_param_routes.py.
#include "ctx.cuh"

extern "C" void limit_tape(afvm_ctx* ctx, size_t bytes) { reinterpret_cast<afvm::Ctx*>(ctx)->paramTapeMost = bytes; }
// 0: nothing, 1: one stage's tape, 2: a whole step's
extern "C" int tape_held(const afvm_ctx* ctx) {
    const afvm::Ctx* c = reinterpret_cast<const afvm::Ctx*>(ctx);
    return c->paramTape ? (c->paramTapeWhole ? 2 : 1) : 0;
}
