// What the C ABI does not show of a context: built against the library's
// internal headers, so it has the layout of the library it is loaded beside.
#include "sys_internal.cuh"

extern "C" unsigned long long ctx_pool_used(soil_ctx* ctx) {
    unsigned long long v = ~0ull;  // a cuuint64_t
    cudaMemPoolGetAttribute(ctx->pool, cudaMemPoolAttrUsedMemCurrent, &v);
    return v;
}

// The launches of `ctx` are shaped for a device of `sms` multiprocessors.
extern "C" void ctx_set_sms(soil_ctx* ctx, unsigned long long sms) { ctx->sms = sms; }
extern "C" unsigned long long ctx_get_sms(const soil_ctx* ctx) { return ctx->sms; }
