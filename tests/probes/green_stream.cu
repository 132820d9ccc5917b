// A stream of a green context with at least `sms` of device 0's SMs (the
// current context is left as it was); 0 on success.
#include <cuda.h>

static CUgreenCtx g_ctx = nullptr;
static CUstream g_stream = nullptr;

extern "C" int green_stream_create(unsigned sms, void** stream, unsigned* got) {
  CUdevResource all, part, rest;
  CUdevResourceDesc desc;
  unsigned groups = 1;
  int e = cuDeviceGetDevResource(0, &all, CU_DEV_RESOURCE_TYPE_SM);
  if (!e) e = cuDevSmResourceSplitByCount(&part, &groups, &all, &rest, 0, sms);
  if (!e) e = cuDevResourceGenerateDesc(&desc, &part, 1);
  if (!e) e = cuGreenCtxCreate(&g_ctx, desc, 0, CU_GREEN_CTX_DEFAULT_STREAM);
  if (!e) e = cuGreenCtxStreamCreate(&g_stream, g_ctx, CU_STREAM_NON_BLOCKING, 0);
  *stream = g_stream;
  *got = part.sm.smCount;
  return e;
}

extern "C" int green_stream_destroy() {
  int e = cuStreamDestroy(g_stream);
  return e ? e : (int)cuGreenCtxDestroy(g_ctx);
}
