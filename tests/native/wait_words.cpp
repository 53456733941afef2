// Test-only host build: the address of a context's wait words, so that a test can leave there what a kernel that gave up leaves.
#include "../../juno_b200/csrc/common.cuh"

extern "C" unsigned *wait_words(void *ctx) { return static_cast<juno_ctx *>(ctx)->gemv_scratch.qerr_host; }
