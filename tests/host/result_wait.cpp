// result_wait against a stand-in for the stream synchronization.
#include <cstdio>
#include "../../nightstream_b200/csrc/internal.cuh"

static uint64_t g_words[6];
static int g_fill, g_syncs;       // words that the synchronization finds written
static cudaError_t g_status;

extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t) {
    g_syncs++;
    for (int i = 0; i < g_fill; i++) g_words[i] = 7 + i;
    return g_status;
}

static bool expect(const char* what, int before, int at_sync, cudaError_t status, cudaError_t want, int syncs) {
    neo_gpu_ctx ctx;
    result_arm(g_words, 6);
    for (int i = 0; i < before; i++) g_words[i] = 1 + i;
    g_fill = at_sync;
    g_syncs = 0;
    g_status = status;
    const cudaError_t got = result_wait(&ctx, g_words, 6);
    if (got == want && g_syncs == syncs) return true;
    printf("%s: got %d, want %d; %d synchronizations\n", what, (int)got, (int)want, g_syncs);
    return false;
}

int main() {
    bool ok = expect("there at once", 6, 6, cudaSuccess, cudaSuccess, 0);
    ok &= expect("late", 2, 6, cudaSuccess, cudaSuccess, 1);
    ok &= expect("one word never written", 0, 5, cudaSuccess, cudaErrorNotReady, 1);
    ok &= expect("a launch that failed", 0, 0, cudaErrorLaunchFailure, cudaErrorLaunchFailure, 1);
    if (ok) puts("ok");
    return ok ? 0 : 1;
}
