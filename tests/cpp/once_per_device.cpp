// What is set once per device (a kernel's shared-memory limit): on every device
// that is used, again after a failure, and past 64 devices every time.  The
// device is this file's own cudaGetDevice: no GPU.
#include <cstdio>
#include "gb_once.h"

static int g_device = 0;
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int *dev) {
    *dev = g_device;
    return cudaSuccess;
}

int main() {
    static gb::OncePerDevice once;
    int runs = 0;
    auto f = [&] {
        runs++;
        return cudaSuccess;
    };
    auto fails = [&] {
        runs++;
        return cudaErrorUnknown;
    };
    const int devices[] = {0, 0, 1, 0, 1, 63, 63, 2}, want[] = {1, 1, 2, 2, 2, 3, 3, 4};
    for (int i = 0; i < 8; i++) {
        g_device = devices[i];
        if (once(f) != cudaSuccess || runs != want[i]) return printf("device %d: %d runs\n", devices[i], runs), 1;
    }
    g_device = 5;
    if (once(fails) == cudaSuccess || once(f) != cudaSuccess || once(fails) != cudaSuccess || runs != 6)
        return printf("after a failure: %d runs\n", runs), 1;
    g_device = 70;
    if (once(f) != cudaSuccess || once(f) != cudaSuccess || runs != 8) return printf("device 70: %d runs\n", runs), 1;
    return 0;
}
