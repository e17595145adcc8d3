// as_devbuf.h against a fake CUDA runtime: every pointer remembers the GPU it was made on.
#include "as_devbuf.h"

#include <cstdio>
#include <cstdlib>
#include <map>

static int current = 0, mallocs = 0, frees = 0;
static bool refuse = false;
static std::map<void*, int> owner;

#define CHECK(c) \
    if (!(c)) { std::fprintf(stderr, "line %d: %s\n", __LINE__, #c); std::exit(1); }

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    if (refuse) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    owner[*p] = current;
    mallocs++;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    CHECK(owner.count(p) && owner[p] == current);  // freed with its own GPU current
    owner.erase(p);
    std::free(p);
    frees++;
    return cudaSuccess;
}
}

int main() {
    {
        asb::DevBuf b;
        CHECK(!b.p && b.dev == -1 && !b.holds(0, 0));
        CHECK(b.alloc(100) == cudaSuccess && owner[b.p] == 0 && mallocs == 1);
        void* first = b.p;
        CHECK(b.holds(100, 0) && !b.holds(100, 1) && !b.holds(101, 0));
        CHECK(b.alloc(50) == cudaSuccess && b.p == first && b.bytes == 100);  // kept
        current = 1;  // the same size on another GPU: moved there
        CHECK(b.alloc(50) == cudaSuccess && owner[b.p] == 1 && b.dev == 1 && b.bytes == 50);
        CHECK(mallocs == 2 && frees == 1 && current == 1);
        CHECK(b.alloc(60) == cudaSuccess && owner[b.p] == 1 && mallocs == 3 && frees == 2);  // grown
        current = 0;
        refuse = true;
        CHECK(b.alloc(10) == cudaErrorMemoryAllocation && !b.p && b.bytes == 0 && b.dev == -1 && current == 0);
        refuse = false;
        CHECK(b.alloc(0) == cudaSuccess && b.p);  // an empty buffer is still a buffer
        current = 3;
    }
    CHECK(owner.empty() && current == 3);  // freed on its GPU, the caller's device left as it was
    std::puts("devbuf ok");
    return 0;
}
