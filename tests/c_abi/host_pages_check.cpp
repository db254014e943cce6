// Prints, for a buffer in use, a fresh one and a large one of each, how often ready_pages asks CUDA about it,
// and whether its contents and its neighbours' are kept.
#include "host_pages.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

static int news_left = -1;   // allocations until one fails (-1: none does)
void *operator new(size_t n)
{
    if (news_left == 0) throw std::bad_alloc();
    if (news_left > 0) --news_left;
    if (void *p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

static int asked;
extern "C" cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
    ++asked;
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

int main()
{
    for (size_t bytes : {(size_t)1000, (size_t)(300 << 10), (size_t)(64 << 20)})
        for (int used = 0; used < 2; ++used) {
            char *p = (char *)mmap(nullptr, bytes + 8192, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
            if (p == MAP_FAILED) return 1;
            if (used) std::memset(p, 7, bytes + 8192);
            asked = 0;
            lbg::ready_pages({{p + 100, bytes}, {nullptr, 5}, {p, 0}});
            bool same = true;
            for (size_t k = 0; k < bytes + 8192; k += 997) same &= p[k] == (used ? 7 : 0);
            std::printf("%zu %d asked %d kept %d\n", bytes, used, asked, (int)same);
            munmap(p, bytes + 8192);
        }
    // no memory for the first, second or third helper thread
    for (int n = 0; n < 3; ++n) {
        const size_t bytes = 64 << 20;
        char *p = (char *)mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        news_left = n;
        lbg::ready_pages({{p, bytes}});
        news_left = -1;
        std::printf("helpers %d\n", n);
        std::fflush(stdout);
        munmap(p, bytes);
    }
    return 0;
}
