// operator new that refuses the g_left-th allocation from now on, or (g_all) every
// one from there on.
#include <atomic>
#include <cstdlib>
#include <new>

std::atomic<long long> g_left{1LL << 60};
std::atomic<int> g_all{0};

void* operator new(std::size_t n)
{
    const long long k = g_left.fetch_sub(1);
    if (k == 1 || (k < 1 && g_all)) throw std::bad_alloc();
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}

void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
