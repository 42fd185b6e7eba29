// Splits of a mesh with the k-th allocation (or every one from the k-th on)
// refused, for every k given: the call returns or throws in the calling thread;
// the process must not end in std::terminate, and a call that had its memory
// afterwards must give the split of the first one.
#include <atomic>
#include <cstdio>
#include <new>

// refused_new.cpp: allocations still granted; whether all later ones are refused
extern std::atomic<long long> g_left;
extern std::atomic<int> g_all;

#include "cf_partition.cu"

using namespace cf;

static HostLayout grid(int X, int Y, int Z)
{
    const int n = X * Y * Z;
    HostLayout L;
    L.nslices = (n + 31) / 32;
    L.maxw = 6;
    L.nnzp = 32LL * 6 * L.nslices;
    L.sliceOff.resize(L.nslices + 1);
    for (int s = 0; s <= L.nslices; ++s) L.sliceOff[s] = 32 * 6 * s;
    L.col.assign(L.nnzp, -1);
    for (int i = 0; i < n; ++i)
    {
        const int x = i % X, y = i / X % Y, z = i / (X * Y);
        int k = 0;
        auto add = [&](bool on, int j) {
            if (on) L.col[L.sliceOff[i / 32] + 32 * k++ + i % 32] = j;
        };
        add(x > 0, i - 1);
        add(x + 1 < X, i + 1);
        add(y > 0, i - X);
        add(y + 1 < Y, i + X);
        add(z > 0, i - X * Y);
        add(z + 1 < Z, i + X * Y);
    }
    return L;
}

int main()
{
    const HostLayout L = grid(30, 28, 26);   // large enough for several threads
    const int n = 30 * 28 * 26;
    ResHost whole;
    const long long before = 1LL << 60;
    g_left = before;
    if (!res_partition(n, L, false, 148, whole, 4)) return 2;
    const long long used = before - g_left;
    long long refused = 0;
    for (int all = 0; all < 2; ++all)
        for (long long k = 1; k <= used; k += k < 80 ? 1 : 1 + used / 60)
        {
            ResHost H;
            bool ok = false;
            g_all = all;
            g_left = k;
            try
            {
                ok = res_partition(n, L, false, 148, H, 4);
            }
            catch (const std::bad_alloc&)
            {
            }
            g_all = 0;
            g_left = before;
            refused += !ok;
            // (a thread that could not be started leaves its work to the others)
            if (ok && (H.idx != whole.idx || H.haloSlot != whole.haloSlot)) return 3;
        }
    ResHost again;
    if (!res_partition(n, L, false, 148, again, 4) || again.idx != whole.idx) return 4;
    std::printf("%lld allocations, refused %lld times\n", used, refused);
    return refused > 0 ? 0 : 5;
}
