// cf_partition.cu -- host-side split of one matrix graph into compact parts
// of equal size, one per CTA of the resident inner PCG (cf_resident.cu).
//
// Every row gets three integer coordinates: its breadth-first distance from
// three landmarks (a peripheral row, and two rows of least degree far from the landmarks taken
// before).  On a structured grid these are three independent linear forms of
// the cell's position; on any mesh they vary by at most one along a face, so
// cutting at a value of one of them separates rows that are far apart.  The
// rows are bisected recursively across the coordinate that spans the widest
// range, by counting (linear time per level).  On a 64^3 grid and 148 parts a
// part has about 560 halo rows for its 1,771 rows, against 880 for the same
// count of axis-aligned boxes and about 3,800 for equal ranges of the
// reverse Cuthill-McKee order.
#include "cf_host.hpp"
#include "cf_resident.cuh"

#include <algorithm>
#include <atomic>
#include <new>
#include <numeric>
#include <thread>
#include <vector>

namespace cf {

namespace {

struct Csr
{
    std::vector<int32_t> start, adj;
};

struct Item
{
    int32_t row;
    int32_t c[3];
};

// distances from `from` (a further component continues beyond the largest
// distance so far) and the visiting order; returns the largest distance
int bfs(int n, const Csr& g, int from, std::vector<int32_t>& queue, std::vector<int32_t>& dist)
{
    dist.assign((size_t)n, -1);
    queue.resize((size_t)n);
    int top = 0;
    int head = 0, tail = 0;
    int next = 0;
    queue[tail++] = from;
    dist[from] = 0;
    for (;;)
    {
        while (head < tail)
        {
            const int v = queue[head++];
            const int d = dist[v] + 1;
            for (int q = g.start[v]; q < g.start[v + 1]; ++q)
            {
                const int w = g.adj[q];
                if (dist[w] < 0)
                {
                    dist[w] = d;
                    queue[tail++] = w;
                }
            }
        }
        top = std::max(top, (int)dist[queue[tail - 1]]);
        if (tail == n) return top;
        while (dist[next] >= 0) ++next;
        dist[next] = ++top;
        queue[tail++] = next;
    }
}

// neighbours of every row, from the slices (entries of a row come first,
// its padding last)
void csr_of_layout(int n, const HostLayout& L, int threads, Csr& g)
{
    g.start.assign((size_t)n + 1, 0);
    auto width = [&](int r) { return (L.sliceOff[r / SLICE + 1] - L.sliceOff[r / SLICE]) / SLICE; };
    host_chunks(n, threads, [&](int b, int e) {
        for (int r = b; r < e; ++r)
        {
            const int32_t* c = L.col.data() + L.sliceOff[r / SLICE] + r % SLICE;
            int d = width(r);
            while (d > 0 && c[(size_t)SLICE * (d - 1)] == -1) --d;
            g.start[r + 1] = d;
        }
    });
    for (int r = 0; r < n; ++r) g.start[r + 1] += g.start[r];
    g.adj.resize((size_t)g.start[n]);
    host_chunks(n, threads, [&](int b, int e) {
        for (int r = b; r < e; ++r)
        {
            const int32_t* c = L.col.data() + L.sliceOff[r / SLICE] + r % SLICE;
            const int d = g.start[r + 1] - g.start[r];
            for (int k = 0; k < d; ++k)
                g.adj[g.start[r] + k] = c[(size_t)SLICE * k] & 0x7fffffff;
        }
    });
}

// rows of it[lo, hi) into parts p0 .. p0 + np - 1: part[row]
// (the two halves on two threads while `threads` > 1).  Out of memory on either
// of them throws here, once the other has ended.
void bisect(std::vector<Item>& it, int lo, int hi, int p0, int np, std::vector<int32_t>& part,
            std::vector<Item>& tmp, int threads)
{
    if (np == 1)
    {
        for (int i = lo; i < hi; ++i) part[it[i].row] = p0;
        return;
    }
    int mn[3], mx[3];
    for (int k = 0; k < 3; ++k)
    {
        mn[k] = mx[k] = it[lo].c[k];
        for (int i = lo + 1; i < hi; ++i)
        {
            mn[k] = std::min(mn[k], it[i].c[k]);
            mx[k] = std::max(mx[k], it[i].c[k]);
        }
    }
    int ax[3] = {0, 1, 2};
    std::sort(ax, ax + 3, [&](int a, int b) {
        const int sa = mx[a] - mn[a], sb = mx[b] - mn[b];
        return sa != sb ? sa > sb : a < b;
    });
    const int pl = np / 2;
    const int nl = (int)((long long)(hi - lo) * pl / np);
    // [a, b): the rows whose side is still open; each axis in turn narrows
    // it to the rows that tie with the cut value
    int a = lo, b = hi;
    const int cut = lo + nl;
    for (int q = 0; q < 3 && a < b; ++q)
    {
        const int k = ax[q];
        const int base = mn[k];
        std::vector<int32_t> hist;
        hist.assign((size_t)(mx[k] - base) + 2, 0);
        for (int i = a; i < b; ++i) ++hist[it[i].c[k] - base + 1];
        int v = 0;
        int below = a;
        while (below + hist[v + 1] <= cut)
        {
            below += hist[v + 1];
            if (below == cut) break;
            ++v;
        }
        const int val = below == cut ? base + v + 1 : base + v;
        // stable three-way split: c < val, c == val, c > val
        int i0 = a;
        const int neq = hist[val - base + 1];
        std::vector<Item>& t = tmp;
        int eq = 0, gt = neq;
        for (int i = a; i < b; ++i)
        {
            const int c = it[i].c[k];
            if (c < val)
                it[i0++] = it[i];
            else if (c == val)
                t[lo + eq++] = it[i];
            else
                t[lo + gt++] = it[i];
        }
        for (int i = 0; i < gt; ++i) it[i0 + i] = t[lo + i];
        if (below == cut) break;
        a = i0;
        b = i0 + neq;
    }
    struct Half
    {
        std::thread thread;
        bool failed = false;
        void join()
        {
            if (thread.joinable()) thread.join();
        }
        ~Half() { join(); }
    } left;
    bool started = false;
    if (threads > 1)
    {
        try
        {
            left.thread = std::thread([&, lo, cut, p0, pl, threads]() {
                try
                {
                    bisect(it, lo, cut, p0, pl, part, tmp, threads / 2);
                }
                catch (...)
                {
                    left.failed = true;
                }
            });
            started = true;
        }
        catch (...)
        {
        }
    }
    if (!started) bisect(it, lo, cut, p0, pl, part, tmp, 1);
    bisect(it, cut, hi, p0 + pl, np - pl, part, tmp, started ? threads - threads / 2 : 1);
    left.join();
    if (left.failed) throw std::bad_alloc();
}

}  // namespace

bool res_partition(int n, const HostLayout& L, bool ordered, int nparts, ResHost& R, int width)
{
    const int W = std::max(width, (int)L.maxw);
    if (W < 1 || W > 8 || nparts < 1 || nparts > n) return false;
    const int nt = host_threads(n);
    Csr g;
    csr_of_layout(n, L, nt, g);
    std::vector<int32_t> part((size_t)n, 0);
    if (nparts > 1)
    {
        // the first landmark: where Cuthill-McKee started (the last internal
        // row) or, unordered, the row farthest from the last one
        std::vector<int32_t> queue, dist[3];
        int from = n - 1;
        if (!ordered)
        {
            bfs(n, g, from, queue, dist[0]);
            from = queue[n - 1];
        }
        const int top = bfs(n, g, from, queue, dist[0]);
        int minDeg = 1 << 30;
        for (int i = 0; i < n; ++i) minDeg = std::min(minDeg, g.start[i + 1] - g.start[i]);
        auto pick = [&](int coords) {
            int best = 0, score = -1;
            for (int i = 0; i < n; ++i)
            {
                if (g.start[i + 1] - g.start[i] != minDeg) continue;
                int s = std::min(dist[0][i], top - dist[0][i]);
                if (coords > 1) s = std::min(s, dist[1][i]);
                if (s > score)
                {
                    score = s;
                    best = i;
                }
            }
            return best;
        };
        bfs(n, g, pick(1), queue, dist[1]);
        bfs(n, g, pick(2), queue, dist[2]);
        std::vector<Item> it((size_t)n), tmp((size_t)n);
        host_chunks(n, nt, [&](int b, int e) {
            for (int i = b; i < e; ++i) it[i] = Item{i, {dist[0][i], dist[1][i], dist[2][i]}};
        });
        bisect(it, 0, n, 0, nparts, part, tmp, nt);
    }
    // rows of every part: those with a neighbour elsewhere first, each group
    // in the internal order
    std::vector<int32_t> loc((size_t)n);
    std::vector<char> bnd((size_t)n, 0);
    R.W = W;
    R.parts.assign(nparts, ResPart());
    host_chunks(n, nt, [&](int b, int e) {
        for (int r = b; r < e; ++r)
            for (int q = g.start[r]; q < g.start[r + 1]; ++q)
                if (part[g.adj[q]] != part[r])
                {
                    bnd[r] = 1;
                    break;
                }
    });
    // rows of every part in each of `nt` ranges of rows: inner, boundary; then,
    // summed up, the local index of the next one there
    std::vector<std::vector<int32_t>> next(nt);
    for (auto& v : next) v.assign(2 * (size_t)nparts, 0);
    auto first = [&](int t) { return (int)((long long)n * t / nt); };
    host_chunks(nt, nt, [&](int b, int e) {
        for (int t = b; t < e; ++t)
            for (int r = first(t); r < first(t + 1); ++r) ++next[t][2 * part[r] + bnd[r]];
    });
    for (int p = 0; p < nparts; ++p)
    {
        ResPart& P = R.parts[p];
        for (int t = 0; t < nt; ++t) P.nb += next[t][2 * p + 1];
        int at[2] = {P.nb, 0};
        for (int t = 0; t < nt; ++t)
            for (int k = 0; k < 2; ++k)
            {
                const int c = next[t][2 * p + k];
                next[t][2 * p + k] = at[k];
                at[k] += c;
            }
        P.nloc = at[0];
    }
    R.maxLocP = 0;
    R.rowsP = 0;
    R.slots = 0;
    for (ResPart& p : R.parts)
    {
        p.nlocP = (p.nloc + SLICE - 1) / SLICE * SLICE;
        p.rowBase = R.rowsP;
        p.llBase = R.slots;
        R.rowsP += p.nlocP;
        R.slots += p.nb;
        R.maxLocP = std::max(R.maxLocP, p.nlocP);
    }
    R.rowMap.assign((size_t)R.rowsP, -1);
    host_chunks(nt, nt, [&](int b, int e) {
        for (int t = b; t < e; ++t)
            for (int r = first(t); r < first(t + 1); ++r)
            {
                const int p = part[r];
                loc[r] = next[t][2 * p + bnd[r]]++;
                R.rowMap[(size_t)R.parts[p].rowBase + loc[r]] = r;
            }
    });
    R.idx.resize((size_t)R.rowsP * W);
    R.emap.assign((size_t)R.rowsP * W, -1);
    std::vector<std::vector<int32_t>> halo(nparts);
    std::atomic<int> nextPart{0};
    std::atomic<bool> fits{true};
    auto work = [&]() {
        try
        {
            std::vector<int32_t> h;
            std::vector<int32_t> pos((size_t)R.slots, -1);   // halo value of a slot
            for (;;)
            {
                const int p = nextPart.fetch_add(1);
                if (p >= nparts) return;
                ResPart& P = R.parts[p];
                h.clear();
                int lo = R.slots, hi = -1;
                for (int l = 0; l < P.nb; ++l)
                {
                    const int r = R.rowMap[(size_t)P.rowBase + l];
                    for (int q = g.start[r]; q < g.start[r + 1]; ++q)
                    {
                        const int c = g.adj[q];
                        if (part[c] == p) continue;
                        const int s = R.parts[part[c]].llBase + loc[c];
                        if (pos[s] >= 0) continue;
                        pos[s] = 0;
                        h.push_back(s);
                        lo = std::min(lo, s);
                        hi = std::max(hi, s);
                    }
                }
                P.nh = (int)h.size();
                // in ascending order: sorted, or (many of few) picked up in it
                if (P.nh > (hi - lo) / 16)
                {
                    int k = 0;
                    for (int s = lo; s <= hi; ++s)
                        if (pos[s] >= 0) h[k++] = s;
                }
                else
                {
                    std::sort(h.begin(), h.end());
                }
                for (int k = 0; k < P.nh; ++k) pos[h[k]] = k;
                if (P.nlocP + P.nh + 1 > 65535)
                {
                    fits = false;
                    return;
                }
                const uint16_t zero = (uint16_t)(P.nlocP + P.nh);
                for (int l = 0; l < P.nlocP; ++l)
                {
                    const long long sb = ((long long)P.rowBase + l / SLICE * SLICE) * W;
                    const int lane = l % SLICE;
                    const int r = R.rowMap[(size_t)P.rowBase + l];
                    int k = 0;
                    if (r >= 0)
                    {
                        const int s = r / SLICE;
                        const int b0 = L.sliceOff[s];
                        const int w = (L.sliceOff[s + 1] - b0) / SLICE;
                        for (int j = 0; j < w; ++j)
                        {
                            const int32_t e = b0 + SLICE * j + (r % SLICE);
                            const int32_t cc = L.col[e];
                            if (cc == -1) continue;
                            const int c = cc & 0x7fffffff;
                            const size_t at = (size_t)pair_index(sb, W, k, lane);
                            if (part[c] == p)
                                R.idx[at] = (uint16_t)loc[c];
                            else
                                R.idx[at] = (uint16_t)(P.nlocP +
                                                       pos[R.parts[part[c]].llBase + loc[c]]);
                            R.emap[at] = e;
                            ++k;
                        }
                    }
                    for (; k < W; ++k) R.idx[(size_t)pair_index(sb, W, k, lane)] = zero;
                }
                for (int s : h) pos[s] = -1;
                halo[p] = h;
            }
        }
        catch (...)
        {
            fits = false;   // out of memory: no split
        }
    };
    // (the longest part: several threads also where the others take one)
    const int workers = n < 4096 ? nt : std::max(nt, 4);
    std::vector<std::thread> pool;
    for (int t = 1; t < workers; ++t)
    {
        try
        {
            pool.emplace_back(work);
        }
        catch (...)
        {
            break;   // fewer threads: the parts are taken from one counter
        }
    }
    work();
    for (auto& t : pool) t.join();
    if (!fits) return false;
    R.haloSlot.clear();
    R.maxHalo = 0;
    for (int p = 0; p < nparts; ++p)
    {
        R.parts[p].haloBase = (int)R.haloSlot.size();
        R.haloSlot.insert(R.haloSlot.end(), halo[p].begin(), halo[p].end());
        R.maxHalo = std::max(R.maxHalo, R.parts[p].nh);
    }
    return true;
}

// Consecutive ranges of rowsPerPart rows (whole slices), rows in the internal
// order; the exchange slot of a row is the row itself.
bool res_blocks(int n, const HostLayout& L, int rowsPerPart, ResHost& R, int width, int maxHalo)
{
    const int W = std::max(width, (int)L.maxw);
    if (W < 1 || W > 8 || rowsPerPart < SLICE || rowsPerPart % SLICE || n < 1) return false;
    const int nparts = (n + rowsPerPart - 1) / rowsPerPart;
    R.W = W;
    R.rowsP = R.slots = nparts * rowsPerPart;
    R.maxLocP = R.maxHalo = 0;
    R.parts.assign(nparts, ResPart());
    R.rowMap.assign((size_t)R.rowsP, -1);
    for (int r = 0; r < n; ++r) R.rowMap[r] = r;
    R.idx.resize((size_t)R.rowsP * W);
    R.emap.assign((size_t)R.rowsP * W, -1);
    R.haloSlot.clear();
    // local index of every column of the part at hand; the halo columns are
    // marked and then numbered in ascending order, so cells numbered at
    // random cost little more than others (12K cells: 1.2 ms, 8.9 with the halo
    // sorted and searched; 0.4 and 1.2 in natural order)
    constexpr int32_t NONE = -1, HALO = -2;
    std::vector<int32_t> local((size_t)n, NONE);
    for (int p = 0; p < nparts; ++p)
    {
        ResPart& P = R.parts[p];
        const int r0 = p * rowsPerPart;
        P.rowBase = P.llBase = r0;
        P.nloc = P.nb = std::min(rowsPerPart, n - r0);
        P.nlocP = (P.nloc + SLICE - 1) / SLICE * SLICE;
        auto each = [&](int r, auto fn) {
            const int s = r / SLICE;
            const int b0 = L.sliceOff[s];
            const int w = (L.sliceOff[s + 1] - b0) / SLICE;
            for (int j = 0; j < w; ++j)
            {
                const int32_t e = b0 + SLICE * j + r % SLICE;
                if (L.col[e] != -1) fn(e, L.col[e] & 0x7fffffff);
            }
        };
        for (int l = 0; l < P.nloc; ++l) local[r0 + l] = l;
        int lo = n, hi = -1;
        for (int r = r0; r < r0 + P.nloc; ++r)
            each(r, [&](int, int c) {
                if (local[c] != NONE) return;
                local[c] = HALO;
                lo = std::min(lo, c);
                hi = std::max(hi, c);
            });
        P.haloBase = (int)R.haloSlot.size();
        for (int c = lo; c <= hi; ++c)
            if (local[c] == HALO)
            {
                local[c] = P.nlocP + P.nh++;
                R.haloSlot.push_back(c);
            }
        R.maxLocP = std::max(R.maxLocP, P.nlocP);
        R.maxHalo = std::max(R.maxHalo, P.nh);
        if (P.nh > maxHalo || P.nlocP + P.nh + 1 > 65535) return false;
        for (int l = 0; l < P.nlocP; ++l)
        {
            const long long sb = ((long long)P.rowBase + l / SLICE * SLICE) * W;
            int k = 0;
            if (l < P.nloc)
                each(r0 + l, [&](int e, int c) {
                    const size_t at = (size_t)pair_index(sb, W, k, l % SLICE);
                    R.idx[at] = (uint16_t)local[c];
                    R.emap[at] = e;
                    ++k;
                });
            for (; k < W; ++k)
                R.idx[(size_t)pair_index(sb, W, k, l % SLICE)] = (uint16_t)(P.nlocP + P.nh);
        }
        for (int l = 0; l < P.nloc; ++l) local[r0 + l] = NONE;
        for (int h = P.haloBase; h < (int)R.haloSlot.size(); ++h) local[R.haloSlot[h]] = NONE;
    }
    return true;
}

}  // namespace cf
