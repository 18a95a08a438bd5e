// GridTable (bulbit_b200/csrc/grid_table.h): values come back, also from
// several threads; a full table stores nothing more and finds what it holds;
// nothing is allocated on the heap. Prints one line per failure and returns
// non-zero if any.
#include "grid_table.h"

#include <cstdio>
#include <cstdlib>
#include <new>
#include <thread>

static bool g_counting = false;
static int g_allocations = 0;

void* operator new(size_t n)
{
    g_allocations += g_counting ? 1 : 0;
    if (void* p = std::malloc(n))
    {
        return p;
    }
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

using namespace bbg;

static int failures = 0;
static void Check(bool ok, const char* what)
{
    if (!ok)
    {
        ++failures;
        std::printf("failed: %s\n", what);
    }
}

// Distinct keys whose numbers differ in one field at a time.
static GridKey Key(int i)
{
    static const char kernels[4096] = {};
    return GridKey{ kernels + 16 * (i / 8 % 256), size_t(i / 4 % 2) * 1024, i % 2 ? 128 : 256, i / 2 % 2 + i / 2048 * 2 };
}

int main()
{
    static GridTable table, full;
    g_counting = true;
    Check(table.Find(Key(0)) == 0, "an empty table finds nothing");
    for (int i = 0; i < 600; ++i)
    {
        table.Store(Key(i), i + 1);
    }
    bool same = true;
    for (int i = 0; i < 600; ++i)
    {
        same = same && table.Find(Key(i)) == i + 1;
    }
    Check(same, "600 stored grids are found");
    Check(table.Find(Key(601)) == 0, "a key that was not stored is not found");
    table.Store(Key(7), 99);
    Check(table.Find(Key(7)) == 99, "a second store replaces the first");
    for (int i = 0; i < GridTable::kCapacity + 100; ++i)
    {
        full.Store(Key(i), i + 1);
    }
    same = true;
    for (int i = 0; i < GridTable::kCapacity + 100; ++i)
    {
        same = same && full.Find(Key(i)) == (i < GridTable::kCapacity ? i + 1 : 0);
    }
    Check(same, "a full table keeps its first entries and stores no others");
    g_counting = false;
    Check(g_allocations == 0, "nothing is allocated");

    static GridTable shared;
    bool ok[4] = { true, true, true, true };
    std::thread threads[4];
    for (int t = 0; t < 4; ++t)
    {
        threads[t] = std::thread([t, &ok] {
            for (int r = 0; r < 50; ++r)
            {
                for (int i = 0; i < 200; ++i)
                {
                    const int g = shared.Find(Key(i));
                    ok[t] = ok[t] && (g == 0 || g == i + 1);
                    shared.Store(Key(i), i + 1);
                    ok[t] = ok[t] && shared.Find(Key(i)) == i + 1;
                }
            }
        });
    }
    for (auto& t : threads)
    {
        t.join();
    }
    Check(ok[0] && ok[1] && ok[2] && ok[3], "four threads");
    std::printf("%d failures\n", failures);
    return failures ? 1 : 0;
}
