// Contexts of one device that take turns find their own entries again
// (context_table.h), as the memory pools are looked up; on the host.
#include <cstdio>

#include "context_table.h"

int main()
{
    sbb::ContextTable<int> pools;
    int made = 0, wrong = 0;
    // the lookup of device_pool: a pool that is not found is made
    auto pool_of = [&](int dev, unsigned long long ctx) {
        if (int *p = pools.find(dev, ctx)) return *p;
        pools.add(dev, ctx, ++made);
        return made;
    };
    for (int turn = 0; turn < 100; turn++)
        for (int dev = 0; dev < 2; dev++)
            for (unsigned long long ctx = 1; ctx <= 2; ctx++)
                wrong += pool_of(dev, ctx) != 2 * dev + (int)ctx;
    // a context that replaces another has a pool of its own
    wrong += pool_of(0, 3) != 5 || pool_of(0, 1) != 1 || pool_of(1, 2) != 4;
    if (made == 5 && !wrong) std::printf("ok\n");
    return made != 5 || wrong;
}
