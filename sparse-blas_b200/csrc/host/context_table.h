// context_table.h — what the library keeps for each device and context.
#pragma once

#include <vector>

namespace sbb {

// One value per device and context identity.  Contexts of one device can take
// turns (a program that pushes its own beside the primary one), so each keeps
// its entry; those of contexts that are gone stay, a few words each, and are never
// found again, because identities are not used twice.
template <typename T> class ContextTable {
public:
    T *find(int dev, unsigned long long ctx)
    {
        for (auto &e : entries_)
            if (e.dev == dev && e.ctx == ctx) return &e.value;
        return nullptr;
    }
    void add(int dev, unsigned long long ctx, const T &value) { entries_.push_back({dev, ctx, value}); }

private:
    struct Entry {
        int dev;
        unsigned long long ctx;
        T value;
    };
    std::vector<Entry> entries_;
};

}  // namespace sbb
