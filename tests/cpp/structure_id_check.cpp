// Host-side check that no two block structures of a process share an id, also
// when one is made at the address of one that is gone; structures of a grid
// that are alive are one object.
#include <cstdio>
#include <set>

#include "structure.h"

using namespace hmb;

int main() {
    std::set<uint64_t> ids;
    std::set<const void*> at;
    const int side[] = {8, 16, 24, 32};   // 3 levels: one topology, four sizes
    int made = 0;
    for (int round = 0; round < 20; ++round)
        for (int n : side) {
            const int sizes[2] = {n, n};
            auto S = build_structure(2, sizes, 3, true);
            auto again = build_structure(2, sizes, 3, true);
            if (again != S || again->id != S->id) {
                std::printf("fail: two structures of one grid\n");
                return 1;
            }
            ids.insert(S->id);
            at.insert(S.get());
            ++made;
        }
    if ((int)ids.size() != made) {
        std::printf("fail: %d structures at %zu addresses, %zu ids\n", made, at.size(), ids.size());
        return 1;
    }
    std::printf("ok\n");
    return 0;
}
