// TEST INFRASTRUCTURE ONLY: knobs and records of batch_class_kernels.cpp.
#pragma once
#include <atomic>
#include <cstdint>
#include <vector>

namespace fake {

extern std::atomic<int> fail_class;           // the launch of this class fails (-1: none)
extern std::atomic<int> class_us, tile_us;    // time of a class's work, and of each of its tiles
extern std::atomic<long> changed_under_work;  // classes whose tiles or descriptors changed while they worked

struct ClassLaunch {
    int id = 0;
    uint32_t begin = 0, all_tiles = 0;
    struct Tile {
        int exp, outk;
        uint64_t f0, nframes, frames;
        int plan;  // plan id of the descriptor's tw_pair table
    };
    std::vector<Tile> tiles;
};
std::vector<ClassLaunch> take_class_launches();
int plan_of(const void* table);  // plan id of a table, -1 if unknown

}  // namespace fake
