// Which of the tables that depend on the active element types stand on the device.  Host bookkeeping without CUDA.
#pragma once

#include <vector>

namespace sxb {

// A table stands for `types` only once its flag has been set, after its upload: a preparation that throws half-way (an
// allocation that fails, a table too large to index) leaves the flags of what is missing down, and the next one with the
// same types makes it.
struct TypeTables {
    std::vector<int> types;      // active element types, ascending
    bool basis = false;          // layer 0 on the functions of the radial network's last hidden layer
    bool folded = false;         // layer 0 on the folded table of every ordered pair
    bool pairs = false;          // layer 1, density scaling and pair repulsion

    // Takes up other types; the tables of the ones before no longer stand.
    void request(const std::vector<int>& requested)
    {
        if (requested == types) return;
        basis = folded = pairs = false;
        types = requested;
    }
};

}  // namespace sxb
