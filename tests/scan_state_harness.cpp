// The unit form's scan states (scan_state.cuh) under every order of a publishing warp's and the
// reading warp's memory accesses: the publisher's writes are recorded, and the reader is run once
// for every number of them that can have been made before each of its reads.
#include <cstddef>
#include <vector>

#include "../mars_b200/csrc/scan_state.cuh"

namespace {

struct Write {
    int at;
    float value;
};

struct Words {
    std::vector<float>* mem;
    std::vector<Write>* log;             // the publisher's
    const std::vector<size_t>* made;     // the reader's: writes made before its k-th read
    size_t* reads;
    float load(int i) const {
        const size_t k = (*reads)++;
        for (size_t j = 0; made && k < made->size() && j < (*made)[k]; ++j)
            (*mem)[(*log)[j].at] = (*log)[j].value;
        return (*mem)[i];
    }
    void store(int i, float v) const { log->push_back({i, v}); }
};

}  // namespace

// From a range's state `from` to `to` (negative: the full form), publisher and reader in every
// order.  Returns the orders tried, or -1 when one showed neither of the two states.
extern "C" int scan_orders(float from, float to) {
    using namespace mars::tc;
    constexpr int kRange = 5, kWords = 32;
    std::vector<float> start(kWords, kScanNothing);
    std::vector<Write> log;
    size_t reads = 0;
    scan_publish(Words{&start, &log, nullptr, &reads}, kRange, from < 0.0f, from);
    for (const Write& w : log) start[w.at] = w.value;
    log.clear();
    scan_publish(Words{&start, &log, nullptr, &reads}, kRange, to < 0.0f, to);
    // How many reads a reader makes.
    std::vector<float> mem = start;
    reads = 0;
    scan_read(Words{&mem, &log, nullptr, &reads}, kRange);
    std::vector<size_t> made(reads, 0);
    int orders = 0;
    for (;;) {
        mem = start;
        reads = 0;
        const ScanState s = scan_read(Words{&mem, &log, &made, &reads}, kRange);
        ++orders;
        auto shows = [&](float state) {
            return state < 0.0f ? s.full : !s.full && s.threshold == state;
        };
        if (!shows(from) && !shows(to)) return -1;
        // The next nondecreasing sequence of 0..log.size().
        size_t k = made.size();
        while (k > 0 && made[k - 1] == log.size()) --k;
        if (k == 0) return orders;
        const size_t v = made[k - 1] + 1;
        for (size_t j = k - 1; j < made.size(); ++j) made[j] = v;
    }
}
