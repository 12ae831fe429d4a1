// Host check of the allocation-free entry point's wait records: over random sequences of direct calls, captures and replays, of
// one and of two launches, with waits that run out now and then, every call starts on a clear record and the reader sees
// what the last executed call left.  The device side (who clears what, when) is modelled here.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../catccos_b200/csrc/wait_records.hpp"

using namespace catccos;

static unsigned records[kWaitRecords];

struct Call {
    bool two, captured;
    unsigned record;
};

// What the GPU does for a call whose waits run out with `code` (0: they do not).  Returns false if it starts on a set record.
static bool execute(const Call& c, unsigned code)
{
    if (c.captured && !c.two) {
        records[c.record] = 0;  // the memset in front
    }
    for (unsigned r = 0; r < kWaitRecords; ++r) {
        if (c.two || r != c.record) {
            records[r] = 0;
        }
    }
    if (records[c.record] != 0) {
        return false;
    }
    records[c.record] = code;
    return true;
}

int main()
{
    std::srand(1);
    WaitRecordTurn turn;
    std::vector<Call> graphs;
    for (int i = 0; i < 1000000; ++i) {
        const int what = std::rand() % 4;
        Call c{std::rand() % 2 == 0, what == 0, 0};
        if (what <= 2) {
            c.record = c.two ? turn.two_launches(c.captured) : turn.one_launch(c.captured);
        }
        if (what == 0) {
            graphs.push_back(c);  // captured: nothing runs yet
            continue;
        }
        if (what == 3) {
            if (graphs.empty()) {
                continue;
            }
            c = graphs[std::rand() % graphs.size()];
        }
        const unsigned code = std::rand() % 3 == 0 ? 1u + std::rand() % 3 : 0u;
        if (!execute(c, code)) {
            std::printf("call %d starts on a set record\n", i);
            return 1;
        }
        unsigned seen = 0;
        for (unsigned r : records) {
            seen = seen != 0 ? seen : r;
        }
        if (seen != code) {
            std::printf("call %d left %u, the reader sees %u\n", i, code, seen);
            return 1;
        }
    }
    std::puts("wait records ok");
    return 0;
}
