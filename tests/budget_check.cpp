// KeptBytes (fcb_budget.hpp): the owners' shares never exceed the cap together and are
// given back.
#include <cstdio>
#include <thread>
#include <vector>

#include "../forestclaw_b200/csrc/fcb_budget.hpp"

int main() {
    int wrong = 0;
    std::atomic<size_t> total{0};
    {
        fcb::KeptBytes a(total, 70, 100), b(total, 100, 100);
        wrong += !a.add(60) || a.add(11) || b.add(50) || !b.add(40) || a.add(1) || total != 100;
        a.clear();
        wrong += total != 40 || !b.add(60) || b.add(1) || b.add((size_t)-1);
    }
    wrong += total != 0;
    std::atomic<int> over{0};
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; ++t)
        ts.emplace_back([&] {
            for (int k = 0; k < 20000; ++k) {
                fcb::KeptBytes mine(total, 600, 1000);
                for (int j = 0; j < 4; ++j) mine.add(170);
                over += total > 1000;
            }
        });
    for (auto& t : ts) t.join();
    wrong += over != 0 || total != 0;
    std::printf("%d wrong\n", wrong);
    return wrong != 0;
}
