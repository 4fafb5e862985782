// besideEarlier and readsOwnRows (codegen.hpp) against their definitions: slot
// sets of every kernel, compared pairwise, on random plans whose rows overlap,
// repeat and point anywhere, and on plans in memory order.
#include <cstdio>
#include <random>
#include <set>

#include "codegen.hpp"

using namespace symgb::engine;

int main() {
    std::mt19937 rng(5);
    auto pick = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
    int wrong = 0, besides = 0, alone = 0, inPlace = 0;
    for (int trial = 0; trial < 20000; ++trial) {
        const bool ordered = trial % 2;  // outputs laid out in plan order, as the front end does
        const int slots = pick(8, 60), kernels = pick(1, 7);
        std::vector<symgb_kernel_desc> descs(kernels);
        std::vector<std::vector<std::int32_t>> access(kernels);
        std::vector<std::uint32_t> index;
        std::vector<std::set<long long>> reads(kernels), writes(kernels);
        std::vector<std::uint64_t> lo(kernels, ~0ull), hi(kernels, 0);
        int next = pick(1, 4);
        for (int k = 0; k < kernels; ++k) {
            symgb_kernel_desc& d = descs[k];
            d = symgb_kernel_desc{};
            d.level = pick(0, 2);
            d.num_instances = (std::uint64_t)pick(0, 4);
            d.num_output_rows = (std::uint32_t)pick(0, 2);
            d.num_index_rows = (std::uint32_t)pick(0, 2);
            const int size = (int)(d.num_instances * d.num_output_rows);
            const int at = ordered ? next : pick(0, slots);
            d.output_offset = (std::uint64_t)at;
            for (int q = 0; q < size; ++q) writes[k].insert(at + q);
            d.index_offset = index.size();
            const int most = ordered ? std::max(1, pick(0, 2) ? next - 1 : 3) : slots;
            for (std::uint64_t q = 0; q < d.num_instances * d.num_index_rows; ++q) index.push_back((std::uint32_t)pick(0, most));
            next += size;
            for (std::uint32_t r = 0; r < d.num_index_rows; ++r)
                for (int c = pick(1, 2); c > 0; --c) {
                    access[k].push_back((std::int32_t)r);
                    access[k].push_back(c - 1);
                }
            d.num_access = (std::uint32_t)(access[k].size() / 2);
            d.access = access[k].data();
            for (std::uint32_t a = 0; a < d.num_access; ++a)
                for (std::uint64_t i = 0; i < d.num_instances; ++i) {
                    const long long s = (long long)index[d.index_offset + access[k][2 * a] * d.num_instances + i] + access[k][2 * a + 1];
                    reads[k].insert(s);
                    lo[k] = std::min(lo[k], (std::uint64_t)s);
                    hi[k] = std::max(hi[k], (std::uint64_t)s);
                }
        }
        const SlotUse use{descs, index.data(), lo, hi};
        const std::vector<char> got = besideEarlier(use), own = readsOwnRows(use);
        auto meet = [](const std::set<long long>& a, const std::set<long long>& b) {
            for (long long s : a)
                if (b.count(s)) return true;
            return false;
        };
        for (int k = 0; k < kernels; ++k) {
            const bool expected = meet(reads[k], writes[k]);
            inPlace += expected;
            if ((bool)own[k] != expected && ++wrong < 5) std::printf("trial %d kernel %d reads its own rows: %d\n", trial, k, (int)own[k]);
        }
        std::vector<int> group;
        for (int k = 0; k < kernels; ++k) {
            if (!descs[k].num_instances) continue;
            bool free = !group.empty();
            for (int g : group)
                free = free && !meet(reads[k], writes[g]) && !meet(writes[k], writes[g]) && !meet(reads[g], writes[k]);
            if (!free) group.clear();
            group.push_back(k);
            (free ? besides : alone) += 1;
            if ((bool)got[k] != free) {
                if (++wrong < 5) std::printf("trial %d kernel %d: %d, expected %d\n", trial, k, (int)got[k], (int)free);
            }
        }
    }
    std::printf("%d beside, %d not, %d in place, %d wrong\n", besides, alone, inPlace, wrong);
    return wrong || !besides || !alone || !inPlace;
}
