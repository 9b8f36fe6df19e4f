// Runs the team traversal's stack step (csrc/team_stack.cuh) on the host with
// its lanes as threads, one at a time: between two barriers the lanes run one
// after another in a given order, the first lane first or last, as warps of
// independently scheduled threads may. Random hierarchies of child masks; every
// lane must visit the nodes that a single walk with its own stack visits.
//
//   team_stack_check -> "ok <nodes visited>", or the first difference.
#include "team_stack.cuh"

#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>

namespace {

constexpr int kDepth = 4;  // shared entries: deeper stacks go on in the lanes' own

struct Entry {
    uint32_t x, y;
};

uint32_t hash(uint32_t a, uint32_t b)
{
    uint64_t x = ((uint64_t)a << 32 | b) * 0x9E3779B97F4A7C15ull;
    x ^= x >> 29;
    x *= 0xBF58476D1CE4E5B9ull;
    return (uint32_t)(x >> 32);
}

// The internal hits and children of a node: `left` bounds the walk's length.
void visit(uint32_t seed, uint32_t node, uint32_t &hits, uint32_t &base, uint32_t &imask, uint32_t oct)
{
    const uint32_t h = hash(seed, node);
    imask = 0xffu;
    uint32_t slots = h & (h >> 8) & 0xffu;  // a quarter of the children on average
    if (node > 40000) slots = 0;
    hits = 0;
    for (uint32_t k = 0; k < 8; ++k)
        if (slots >> (k ^ oct) & 1u) hits |= 1u << k;
    base = 8 * node + 1;
}

// Lets one lane run at a time; at a barrier a lane waits until all have come.
struct Turns {
    std::mutex m;
    std::condition_variable cv;
    std::vector<int> order;
    size_t at = 0;
    uint64_t round = 0;
    explicit Turns(std::vector<int> o) : order(std::move(o)) {}
    void begin(int lane)
    {
        std::unique_lock<std::mutex> l(m);
        cv.wait(l, [&] { return order[at] == lane; });
    }
    void barrier(int lane)
    {
        std::unique_lock<std::mutex> l(m);
        const uint64_t r = round;
        if (++at == order.size()) at = 0, ++round;
        cv.notify_all();
        cv.wait(l, [&] { return round > r && order[at] == lane; });
    }
    void end()
    {
        std::unique_lock<std::mutex> l(m);
        if (++at == order.size()) at = 0, ++round;
        cv.notify_all();
    }
};

std::vector<uint32_t> walk_alone(uint32_t seed, uint32_t oct, uint32_t limit, size_t steps)
{
    std::vector<uint32_t> nodes;
    std::vector<Entry> stack;
    uint32_t node = 0;
    while (nodes.size() < steps) {
        nodes.push_back(node);
        uint32_t hits, base, imask;
        visit(seed, node, hits, base, imask, oct);
        if (hits == 0) {
            if (stack.empty()) break;
            base = stack.back().x;
            imask = stack.back().y & 0xffu;
            hits = stack.back().y >> 8;
            stack.pop_back();
        }
        const uint32_t slot = (uint32_t)__builtin_ctz(hits) ^ oct;
        node = base + (uint32_t)__builtin_popcount(imask & ((1u << slot) - 1u));
        if (hits & (hits - 1)) {
            if (stack.size() >= limit) break;
            stack.push_back(Entry{base, ((hits & (hits - 1)) << 8) | imask});
        }
    }
    return nodes;
}

bool run(int lanes, uint32_t seed, uint32_t oct, uint32_t limit, const std::vector<int> &order, size_t &total)
{
    constexpr size_t kSteps = 100;
    const std::vector<uint32_t> want = walk_alone(seed, oct, limit, kSteps);
    std::vector<Entry> stack(kDepth);
    std::vector<std::vector<uint32_t>> got(lanes);
    Turns turns(order);
    std::vector<std::thread> pool;
    for (int lane = 0; lane < lanes; ++lane)
        pool.emplace_back([&, lane] {
            std::vector<Entry> over(64);
            int sp = 0;
            uint32_t node = 0;
            bool walking = true;
            turns.begin(lane);
            for (size_t s = 0; s < kSteps; ++s) {  // every lane takes every step, as a warp's do
                uint32_t hits = 0, base = 0, imask = 0;
                if (walking) {
                    got[lane].push_back(node);
                    visit(seed, node, hits, base, imask, oct);
                }
                bool full = false;
                const bool end = dr::team_next_node<kDepth>(walking, lane == 0, oct, base, imask, hits, stack.data(), over.data(),
                                                            limit, sp, node, full, [&] { turns.barrier(lane); });
                walking = walking && !end;
            }
            turns.end();
        });
    for (std::thread &t : pool) t.join();
    for (int lane = 0; lane < lanes; ++lane)
        if (got[lane] != want) {
            size_t i = 0;
            while (i < got[lane].size() && i < want.size() && got[lane][i] == want[i]) ++i;
            std::printf("lane %d of %d, seed %u, octant %u, limit %u: step %zu differs\n", lane, lanes, seed, oct, limit, i);
            return false;
        }
    total += want.size();
    return true;
}

}  // namespace

int main()
{
    size_t total = 0;
    for (int lanes : {4, 8}) {
        std::vector<int> up, down, odd;
        for (int i = 0; i < lanes; ++i) up.push_back(i), down.push_back(lanes - 1 - i), odd.push_back((3 * i + 1) % lanes);
        for (uint32_t seed = 1; seed <= 4; ++seed)
            for (uint32_t limit : {2u, 64u})
                for (const std::vector<int> &order : {up, down, odd})
                    if (!run(lanes, seed, seed & 7u, limit, order, total)) return 1;
    }
    std::printf("ok %zu\n", total);
    return 0;
}
