// Host check of the block-wide order by receptor type
// (autogrid_b200/csrc/kernels/type_sort.cuh, the code the kernels run), under
// the weakest memory order that CUDA promises: a thread's shared-memory stores
// become visible to others only at __syncwarp (within its warp) and
// __syncthreads, the stores of different threads in any order; votes and
// shuffles order nothing.  Every thread is a host thread with a list of stores
// in flight; a barrier applies the lists of its threads in a random order.
// Exits 1 where a candidate's place is not that of a stable sort by type.
#include <algorithm>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <mutex>
#include <numeric>
#include <random>
#include <thread>
#include <vector>

#define __device__
#define __forceinline__ inline

constexpr int THREADS = 256, WARPS = THREADS / 32;

// `body` runs once, by the last of n threads to arrive, before any leaves.
class Meeting {
public:
    explicit Meeting(int n) : n_(n) {}
    template <class F> void meet(F body)
    {
        std::unique_lock<std::mutex> lock(mu_);
        const long long round = round_;
        if (++here_ == n_) {
            body();
            here_ = 0;
            round_++;
            cv_.notify_all();
        } else {
            cv_.wait(lock, [&] { return round_ != round; });
        }
    }

private:
    std::mutex mu_;
    std::condition_variable cv_;
    const int n_;
    int here_ = 0;
    long long round_ = 0;
};

struct Store {
    int *at, value;
};
struct Thread {
    int x = 0;
    std::vector<Store> in_flight;
    std::mt19937 rng;
};
thread_local Thread self;
std::vector<Thread *> all(THREADS);
Meeting block(THREADS);
std::vector<std::unique_ptr<Meeting>> warp;
int posted[WARPS][32], seen[WARPS][32];

struct {
    struct {
        operator int() const { return self.x; }
    } x;
} threadIdx;

void apply(int first, int n)
{
    std::vector<int> order(n);
    std::iota(order.begin(), order.end(), first);
    std::shuffle(order.begin(), order.end(), self.rng);
    for (int t : order) {
        for (const Store &s : all[t]->in_flight) *s.at = s.value;
        all[t]->in_flight.clear();
    }
}

void __syncthreads() { block.meet([] { apply(0, THREADS); }); }
void __syncwarp()
{
    const int w = self.x / 32;
    warp[w]->meet([w] { apply(32 * w, 32); });
}

// A warp's values, without any memory order.
const int *exchange(int value)
{
    const int w = self.x / 32;
    posted[w][self.x % 32] = value;
    warp[w]->meet([w] { std::copy(posted[w], posted[w] + 32, seen[w]); });
    return seen[w];
}
unsigned __match_any_sync(unsigned, int value)
{
    const int *v = exchange(value);
    unsigned m = 0;
    for (int l = 0; l < 32; l++)
        if (v[l] == value) m |= 1u << l;
    warp[self.x / 32]->meet([] {});
    return m;
}
int __shfl_up_sync(unsigned, int value, int o)
{
    const int lane = self.x % 32, *v = exchange(value), r = lane >= o ? v[lane - o] : value;
    warp[self.x / 32]->meet([] {});
    return r;
}
int __popc(unsigned v) { return __builtin_popcount(v); }

// Shared ints: a thread sees its own stores, others' only when applied.
struct Cell {
    int *at;
    void operator=(int value) const { self.in_flight.push_back({at, value}); }
    operator int() const
    {
        for (size_t k = self.in_flight.size(); k-- > 0;)
            if (self.in_flight[k].at == at) return self.in_flight[k].value;
        return *at;
    }
};
struct Row {
    int *at;
    Cell operator[](int k) const { return {at + k}; }
};
struct Counts {
    int v[WARPS][32];
    Row operator[](int w) { return {v[w]}; }
};

#include "kernels/type_sort.cuh"

int main(int argc, char **argv)
{
    std::mt19937 rng(argc > 1 ? (unsigned)std::atoi(argv[1]) : 1u);
    for (int w = 0; w < WARPS; w++) warp.emplace_back(new Meeting(32));
    int bad = 0;
    for (int trial = 0; trial < 12; trial++) {
        const int n = trial == 0 ? 0 : trial == 1 ? 1 : trial == 2 ? THREADS : 1 + (int)(rng() % THREADS);
        const int types = 1 + (int)(rng() % 32);
        std::vector<int> type(THREADS, 32), place(THREADS, -1), seed(THREADS);
        for (int t = 0; t < n; t++) type[t] = (int)(rng() % types);
        for (int &s : seed) s = (int)rng();
        Counts counts;
        for (auto &row : counts.v)
            for (int &c : row) c = (int)(rng() % 1000);  // what shared memory held before
        std::vector<std::thread> threads;
        for (int t = 0; t < THREADS; t++)
            threads.emplace_back([&, t] {
                self.x = t;
                self.rng.seed((unsigned)seed[t]);
                all[t] = &self;
                block.meet([] {});
                place[t] = agb::type_sorted_place<WARPS>(counts, type[t], t < n);
                block.meet([] {});
            });
        for (auto &t : threads) t.join();
        std::vector<int> order(n), want(n);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return type[a] < type[b]; });
        for (int k = 0; k < n; k++) want[order[k]] = k;
        for (int t = 0; t < n; t++) bad += place[t] != want[t];
    }
    if (bad) std::printf("%d candidates out of place\n", bad);
    return bad ? 1 : 0;
}
