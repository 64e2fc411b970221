// A model of the exchanges of the cluster sort (k_codes_sort): blocks that send
// each other the digit counts and the pairs of their passes, messages that
// arrive in any order and as late as can be, and the mbarriers that count them.
// Searches every schedule of `blocks` blocks and four passes.
//
//   argv: blocks, and for each of the three passes that send pairs a digit per
//   (from, to): 1 if `from` has pairs for `to`.
//   Prints "ok STATES", or "wrong WHAT" for a schedule in which a block reads
//   another pass's counts or pairs, or an array is written that is still read,
//   or nobody can go on.
//
// A block's steps in pass p: 0 expect the bytes of the pass and send the counts;
// 1 wait for the counts; 2 read them, send the pairs; 3 wait for the pairs.
// (Within a block all threads have sent a pass's counts before any goes past
// the block's barrier that follows its wait, hence before its pairs.)
#include "../forceatlas2_rc_gb300/csrc/cluster_exchange.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <string>
#include <vector>

using namespace fa2cu;

constexpr int B = 3, PASSES = 4;
struct Bar { // one arrival a phase, and the messages counted against the expected
    signed char phase, arrived, tx;
    void settle()
    {
        if (arrived && tx == 0) phase++, arrived = 0;
    }
    void expect(int n) { arrived = 1, tx += n, settle(); }
    void message() { tx--, settle(); }
    bool done(unsigned parity) const { return (unsigned) (phase & 1) != parity; }
};
struct State {
    signed char pass[B], step[B];
    Bar counts[B][CS_COUNT_BARS], pairs[B];
    signed char table[B][2][B];  // [at][half][from]: the pass whose counts these are
    signed char array[B][2][B];  // [at][array][from]: the pass whose pairs these are
    // under way: [from][to], the pass + 1; at most two of a kind
    signed char count_msg[B][B][2], pair_msg[B][B][2];
};

static int blocks;
static bool flow[PASSES - 1][B][B];

static bool put(signed char (&m)[2], int pass)
{
    for (auto &x : m)
        if (!x) return x = pass + 1, true;
    return false;
}

// What is wrong with the move, or null. `to` is the state after it.
static const char *step(const State &s, int b, State &to, bool &can)
{
    to = s;
    can = true;
    const int p = s.pass[b];
    if (p == PASSES) return can = false, nullptr;
    switch (s.step[b]) {
    case 0: {
        to.counts[b][cs_count_bar(p)].expect(blocks);
        if (p < PASSES - 1) {
            int n = 0;
            for (int x = 0; x < blocks; x++) n += flow[p][x][b];
            to.pairs[b].expect(n);
        }
        // the pass's own pairs (the codes, at first), read for the ranks
        for (int x = 0; p > 0 && x < blocks; x++)
            if (flow[p - 1][x][b] && s.array[b][p & 1][x] != p - 1) return "pairs read";
        for (int y = 0; y < blocks; y++)
            if (!put(to.count_msg[b][y], p)) return "model too small";
        break;
    }
    case 1: can = s.counts[b][cs_count_bar(p)].done(cs_count_parity(p)); break;
    case 2:
        for (int x = 0; x < blocks; x++)
            if (s.table[b][p & 1][x] != p) return "counts read";
        if (p < PASSES - 1)
            for (int y = 0; y < blocks; y++)
                if (flow[p][b][y] && !put(to.pair_msg[b][y], p)) return "model too small";
        break;
    case 3: can = p == PASSES - 1 || s.pairs[b].done(p & 1); break;
    }
    if (++to.step[b] == 4) to.step[b] = 0, to.pass[b]++;
    return nullptr;
}

static const char *deliver(const State &s, int x, int y, int q, bool counts, State &to, bool &can)
{
    to = s;
    signed char &m = counts ? to.count_msg[x][y][q] : to.pair_msg[x][y][q];
    can = m != 0;
    if (!can) return nullptr;
    const int p = m - 1;
    m = 0;
    // still to be read at y?
    if (counts) {
        if (s.pass[y] < p - 2 || (s.pass[y] == p - 2 && s.step[y] <= 2)) return "counts overwritten";
        to.table[y][p & 1][x] = p;
        to.counts[y][cs_count_bar(p)].message();
    } else { // into the array that held the pairs of pass p - 1
        if (s.pass[y] < p - 1 || (s.pass[y] == p - 1 && s.step[y] <= 2)) return "pairs overwritten";
        to.array[y][(p + 1) & 1][x] = p;
        to.pairs[y].message();
    }
    return nullptr;
}

int main(int argc, char **argv)
{
    if (argc != 3) return 2;
    blocks = atoi(argv[1]);
    const char *f = argv[2];
    if (blocks < 1 || blocks > B || (int) strlen(f) != (PASSES - 1) * blocks * blocks) return 2;
    for (int p = 0; p < PASSES - 1; p++)
        for (int x = 0; x < blocks; x++)
            for (int y = 0; y < blocks; y++) flow[p][x][y] = *f++ == '1';
    State first;
    memset(&first, 0, sizeof first);
    memset(first.table, -1, sizeof first.table);
    memset(first.array, -1, sizeof first.array);
    std::set<std::string> seen;
    std::vector<State> todo{first};
    auto key = [](const State &s) { return std::string((const char *) &s, sizeof s); };
    seen.insert(key(first));
    while (!todo.empty()) {
        const State s = todo.back();
        todo.pop_back();
        bool any = false, end = true;
        for (int b = 0; b < blocks; b++) end &= s.pass[b] == PASSES;
        auto next = [&](const char *wrong, const State &to, bool can) {
            if (!can) return true;
            if (wrong) return printf("wrong: %s\n", wrong), false;
            any = true;
            if (seen.insert(key(to)).second) todo.push_back(to);
            return true;
        };
        State to;
        bool can;
        for (int b = 0; b < blocks; b++) {
            const char *wrong = step(s, b, to, can);
            if (!next(wrong, to, can)) return 0;
        }
        for (int x = 0; x < blocks; x++)
            for (int y = 0; y < blocks; y++)
                for (int q = 0; q < 2; q++)
                    for (bool counts : {true, false}) {
                        const char *wrong = deliver(s, x, y, q, counts, to, can);
                        if (!next(wrong, to, can)) return 0;
                    }
        if (!any && !end) return printf("wrong: nobody can go on\n"), 0;
    }
    printf("ok %zu\n", seen.size());
    return 0;
}
