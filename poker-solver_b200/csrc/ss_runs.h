// ss_runs.h -- which launches of a batch may go side by side.
//
// A batch is a list of merged launches in order.  One traverser's terminal
// launches write disjoint value rows and only read reach, so a run of them
// may be forked over streams and reordered.  Another traverser's write the
// same rows: a run ends where the traverser changes.  (Launches of other
// types usually come between two traversers, but not where the first of them
// makes no decision in any member: then it has no values or reach to update.)
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace ssb {

// The end of the run that starts at launch i: the launches of its type and
// traverser that follow it where it is a terminal launch, else itself alone.
template <class Launch, class Terminal>
size_t run_end(const std::vector<Launch> &q, size_t i, Terminal terminal) {
    size_t j = i + 1;
    if (terminal(q[i]))
        while (j < q.size() && q[j].type == q[i].type && q[j].t == q[i].t) ++j;
    return j;
}

// Orders every run by weight, the heaviest last.
template <class Launch, class Terminal, class Weight>
void order_runs(std::vector<Launch> *q, Terminal terminal, Weight weight) {
    for (size_t i = 0, j; i < q->size(); i = j) {
        j = run_end(*q, i, terminal);
        std::stable_sort(q->begin() + static_cast<std::ptrdiff_t>(i), q->begin() + static_cast<std::ptrdiff_t>(j),
                         [&](const Launch &x, const Launch &y) { return weight(x) < weight(y); });
    }
}

}  // namespace ssb
