// Schedule of the Trotter rotations of whole time steps (rotsched.h).
#include "rotsched.h"

#include <algorithm>

int nise_step_schedule(const std::vector<int2> &pairs, int n, int ts, int steps, std::vector<uint32_t> &rows) {
    const size_t K = pairs.size();
    std::vector<int> last(n, 0);
    std::vector<std::vector<uint32_t>> level;
    for (int w = 0; w < steps; w++)
        for (int s = 0; s < ts; s++)
            for (size_t k = 0; k < K; k++) {
                const int l = std::max(last[pairs[k].x], last[pairs[k].y]);
                last[pairs[k].x] = last[pairs[k].y] = l + 1;
                if ((int)level.size() == l) level.emplace_back();
                level[l].push_back((uint32_t)k | (uint32_t)w << 20 | (uint32_t)(s == 0) << 30 |
                                   (uint32_t)(s == ts - 1) << 31);
            }
    rows.clear();
    for (const auto &l : level)
        for (size_t q = 0; q < l.size(); q += 32)
            for (size_t i = 0; i < 32; i++) rows.push_back(q + i < l.size() ? l[q + i] : NISE_SCHED_NONE);
    return (int)level.size();
}

void nise_schedule_parts(const std::vector<int2> &pairs, int n, std::vector<uint32_t> &parts, std::vector<int> &iso) {
    const int K = (int)pairs.size();
    std::vector<int> first(n, -1), last(n, -1);
    for (int k = 0; k < K; k++)
        for (int a : {pairs[k].x, pairs[k].y}) {
            if (first[a] < 0) first[a] = k;
            last[a] = k;
        }
    parts.resize(K);
    for (int k = 0; k < K; k++) {
        const int a = pairs[k].x, b = pairs[k].y;
        parts[k] = (uint32_t)a | (uint32_t)b << 14 | (uint32_t)(first[a] == k) << 28 | (uint32_t)(first[b] == k) << 29 |
                   (uint32_t)(last[a] == k) << 30 | (uint32_t)(last[b] == k) << 31;
    }
    iso.clear();
    for (int a = 0; a < n; a++)
        if (first[a] < 0) iso.push_back(a);
}

int nise_row_schedule(const std::vector<int2> &pairs, int n, int ts, int width, std::vector<uint32_t> &ab,
                      std::vector<uint16_t> &id) {
    std::vector<int> ready(n, 0);               // first row after the site's last operation
    std::vector<std::vector<uint2>> row;
    std::vector<int> next;                      // next[r]: a row >= r that may have room (path-compressed)
    auto place = [&](int a, int b, uint32_t y) {
        int r = std::max(ready[a], ready[b]);
        while (r < (int)next.size() && next[r] != r) r = next[r] = next[r] < (int)next.size() ? next[next[r]] : next[r];
        while (r >= (int)row.size()) {
            next.push_back((int)row.size());
            row.emplace_back();
        }
        row[r].push_back(make_uint2((uint32_t)a | (uint32_t)b << 16, y));
        if ((int)row[r].size() == width) next[r] = r + 1;
        ready[a] = ready[b] = r + 1;
    };
    for (int s = 0; s < ts; s++) {
        for (int a = 0; a < n; a++) place(a, a, NISE_ROW_PHASE | (uint32_t)a);
        for (size_t k = 0; k < pairs.size(); k++) place(pairs[k].x, pairs[k].y, (uint32_t)k);
        for (int a = 0; a < n; a++) place(a, a, NISE_ROW_PHASE | (uint32_t)a);
    }
    const int nrow = (int)row.size();
    ab.clear();
    id.clear();
    for (int r = 0; r < nrow + 2; r++)
        for (int i = 0; i < width; i++) {
            const uint32_t spare = (uint32_t)(n + i);
            const bool op = r < nrow && i < (int)row[r].size();
            ab.push_back(op ? row[r][i].x : spare | spare << 16);
            id.push_back((uint16_t)(op ? row[r][i].y : NISE_ROW_PHASE | (uint32_t)n));
        }
    return nrow;
}
