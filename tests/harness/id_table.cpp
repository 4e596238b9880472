// Test harness (CPU): the bigraph-id lookup (gaf_format.cuh: IdTable) against a std::map, on both
// sides of the rule that chooses direct indexing.
#include <algorithm>
#include <cstdio>
#include <map>
#include <random>
#include "../../graphaligner_gb300/csrc/gaf_format.cuh"

static bool check(const char* what, const std::vector<int32_t>& ids, bool dense)
{
    gaf::IdTable t;
    t.build({ 7, 1 << 30 });            // tables are rebuilt from any earlier state
    t.build(ids);
    std::map<int32_t, uint32_t> want;
    for (size_t i = 0; i < ids.size(); i++) want[ids[i]] = (uint32_t)i;
    std::vector<int32_t> ask = { INT32_MIN, INT32_MIN + 1, -1, 0, 1, INT32_MAX - 1, INT32_MAX };
    for (int32_t id : ids)
    {
        ask.push_back(id);
        if (id > INT32_MIN) ask.push_back(id - 1);
        if (id < INT32_MAX) ask.push_back(id + 1);
    }
    bool ok = t.key.empty() == dense;
    for (int32_t id : ask)
    {
        const auto f = want.find(id);
        ok = ok && t.find(id) == (f == want.end() ? gaf::kNoId : f->second);
    }
    if (!ok) printf("FAIL %s\n", what);
    return ok;
}

int main()
{
    std::mt19937 rng(11);
    bool ok = check("none", {}, true) && check("one", { 5 }, true) && check("ends", { INT32_MIN, INT32_MAX }, false);
    std::vector<int32_t> ids;
    for (int32_t i = 0; i < 5000; i++) ids.push_back(2 * i + 100);
    ok = check("ascending", ids, true) && ok;
    std::shuffle(ids.begin(), ids.end(), rng);
    ids.push_back(ids[3]);              // an id given twice
    ok = check("shuffled", ids, true) && ok;
    // the rule's line: a range of 4 n + 16 is dense, one more is not
    for (int32_t n : { 2, 3, 1000 })
        for (int32_t over : { 0, 1 })
        {
            ids.clear();
            for (int32_t i = 0; i + 1 < n; i++) ids.push_back(-7 + i);
            ids.push_back(-7 + 4 * n + 16 - 1 + over);
            ok = check("line", ids, over == 0) && ok;
        }
    ids.clear();
    for (int32_t i = 0; i < 5000; i++) ids.push_back((int32_t)rng());
    ids.push_back(INT32_MIN);
    ids.push_back(ids[9]);
    ok = check("random", ids, false) && ok;
    ids.clear();
    for (int32_t i = 0; i < 5000; i++) ids.push_back((i - 2500) * 65536);
    ok = check("strided", ids, false) && ok;
    if (ok) printf("ok\n");
    return ok ? 0 : 1;
}
