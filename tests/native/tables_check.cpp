// Which tables a plan's request makes (PlanRequest::tables) -- TEST INFRASTRUCTURE ONLY.
#include <string>

#include "../../sycl-fft_b200/csrc/planner.hpp"

using namespace sfb;

// Compares the tables of TableChoice::read with those of TableChoice::all: every table a pass of the plan reads is
// there and equal, every other one is empty, sizes and passes are the same, and TableChoice::none makes none.
// Returns the number of tables left out, or -1 with the difference in `why`.
extern "C" int tables_left_out(int dbl, int fused, unsigned rank, const uint64_t* shape, uint64_t batch, char* why, size_t cap) {
    auto fail = [&](const std::string& what) {
        what.copy(why, cap - 1);
        why[std::min(cap - 1, what.size())] = 0;
        return -1;
    };
    PlanRequest req;
    req.dbl = dbl != 0;
    req.fused_passes = fused != 0;
    req.shape.assign(shape, shape + rank);
    req.batch = batch;
    const PlanSpec all = make_plan(req);
    req.tables = TableChoice::read;
    const PlanSpec read = make_plan(req);
    req.tables = TableChoice::none;
    const PlanSpec none = make_plan(req);
    if (describe_plan(all) != describe_plan(read) || describe_plan(all) != describe_plan(none)) return fail("passes differ");
    if (all.table_sizes != read.table_sizes || all.table_read != read.table_read || all.table_sizes != none.table_sizes)
        return fail("sizes differ");
    for (const PassSpec& ps : read.passes) {
        const TableIds& t = ps.tables;
        const bool own = !fused && (ps.smooth_id >= 0 || ps.conv_id >= 0);
        for (int id : {own ? -1 : t.tw1, own ? -1 : t.tw2, t.premul, t.pointwise, t.postmul, t.tw4_hi, t.tw4_lo, t.smooth, t.spiped})
            if (id >= 0 && !read.table_read[id]) return fail("table " + std::to_string(id) + " is read but not marked");
    }
    int left_out = 0;
    for (size_t i = 0; i < all.tables.size(); ++i) {
        if (all.tables[i].size() != all.table_sizes[i]) return fail("table " + std::to_string(i) + " has another size");
        if (read.table_read[i] ? read.tables[i] != all.tables[i] : !read.tables[i].empty())
            return fail("table " + std::to_string(i) + " differs");
        left_out += read.tables[i].empty();
    }
    return left_out;
}
