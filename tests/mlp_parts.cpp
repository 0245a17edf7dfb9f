// The layout of the training workspace's partial sums (csrc/emp_mlp.h): prints the first row count
// nb and workspace size B >= nb whose parts do not fit, or "fits".  Used by test_mlp_parts.py.
#include "emp_mlp.h"

#include <algorithm>
#include <cstdio>

int main()
{
    uint64_t need = 0, by = 0;  // the largest need of any row count so far
    for (uint64_t rows = 1; rows <= 70000; ++rows) {
        const emp::MlpParts p = emp::mlp_parts(rows);
        // every row is in a part, and the parts follow one another
        if (static_cast<uint64_t>(p.z1) * p.w1_rows < rows || static_cast<uint64_t>(p.z2) * p.w2_rows < rows ||
            p.w1_rows % 16 || p.w2_rows % 16 || static_cast<uint64_t>(p.row_tiles) * emp::kMlpTile < rows ||
            static_cast<uint64_t>(p.col_blocks) * emp::kMlpColRows < rows || p.w2 > p.b1 || p.b1 > p.col || p.col > p.end) {
            std::printf("layout of %llu rows\n", static_cast<unsigned long long>(rows));
            return 0;
        }
        if (p.end > need) {
            need = p.end;
            by = rows;
        }
        if (need > emp::mlp_part_floats(rows)) {
            std::printf("%llu rows in a workspace for %llu\n", static_cast<unsigned long long>(by),
                        static_cast<unsigned long long>(rows));
            return 0;
        }
    }
    std::printf("fits\n");
    return 0;
}
