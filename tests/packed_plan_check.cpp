// Checks plan_packed / plan_packed_gw (lutgemm_kernels.h) over random sizes: every row block belongs to one group, every
// cell to one work item or to one item per part of K, and no item is empty.
#include <stdio.h>

#include <random>

#include "lutgemm_kernels.h"

int main() {
    std::mt19937_64 gen(1);
    auto draw = [&](long lo, long hi) { return std::uniform_int_distribution<long>(lo, hi)(gen); };
    long grouped = 0, cut = 0;
    for (int i = 0; i < 100000; ++i) {
        const bool gw = draw(0, 1);
        const int rt = gw ? 512 : 384 + 64 * (int)draw(0, 3), sms = draw(0, 3) ? 148 : (int)draw(1, 200);
        const long rows = draw(1, draw(0, 1) ? 2000 : 300000), cols = draw(1, draw(0, 1) ? 300 : 300000);
        const int K = (int)draw(1, draw(0, 1) ? 70 : 5000);
        const lutgemm::PackedPlan p = gw ? lutgemm::plan_packed_gw(rows, cols, K, sms) : lutgemm::plan_packed(rows, cols, K, rt, sms);
        const long blocks = (rows + rt - 1) / rt, cells = p.groups * ((cols + 63) / 64);
        const bool ok = p.groups >= 1 && (long)p.groups * p.group_blocks >= blocks && (p.groups - 1L) * p.group_blocks < blocks &&
                        p.main_cells >= 0 && p.main_cells <= cells && (p.main_cells == cells || p.tail_parts >= 1) &&
                        p.tail_per % 16 == 0 && (long)p.tail_parts * p.tail_per >= K && (p.tail_parts - 1L) * p.tail_per < K &&
                        !(gw && p.group_blocks > 16);
        if (!ok) {
            printf("rows %ld cols %ld K %d tile %d sms %d: groups %d x %d, main %d, tail %d x %d\n", rows, cols, K, rt, sms,
                   p.groups, p.group_blocks, p.main_cells, p.tail_parts, p.tail_per);
            return 1;
        }
        grouped += p.group_blocks > 1;
        cut += p.main_cells > 0 && p.tail_parts > 1;
    }
    return grouped > 1000 && cut > 1000 ? 0 : 2;
}
