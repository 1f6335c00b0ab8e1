// Reads calls from standard input and prints what csrc/sddmm_route.h makes of them, for 148 SMs:
//   alone M K N nnz masked wide         ->  taken (0/1) and the microseconds of the tensor cores
//   group count, then M K N nnz each    ->  problems taken, and the microseconds of the launch over those that would be
#include <cstdio>
#include <cstring>

#include ROUTE_HEADER

using namespace dlspm;

int main()
{
    char kind[8];
    while (scanf("%7s", kind) == 1) {
        if (!strcmp(kind, "alone")) {
            SddmmSizes q = {};
            int masked, wide;
            if (scanf("%d %d %d %lf %d %d", &q.M, &q.K, &q.N, &q.nnz, &masked, &wide) != 6) return 1;
            q.masked = masked != 0;
            q.wide = wide != 0;
            printf("%d %.3f\n", pick_pays_alone(148, q) ? 1 : 0, pick_takes(q) ? pick_shape(148, q).us : 0.0);
            continue;
        }
        int n;
        if (scanf("%d", &n) != 1) return 1;
        std::vector<SddmmSizes> problems, dense;
        for (int i = 0; i < n; i++) {
            SddmmSizes q = {};
            q.wide = true;
            if (scanf("%d %d %d %lf", &q.M, &q.K, &q.N, &q.nnz) != 4) return 1;
            problems.push_back(q);
        }
        std::vector<unsigned char> chosen(problems.size());
        sddmm_route_group(148, problems, chosen.data());
        int taken = 0;
        for (size_t i = 0; i < problems.size(); i++) {
            taken += chosen[i];
            if (chosen[i]) dense.push_back(problems[i]);
        }
        printf("%d %.3f\n", taken, dense.empty() ? 0.0 : pick_group_us(148, dense));
    }
    return 0;
}
