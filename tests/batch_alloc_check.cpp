// CPU check of alloc_directions (batch_alloc.h): an allocator that refuses its N-th request, or everything beyond a budget.
// Whatever is refused, the call either holds every buffer of one batch or nothing, and the batch is halved until it fits.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "batch_alloc.h"

int main()
{
	int bad = 0;
	for (int most : {1, 2, 7, 396})
		for (int fail_at = 0; fail_at <= 9; ++fail_at)
			for (size_t budget : {(size_t)-1, (size_t)40000, (size_t)9000, (size_t)700, (size_t)100}) {
				double* p[6] = {};
				std::map<void*, size_t> live;
				size_t used = 0;
				int request = 0;
				auto get = [&](void** q, size_t bytes) {
					if (++request == fail_at || bytes > budget - used) { *q = (void*)8; return false; }   // no pointer on failure
					*q = std::malloc(bytes);
					live[*q] = bytes;
					used += bytes;
					return true;
				};
				auto drop = [&](void* q) {
					if (!live.count(q)) { std::printf("dropped %p, which is not held\n", q); ++bad; return; }
					used -= live[q];
					live.erase(q);
					std::free(q);
				};
				const size_t per[6] = {5, 3, 0, 4, 2, 1};   // 15 doubles a direction
				const int n = dpg::alloc_directions(most, {{&p[0], 5}, {&p[1], 3}, {&p[2], 0}, {&p[3], 4}}, {{&p[4], 2}, {&p[5], 1}}, get, drop);
				bool ok = n >= 0 && n <= most;
				for (int k = 0; k < 6; ++k) {
					const bool held = n > 0 && per[k] > 0;
					ok = ok && (held ? live.count(p[k]) && live[p[k]] == n * per[k] * sizeof(double) : p[k] == nullptr);
				}
				ok = ok && live.size() == (n > 0 ? 5u : 0u);
				// the largest of most, most / 2, .. that the budget takes, one halving more where a request of it was refused
				int want = most;
				while (want >= 1 && budget != (size_t)-1 && want * 15 * sizeof(double) > budget) want /= 2;
				if (fail_at == 0) ok = ok && n == want;
				else ok = ok && (n == want || n == want / 2);
				if (!ok) { std::printf("most %d fail_at %d budget %zu: batch %d\n", most, fail_at, budget, n); ++bad; }
				for (auto& b : live) std::free(b.first);
			}
	std::printf("%s\n", bad ? "FAILED" : "all checks passed");
	return bad ? 1 : 0;
}
