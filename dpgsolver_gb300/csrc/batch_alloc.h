// Buffers of a batch of directions: all of them for the largest batch that fits, or none.
#pragma once

#include <cstddef>
#include <initializer_list>

namespace dpg {

struct DirBuffer {
	double** p;        // null on entry
	std::size_t per;   // doubles per direction; 0: not needed
};

// The largest batch of most, most / 2, most / 4, .. 1 directions whose buffers can all be had; 0 where not even one
// direction's can, and then (as for every batch that did not fit) nothing is held and the pointers are null.
// get(void**, bytes): true on success; drop(void*).
template <class Get, class Drop>
int alloc_directions(int most, std::initializer_list<DirBuffer> a, std::initializer_list<DirBuffer> b, Get&& get, Drop&& drop)
{
	for (int n = most; n >= 1; n /= 2) {
		bool ok = true;
		for (const auto& list : {a, b})
			for (const DirBuffer& x : list)
				if (ok && x.per && !get((void**)x.p, (std::size_t)n * x.per * sizeof(double))) { *x.p = nullptr; ok = false; }
		if (ok) return n;
		for (const auto& list : {a, b})
			for (const DirBuffer& x : list) {
				if (*x.p) drop(*x.p);
				*x.p = nullptr;
			}
	}
	return 0;
}

} // namespace dpg
