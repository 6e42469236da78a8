// Prints plan_tail() of the queue lengths on standard input:
// maxBounces firstBounce tailPaths neeCount costRule launched keep count length...
#include "../../mufflon_b200/csrc/trace/wavefront.hpp"
#include <cstdio>

int main() {
	int m, f, t, n, r, l, k, c;
	while(std::scanf("%d %d %d %d %d %d %d %d", &m, &f, &t, &n, &r, &l, &k, &c) == 8) {
		unsigned queue[mb::WF_BOUNCE_STATS] = {};
		for(int i = 0; i < c; ++i)
			if(std::scanf("%u", queue + i) != 1) return 1;
		std::printf("%d\n", mb::plan_tail(queue, m, f, t, n, r != 0, l, k));
	}
	return 0;
}
