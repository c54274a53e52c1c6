// The index arithmetic of the block copies (copy_first, copy_entry, copy_next in ctg_kernels.h), walked on the host as
// k_permute and k_rowmap walk it: every entry of a chunk once and none outside, up to blocks of 2^31 - 1 entries.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "ctg_kernels.h"
using namespace ctg;

int main()
{
	int bad = 0;
	const unsigned threads = 256;
	for (i64 n : {(i64)1, (i64)255, (i64)4097, (i64)1 << 30, ((i64)1 << 31) - 1025, ((i64)1 << 31) - 769, ((i64)1 << 31) - 256, ((i64)1 << 31) - 1})
		for (i64 start : {(i64)0, (n - 1) / COPY_CHUNK * COPY_CHUNK})
		{
			const i64 end = std::min(n, start + (i64)COPY_CHUNK);
			std::vector<int> seen((size_t)(end - start), 0);
			for (unsigned t = 0; t < threads; t++)
			{
				int rounds = 0;
				for (auto e0 = copy_first(start, t); e0 < (decltype(e0))end && rounds++ < COPY_CHUNK; e0 = copy_next(e0, threads))
					for (int u = 0; u < COPY_BATCH; u++)
					{
						const auto e = copy_entry(e0, u, threads);
						if (!(e < (decltype(e))end)) continue;
						if ((i64)e < start || (i64)e >= end) bad++;
						else seen[(size_t)((i64)e - start)]++;
					}
				if (rounds > COPY_CHUNK / (int)threads) bad++;
			}
			for (int s : seen) bad += s != 1;
		}
	printf("mismatches: %d\n", bad);
	return bad != 0;
}
