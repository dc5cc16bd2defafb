// Walks the chunks of the embedding backward for the token counts given as arguments and searches
// every chunk border as the kernels do; prints the first violation, or "ok".
#include <stdio.h>
#include <stdlib.h>

#include <initializer_list>

#include "embedding_chunks.h"

int main(int argc, char** argv) {
  for (int a = 1; a < argc; ++a) {
    const long long n = atoll(argv[a]);
    const int ni = (int)n, chunk = dion::emb_chunk(n), count = dion::emb_num_chunks(n, chunk);
    if (count < 1 || count > 1024) return printf("%lld: %d chunks\n", n, count), 1;
    long long at = 0;
    for (int c = 0; c < count; ++c) {
      const int p0 = c * chunk, p1 = dion::emb_chunk_end(p0, chunk, ni);
      if (p0 != at || p1 <= p0 || p1 > ni)
        return printf("%lld: chunk %d is [%d, %d)\n", n, c, p0, p1), 1;
      at = p1;
      for (int target : {p0, p1 - 1}) {                 // the search for a sorted position
        int lo = 0, hi = ni;
        while (lo < hi) {
          const int mid = dion::emb_mid(lo, hi);
          if (mid < lo || mid >= hi) return printf("%lld: middle of [%d, %d) is %d\n", n, lo, hi, mid), 1;
          if (mid < target) lo = mid + 1; else hi = mid;
        }
        if (lo != target) return printf("%lld: search ends at %d, not %d\n", n, lo, target), 1;
      }
    }
    if (at != n) return printf("%lld: chunks end at %lld\n", n, at), 1;
  }
  printf("ok\n");
  return 0;
}
