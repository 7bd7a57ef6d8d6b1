// Walks the pixels that the plane-staging depthwise kernel reads as words, over tensors of a few bytes at every alignment,
// and counts the words of which a byte lies outside the tensor. Host code only.
#include <cstdio>

#include "unaligned16.cuh"

int main()
{
  int words = 0, outside = 0;
  for (int B = 1; B <= 5; B++)
    for (int H = 1; H <= 3; H++)
      for (int W = 1; W <= 6; W++)
        for (int C = 1; C <= 40; C++)
          for (int start = 0; start < 4; start++)
            for (int b = 0; b < B; b++) {
              const int own = H * W * C, off = b * own, lead = (start + off) & 3;
              const pulpnn::ImageSpan span(lead, own, (size_t)off, (size_t)(B - 1 - b) * own);
              for (int iy = 0; iy < H; iy++)
                for (int pad = 1; pad <= 2; pad++)
                  for (int ix = -pad; ix < W; ix += 4)
                    for (int c = 0; c < C; c += 4) {
                      const int at = (iy * W + ix) * C + c + lead;
                      if (!span.holds_words(at, C)) continue;
                      for (int i = 0; i < 4; i++) {
                        if (ix + i < 0 || ix + i >= W) continue;
                        const int first = off - lead + ((at + i * C) & ~3);
                        words += 2;
                        outside += (first < 0) + (first + 8 > B * own);
                      }
                    }
            }
  printf("%d %d\n", words, outside);
  return 0;
}
