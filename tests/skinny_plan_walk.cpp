// Walks the plans of csrc/skinny_plan.h: every plan that a launch would use stays within what the kernel keeps and the GPU has, and reads
// every block of K once, int8 weights in the order of the kernels whose sums it repeats.  Prints what does not hold; 0 findings: exit 0.
#include <stdio.h>

#include <vector>

#include "skinny_plan.h"

static int findings = 0;
static void found(const char* what, int type, bool glu, int M, int N, int K, int block, const SkPlan& p) {
  if (findings++ < 20)
    printf("%s: type %d glu %d M %d N %d K %d block %d: tr %d tiles %d tp %d ks %d units %d runs %d slice %d pieces %d stages %d smem %d\n", what, type, glu, M, N, K,
           block, p.tr, p.tiles, p.tp, p.ks, p.units, p.runs, p.slice, p.pieces, p.stages, p.smem);
}

// blocks of 64 k that warp `k` of a tile multiplies, in order (-1: past K)
static std::vector<int> blocks_of(const SkPlan& p, int K, int k) {
  std::vector<int> out;
  for (int piece = 0; piece < p.pieces; piece++)
    for (int u = 0; u < p.units; u++)
      for (int h = 0; h < 2; h++) {
        const int per = p.slice / p.units, q = piece / per * p.ks + k;  // the box's slice; past the last one it reads zeros
        out.push_back(q < K / 128 / p.slice ? (q * p.slice + piece % per * p.units + u) * 2 + h : -1);
      }
  while (!out.empty() && out.back() < 0) out.pop_back();  // zeros at the end add nothing
  return out;
}

static void walk(int type, bool glu, int M, int N, int K, int block, int sms) {
  int shift = 0;
  while (block && (1 << shift) < block) shift++;
  const SkPlan p = sk_plan(type, glu, M, N, K, shift, sms);
  if (!p.ok) return;
  auto bad = [&](const char* what) { found(what, type, glu, M, N, K, block, p); };
  const int nt = M <= 8 ? 1 : 2, to = glu ? 8 : 16, nw = glu ? 2 : 1, per = (N + p.grid - 1) / p.grid, passes = (per + p.tr - 1) / p.tr;
  const int warps = (p.tiles + p.tp - 1) / p.tp, head = sk_head(type, nt, p.tp), row_bytes = type == SK_NF4 ? K / 2 : type == SK_W8 ? K : K * 2;
  if (p.units > sk_units(type, nt)) bad("more runs of a stage than a warp has offsets for");
  if (p.stages < 2 || p.stages > SK_MAX_STAGES) bad("stages");
  if (p.smem + 1024 + 64 > 227 * 1024 || p.smem != head + 4096 + p.stages * p.stage_bytes) bad("shared memory");
  if (p.tp > 2 || warps * p.ks > SK_WARPS || p.tiles * to < p.tr || p.tiles > 16) bad("warps");
  if (p.tr > 256 || p.runs * sk_runs_x(type) > 256 || M > 256 || p.tr < 1) bad("box");
  if ((long long)passes * p.tr < per) bad("outputs left out");
  // one thread finishes a sum for at most EPT tiles' worth
  if (p.tiles * nt * 4 > SK_WARPS * 4 * nt) bad("sums to finish");
  // the furthest fragment: the last row of the last tile of the last warp, in the last run of the last stage
  const int w_al = sk_align(p.runs * p.tr * 128, 1024), x_al = sk_align(p.runs * sk_runs_x(type) * M * 128, 1024), s_al = sk_align(p.tr * p.sp, 128);
  const int last_row = (warps * p.tp - 1) * to + to - 1, stage = (p.stages - 1) * p.stage_bytes;
  const int far_w = stage + (nw - 1) * w_al + ((p.runs - 1) * p.tr + last_row) * 128 + 128;
  const int far_s = stage + nw * w_al + x_al + (nw - 1) * s_al + last_row * p.sp + p.sp;
  if (head + far_w > p.smem || head + far_s > p.smem) bad("fragment past the ring");
  if (nw * p.tr * (p.runs * 128 + p.sp) + M * sk_runs_x(type) * p.runs * 128 >= 1 << 20) bad("bytes of a stage");
  if (type == SK_NF4 && (p.sp % 16 != 0 || p.sp != p.runs * (512 >> shift))) bad("scales of a stage");
  if (type != SK_W8) {
    if (p.runs != p.ks * p.units || p.pieces != (row_bytes / 128 + p.runs - 1) / p.runs) bad("runs");
    return;
  }
  if (p.pieces * p.runs * 128 - K >= p.ks * p.slice * 128) bad("stages past K");
  for (int k = 0; k < p.ks; k++) {
    std::vector<int> want;
    const int kt = gs_k_tile(nt * 8, p.ks, true), kw = kt / p.ks;
    for (int t = 0; t < K; t += kt)
      for (int b = t + k * kw; b < t + (k + 1) * kw; b += 64)
        if (b < K) want.push_back(b / 64);
    if (blocks_of(p, K, k) != want) bad("order of K");
  }
}

int main() {
  const int Ks[] = {64, 128, 192, 256, 384, 512, 576, 768, 1024, 1152, 1536, 1792, 2048, 2176, 2304, 3072, 3584, 4096, 5120, 6656, 7168, 8192, 11008, 13824, 14336, 28672};
  const int odd[] = {30001, 32000, 50257, 65536, 100003, 128256, 140000, 151936, 256000};
  std::vector<int> Ns;
  for (int n = 1; n < 30000; n += n < 200 ? 1 : n < 5000 ? 37 : 149) Ns.push_back(n);
  for (int n : {2048, 3072, 4096, 5120, 6144, 8192, 11008, 14336, 28672}) Ns.push_back(n);
  for (int n : odd) Ns.push_back(n);
  long long plans = 0;
  for (int sms : {148, 132})
    for (int K : Ks)
      for (int N : Ns)
        for (int glu = 0; glu < 2; glu++) {
          for (int M = 1; M <= 16; M++) {
            if (K % 64 == 0 && (M <= 8 || !glu)) walk(SK_F16, glu, M, N, K, 0, sms), plans++;
            if (K % 128 == 0 && (M <= 8 || !glu)) walk(SK_W8, glu, M, N, K, 0, sms), plans++;
          }
          for (int block = 32; block <= 256; block *= 2)
            if (K % (8 * block) == 0 && K % 256 == 0)
              for (int M : {1, 2, 4, 5, 8}) walk(SK_NF4, glu, M, N, K, block, sms), plans++;
        }
  printf("%lld plans, %d findings\n", plans, findings);
  return findings != 0;
}
