"""CPU-only checks of the host rules that size launches: a small program includes the launch header and walks every form a rule accepts."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, body):
    from kernelschema_b200 import build
    src = tmp_path / "rules.cu"
    src.write_text('#include <stdio.h>\n#include "kernels.cuh"\nusing namespace b200;\nint main() {\n' + body + "\n}\n")
    exe = str(tmp_path / "rules")
    subprocess.run([build._nvcc(), "-std=c++17", "-I", os.path.join(ROOT, "kernelschema_b200", "csrc"), str(src), "-o", exe], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()


def test_selection_inside_the_route_map_owns_at_most_one_warp_of_routes(tmp_path):
    """The launch that selects experts itself has one warp of 32 lanes per block for the block's own routes, and 32 ids per token in
    shared memory: no accepted call may own more, on a full device or on a slice with few multiprocessors. A full device accepts
    every batch of up to eight tokens and 1024 routes."""
    widest, full = _run(tmp_path, """
  int widest = 0, full = 1;
  for (int sms = 1; sms <= 160; ++sms)
    for (int T = 1; T <= 12; ++T)
      for (int K = 1; K <= 40; ++K)
        for (int S = 0; S <= 130; ++S) {
          const bool fits = route_gather_topk_fits(T, K, S, 256, sms);
          const bool small = T <= 8 && K <= 32 && T * (K + S) <= 1024;
          if (fits && !small) return 1;
          if (sms >= 148 && fits != small) full = 0;
          if (!fits) continue;
          const int total = T * (K + S), chunk = route_gather_chunk(total, kTopkGatherThreads, sms);
          const int blocks = (total + chunk - 1) / chunk;
          if (blocks > sms || blocks * chunk < total) return 1;
          if (chunk > widest) widest = chunk;
        }
  if (route_gather_topk_fits(8, 8, 0, 257, 148)) return 1;
  printf("%d %d", widest, full);
  return 0;""")
    assert int(widest) == 32 and int(full) == 1
