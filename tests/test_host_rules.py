"""CPU-only checks of the host rules that size launches: a small program includes the launch header and walks every form a rule accepts."""
import os
import re
import subprocess
import sys
import threading

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


def test_no_cluster_kernel_lets_the_next_launch_in_early():
    """A kernel that runs as clusters releases its dependents by its end alone: it has no pdl_trigger, or only where it runs without
    a cluster. (Blocks of a next launch that wait on the SMs while clusters look for room are what this rules out.)"""
    csrc, seen = os.path.join(ROOT, "kernelschema_b200", "csrc"), set()
    for name in sorted(os.listdir(csrc)):
        if not name.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, name)).read())
        for kernel in re.split(r"\b__global__\b", text)[1:]:
            body = kernel[:kernel.index("\n}\n")]
            if "cluster" not in body:
                continue
            seen.add(re.search(r"\b(k_\w+)\s*\(", body).group(1))
            for line in re.findall(r"[^\n]*pdl_trigger\(\);", body):
                assert re.match(r"\s*if \((k_)?split == 1\) pdl_trigger\(\);", line), (name, line)
    assert seen == {"k_gemm_nvfp4_pair", "k_gemm_bf16_pair", "k_gemm_w4a16_decode", "k_router_logits_ksplit"}


def test_expanded_weights_need_a_workspace_on_a_32_byte_boundary(tmp_path):
    """The entry accepts a workspace on any 16-byte boundary; the expansion stores 32 bytes at a time and takes only one on a 32-byte
    boundary that holds all weights."""
    assert _run(tmp_path, """
  const int64_t n = 128, k = 1280;
  for (uintptr_t at = 1 << 20; at < (1 << 20) + 512; at += 16)
    for (int64_t bytes : {(int64_t)-1, (int64_t)0, n * k * 2 - 1, n * k * 2, n * k * 2 + 1})
      if (w4a16_expand_room((const void*)at, bytes, n, k) != (at % 32 == 0 && bytes >= n * k * 2)) return 1;
  printf("%d", (int)w4a16_expand_room(nullptr, n * k * 2, n, k));
  return 0;""") == ["0"]


def test_split_k_scratch_of_many_threads(monkeypatch):
    """Threads that use more streams than a thread keeps scratch for: every call gets a buffer that no other thread holds, nothing
    raises while buffers are replaced, and each thread keeps at most eight."""
    import torch
    from kernelschema_b200 import ops
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    held, errors, kept = [set() for _ in range(12)], [], [0] * 12
    done = threading.Barrier(12)

    def work(i):
        try:
            for j in range(1500):
                ws = ops._w4a16_workspace(torch.device("cpu"), (i + j * 5) % 24, 64 + (j % 3) * 64)
                assert ws.numel() >= 64 + (j % 3) * 64
            mine = ops._W4A16_WORKSPACE.kept
            held[i], kept[i] = {w.data_ptr() for w in mine.values()}, len(mine)
        except Exception as exc:
            errors.append(repr(exc))
        done.wait(60)                                   # the buffers of all threads are alive at the same time

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=work, args=(i,)) for i in range(12)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not errors, errors
    assert max(kept) <= 8 and len(set().union(*held)) == sum(kept)


def test_w4a16_scratch_of_a_captured_call_lies_in_a_graph_pool(monkeypatch):
    """On a stream that is being captured a call keeps scratch only of a graph's pool; in ordinary memory (a capture that torch did not
    begin), under an allocator that does not tell, and where there is no memory, many rows run without."""
    import torch
    from kernelschema_b200 import ops
    pool = []
    monkeypatch.setattr(torch.cuda, "memory_snapshot", lambda: [dict(address=0, total_size=1 << 62, **p) for p in pool])
    dev = torch.device("cpu")
    for capturing, pool[:], kept in ((False, [], True), (True, [dict(segment_pool_id=(1, 0))], True), (True, [dict(segment_pool_id=(0, 3))], True),
                                     (True, [dict(segment_pool_id=(0, 0))], False), (True, [dict()], False), (True, [], False)):
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
        for ws in (ops._w4a16_expanded(dev, 4096), ops._w4a16_workspace(dev, 7, 4096)):
            assert (ws is not None) == kept and (ws is None or ws.numel() >= 4096)

    def no_memory(*args, **kwargs):
        raise torch.OutOfMemoryError("none left")

    monkeypatch.setattr(torch, "empty", no_memory)
    for capturing in (False, True):
        assert ops._w4a16_expanded(dev, 4096) is None
