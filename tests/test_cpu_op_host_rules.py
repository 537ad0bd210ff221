"""Host-side rules of the model kernels (flagcx_b200/ops/csrc), compiled without CUDA."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, text, flags=()):
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(text)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", *flags, "-I" + os.path.join(ROOT, "flagcx_b200", "ops", "csrc"),
                           str(src), "-lpthread", "-o", str(exe)])
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout + res.stderr
    return res.stdout


def test_norm_backward_of_few_rows_runs_one_row_per_cta(tmp_path):
    # rows, hidden size -> one row per CTA, where both kernels were measured and differ by more
    # than 3 % on 148 SMs
    cases = [(1, 1024, 1), (64, 4096, 1), (148, 8192, 1), (257, 2048, 1), (257, 3584, 1), (592, 1024, 1), (257, 768, 1), (360, 3584, 1),
             (16, 256, 1), (592, 2048, 1), (296, 1536, 1), (592, 256, 0), (4096, 256, 0), (1021, 2048, 0), (592, 3072, 0),
             (200, 5120, 0), (257, 7168, 0), (4096, 5120, 0), (4096, 4096, 0), (8192, 7168, 0), (1024, 1024, 0), (200, 8192, 0)]
    rows = "".join(f"  bad += fcxops::rmsnormRowPerCta({r}, {h}, 148) != {w} && printf(\"{r} x {h}\\n\");\n" for r, h, w in cases)
    _run(tmp_path, '#include <cstdio>\n#include <initializer_list>\n#include "norm_route.h"\nint main() {\n  int bad = 0;\n' + rows + """
  for (int sms : {1, 20, 148}) // no CTA ever gets more rows than the kernel has slots for
    for (int H = 8; H <= 16384; H += 8)
      for (long rows = 1; rows <= 5 * sms; ++rows)
        if (fcxops::rmsnormRowPerCta(rows, H, sms)) bad += rows > fcxops::kNormFewRows * (rows < 2 * sms ? rows : 2L * sms) || H > 8192;
  return bad != 0;
}
""")


def test_a_limit_is_set_once_per_device_and_never_skipped(tmp_path):
    """Eight threads on three devices; the first call of a device fails and is tried again."""
    _run(tmp_path, """
#include <cstdio>
#include <thread>
#include <vector>
#include "launch_state.h"
int main() {
  fcxops::OncePerDevice once;
  std::atomic<int> calls[3] = {}, bad{0};
  if (once(1, [&] { return ++calls[1], 7; }) != 7) return 1; // passed on
  std::vector<std::thread> ts;
  for (int k = 0; k < 8; ++k)
    ts.emplace_back([&, k] {
      for (int i = 0; i < 3000; ++i) {
        const int d = (k + i) % 3;
        if (once(d, [&] { return ++calls[d], 0; }) != 0) ++bad;
        if (calls[d] == 0) ++bad; // whoever goes on finds it set
      }
    });
  for (auto &t : ts) t.join();
  for (int d = 0; d < 3; ++d)
    if (calls[d] < 1 || calls[d] > 9) return 2; // at most once per thread that came first together
  int far = 0;
  for (int i = 0; i < 2; ++i) once(64, [&] { return ++far, 0; });
  return bad || far != 2;
}
""")


def test_cluster_count_is_kept_per_device_and_shape(tmp_path):
    _run(tmp_path, """
#include "launch_state.h"
int main() {
  fcxops::ClusterCount count;
  int asked = 0, n = 0, bad = 0;
  auto get = [&](int dev, int smem, int ctas, int answer) {
    if (count(dev, smem, ctas, [&](int *c) { ++asked; *c = answer; return 0; }, &n) != 0) ++bad;
    return n;
  };
  bad += get(0, 65536, 4, 71) != 71 || get(0, 65536, 4, 99) != 71 || asked != 1;
  bad += get(1, 65536, 4, 30) != 30 || asked != 2; // another device
  bad += get(1, 65520, 4, 31) != 31 || get(1, 65520, 8, 12) != 12 || asked != 4;
  bad += get(1, 0, 1, 0) != 1 || get(2, 0, 1, 1 << 20) != 0xffff;
  if (count(3, 16, 1, [&](int *) { return 5; }, &n) != 5) ++bad; // passed on, nothing kept
  bad += get(3, 16, 1, 9) != 9;
  return bad;
}
""")


def test_launch_count_can_be_set():
    from flagcx_b200 import ops
    before = ops.launch_count
    try:
        ops.launch_count = 5
        ops._count(2)
        assert ops.launch_count == 7
    finally:
        ops.launch_count = before


def test_tensors_without_memory_are_refused():
    """Fake tensors (export, shape propagation) have no address: a kernel must not get it."""
    import pytest
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from flagcx_b200 import ops
    e = ops.ext()
    with FakeTensorMode():
        x = torch.empty(4, 512, device="cuda", dtype=torch.bfloat16)
        w, r, t = x.new_empty(512), x.new_empty(4, dtype=torch.float32), x.new_empty(4, dtype=torch.long)
        for call in (lambda: ops.swiglu(x), lambda: ops.rmsnorm_branch(x, w), lambda: ops.rope_fused_qkv(x, 4, 2, 64),
                     lambda: e.swiglu_bwd(x[:, :256].contiguous(), x), lambda: e.rmsnorm_bwd(x, x, w, r),
                     lambda: e.rope_inplace(x.view(4, 8, 64), None, 1e4, False), lambda: e.cross_entropy_fwd_bwd_(x, t, 1.0),
                     lambda: ops.adamw_flat_(x, x, x, x, 1e-3, 0.9, 0.95, 1e-8, 0.1, 1)):
            with pytest.raises(RuntimeError, match="not allocated"):
                call()


def test_a_tensor_subclass_takes_the_python_functions():
    """What they do to it goes through the subclass (the skip output of a norm keeps its class)."""
    import torch
    from flagcx_b200 import ops
    x = torch.zeros(2)
    assert not ops._in_python(x) and not ops._in_python(torch.nn.Parameter(x))
    assert ops._in_python(x.as_subclass(type("Own", (torch.Tensor,), {})))
