"""Rules that pick a kernel or refuse a call, without a GPU: the launching functions are replaced by recorders."""
import os
import shutil
import subprocess

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture
def wgrad_calls(monkeypatch):
    """Names of the launching functions that the gradients of a linear layer reach, in order."""
    from torsh_b200.ops import linear as L
    calls = []
    monkeypatch.setattr(L, "gemm_wgrad_bias", lambda *a, **k: calls.append("wgrad_bias"))
    monkeypatch.setattr(L, "gemm", lambda a, b, **k: calls.append("gemm") or k.get("out"))
    monkeypatch.setattr(L.ew, "colsum_into", lambda *a: calls.append("colsum"))
    monkeypatch.setattr(L, "dynamic_tiles", lambda: False)
    return calls


def _layer(wmg, bmg, m=512, n=256):
    w, b = torch.zeros(m, n, dtype=torch.bfloat16), torch.zeros(m, dtype=torch.bfloat16)
    w.main_grad, b.main_grad = wmg, bmg
    return torch.zeros(64, m, dtype=torch.bfloat16), torch.zeros(64, n, dtype=torch.bfloat16), w, b


@pytest.mark.parametrize("wmg,bmg,carried", [
    (torch.zeros(512, 256), torch.zeros(512), True),
    (torch.zeros(512, 256, dtype=torch.bfloat16), torch.zeros(512), False),
    (torch.zeros(512, 256), torch.zeros(512, dtype=torch.bfloat16), False),
    (torch.zeros(256, 512), torch.zeros(512), False),
    (torch.zeros(511, 256), torch.zeros(512), False),
    (torch.zeros(512, 256), torch.zeros(256), False),
    (torch.zeros(512, 512)[:, ::2], torch.zeros(512), False),
])
def test_bias_gradient_rides_only_into_fp32_buffers_of_the_right_shape(wgrad_calls, wmg, bmg, carried):
    """The fused launch adds through raw pointers: a buffer that it would overrun goes to the ops that check theirs."""
    from torsh_b200.ops.linear import _wgrad_bgrad
    dy, x, w, b = _layer(wmg, bmg)
    assert _wgrad_bgrad(dy, x, w, "nk", b, True, True) == (None, None)
    assert wgrad_calls == (["wgrad_bias"] if carried else ["gemm", "colsum"])


@pytest.mark.parametrize("main_grads", [True, False])
def test_dynamic_tiles_keep_weight_gradients_off_static_pairs(wgrad_calls, monkeypatch, main_grads):
    """The switch asks for tiles that late CTAs can leave to others; pairs are dealt statically and hold two SMs each."""
    from torsh_b200.ops import linear as L
    m, n, tokens = 4096, 2304, 8192
    w, b = torch.zeros(m, n, dtype=torch.bfloat16), torch.zeros(m, dtype=torch.bfloat16)
    if main_grads:
        w.main_grad, b.main_grad = torch.zeros(m, n), torch.zeros(m)
    dy, x = torch.zeros(tokens, m, dtype=torch.bfloat16), torch.zeros(tokens, n, dtype=torch.bfloat16)
    plans = []
    monkeypatch.setattr(L, "gemm", lambda a, b, **k: plans.append((k.get("bn"), k.get("split_k", 1))) or torch.zeros(m, n))
    monkeypatch.setattr(L, "dynamic_tiles", lambda: True)
    L._wgrad_bgrad(dy, x, w, "nk", b, True, True)
    assert "wgrad_bias" not in wgrad_calls and plans == [L._wgrad_plan(m, n, tokens)]
    monkeypatch.setattr(L, "dynamic_tiles", lambda: False)
    L._wgrad_bgrad(dy, x, w, "nk", b, True, True)
    assert "wgrad_bias" in wgrad_calls


def test_column_sums_refuse_other_buffers(monkeypatch):
    """The kernel adds fp32 values through the buffer's pointer; without the kernel any buffer that add_ takes is fine."""
    from torsh_b200.ops import elementwise as ew
    x, other = torch.ones(4, 8), (torch.zeros(8, dtype=torch.bfloat16), torch.zeros(7), torch.zeros(16)[::2])
    out = torch.zeros(8, dtype=torch.bfloat16)
    ew.colsum_into(x, out)
    assert (out == 4).all()
    calls = []
    monkeypatch.setattr(ew, "kernel_ok", lambda *t: True)
    monkeypatch.setattr(ew, "call", lambda name, *a: calls.append(name))
    monkeypatch.setattr(ew.nv, "stream_ptr", lambda *a: None)
    for bad in other:
        with pytest.raises(AssertionError):
            ew.colsum_into(x, bad)
    assert calls == []
    ew.colsum_into(x, torch.zeros(8))
    assert calls == ["tb_colsum"]


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists(CUDA_INCLUDE), reason="needs g++ and the CUDA headers")
def test_shared_memory_opt_in_is_per_device(tmp_path):
    """More than 48 KB of shared memory is an attribute of a kernel on ONE device: a launcher that sets it once per process
    fails on the second GPU. The helper runs against a fake runtime, and no launcher keeps a flag of its own."""
    exe = str(tmp_path / "smem_opt_in_check")
    src = os.path.join(ROOT, "tests", "native", "smem_opt_in_check.cpp")
    build = subprocess.run(["g++", "-std=c++17", "-O1", "-I", CUDA_INCLUDE, "-I", os.path.join(ROOT, "csrc", "kernels"), src, "-o", exe],
                           capture_output=True, text=True, timeout=300)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout
    assert run.stdout.split() == ["0:100", "1:100", "1:200", "63:200", "2:100!", "2:100", "64:100", "64:100"]
    kernels = os.path.join(ROOT, "csrc", "kernels")
    for name in sorted(os.listdir(kernels)):
        with open(os.path.join(kernels, name)) as f:
            text = f.read()
        assert not ("MaxDynamicSharedMemorySize" in text and "static bool" in text and "configured" in text), name
        assert "static bool cfg" not in text, name


def _route(M, N, K, majors=(0, 0), flags=0, split_k=1, ldd=None, ldr=None):
    """(kernel, tile width, K splits) that a product of these sizes runs on; 148 SMs are assumed without a GPU."""
    from torsh_b200 import _native as nv
    am, bm = majors
    r = nv.cuda().tb_gemm_route(M, N, K, am, bm, M if am else K, N if bm else K, N if ldd is None else ldd, N if ldr is None else ldr,
                                flags, split_k)
    return ("one", 0, 1) if r == 0 else ("pair", 256, 1) if r == 1 else ("split", r % 4096 // 16, r // 4096)


BIAS, GELU, RESIDUAL, OUT_F32, ATOMIC, PREACT, DGELU = 1, 2, 4, 8, 16, 32, 64


def test_rows_that_overlap_stay_off_the_pair_kernel():
    """Its residual comes through a tensor map, which takes no row stride below the row's length (an expanded residual has 0)."""
    shape = (8192, 1024, 4096)
    assert _route(*shape, flags=BIAS | RESIDUAL)[0] == "pair" and _route(*shape, flags=RESIDUAL, ldr=1032)[0] == "pair"
    for ldr in (0, 8, 1016):
        assert _route(*shape, flags=RESIDUAL, ldr=ldr)[0] == "one"
    assert _route(*shape, ldr=0)[0] == "pair"   # no residual: its stride says nothing
    assert _route(*shape, flags=OUT_F32 | ATOMIC, ldd=0)[0] == "one" and _route(*shape, ldd=0)[0] != "pair"


@pytest.mark.parametrize("shape,kernel", [
    ((8192, 4096, 1024), "pair"), ((8192, 1024, 4096), "pair"), ((2048, 4096, 1024), "pair"), ((4096, 50304, 1024), "pair"),
    ((13, 1024, 4096), "split"), ((256, 1024, 1024), "split"), ((1024, 1024, 4096), "split"), ((64, 768, 3072), "split"),
    # three rows of 128: 256-wide one-CTA tiles waste nothing (62 us, pairs 73)
    ((384, 22016, 4096), "one"), ((384, 50304, 1024), "one"),
    # one or two K blocks: what a CTA writes costs more than what it reads (6.0 us, one split CTA per tile 6.9)
    ((8192, 256, 64), "one"), ((3136, 512, 128), "one"), ((1500, 1024, 256), "one"), ((512, 4096, 8), "one"),
    # fewer rows than half a pair's
    ((1, 50304, 768), "one"), ((128, 50304, 1024), "one")])
def test_route_takes_the_faster_kernel(shape, kernel):
    """Products timed on all three kernels, on both sides of where the choice changes."""
    assert _route(*shape)[0] == kernel


def _params(test, name):
    import test_kernels_gpu as G
    marks = [m for m in getattr(G, test).pytestmark if m.name == "parametrize" and m.args[0] == name]
    return marks[0].args[1]


@pytest.mark.parametrize("test,kernel,flags", [
    ("test_gemm_pair_tiles_and_epilogues", "pair", (0, BIAS | RESIDUAL, BIAS | GELU | PREACT, DGELU)),
    ("test_gemm_cluster_split_k", "split", (0, BIAS | GELU | RESIDUAL | PREACT, DGELU)),
    ("test_gemm_cluster_split_widths", "split", (0, BIAS | RESIDUAL)),
    ("test_gemm_narrow_outputs", "one", (0, BIAS | RESIDUAL))])
def test_gpu_tests_reach_the_kernel_that_they_name(test, kernel, flags):
    """The GEMM tests choose their kernel by size: every product of theirs is on the kernel that it is there for."""
    seen = set()
    for shape in _params(test, "shape"):
        for majors in _params(test, "majors"):
            for f in flags:
                r = _route(*shape, majors=majors, flags=f)
                assert r[0] == kernel, (shape, majors, f, r)
                seen.add(r[1:])
    if test == "test_gemm_cluster_split_widths":
        assert seen >= {(128, 4), (64, 2), (64, 8)}


def test_wide_row_gemm_test_reaches_all_three_kernels():
    shapes = _params("test_gemm_rows_wider_than_the_matrix", "shape")
    for majors in _params("test_gemm_rows_wider_than_the_matrix", "majors"):
        for f in (BIAS | RESIDUAL, BIAS | GELU | PREACT, DGELU):
            assert [_route(*s, majors=majors, flags=f)[0] for s in shapes] == ["pair", "split", "one"]


@pytest.mark.parametrize("B,S,H,D,causal,ctas", [
    (1, 384, 24, 64, 0, 1), (1, 1024, 18, 128, 1, 1),                              # at most a tile per SM
    (1, 2048, 10, 128, 1, 1), (1, 4096, 9, 128, 1, 1), (1, 2048, 10, 64, 1, 1),    # the longest tile decides
    (1, 4096, 12, 128, 0, 1), (1, 3000, 25, 128, 0, 1),                            # a last round that leaves CTAs alone
    (1, 2048, 15, 64, 1, 2), (1, 700, 48, 128, 1, 2), (1, 256, 100, 128, 0, 2), (1, 4096, 18, 128, 0, 2),
    (8, 1024, 16, 64, 1, 2), (3, 1531, 12, 64, 0, 2), (2, 4096, 16, 128, 1, 2), (1, 2048, 32, 128, 1, 2),
    (16, 4096, 32, 128, 0, 2), (64, 128, 64, 64, 1, 2)])
def test_attention_forward_takes_the_faster_kernel(B, S, H, D, causal, ctas):
    """Launches timed on both forward kernels (one and two CTAs per SM), on both sides of where the choice changes."""
    from torsh_b200 import _native as nv
    assert nv.cuda().tb_flash_attn_fwd_ctas(B, S, H, D, causal) == ctas


def test_attention_gpu_tests_reach_both_forward_kernels():
    from torsh_b200 import _native as nv
    ctas = nv.cuda().tb_flash_attn_fwd_ctas
    many = {ctas(5, S, 32, D, c) for S in _params("test_flash_attention_many_tiles", "S") for D in (64, 128) for c in (0, 1)}
    assert many == {2}
    packed = [(B * H * -(-S // 128), ctas(B, S, H, D, c)) for B, S, H, D in _params("test_flash_attention_packed_many_tiles", "B,S,H,D")
              for c in (0, 1)]
    assert all(tiles > 148 for tiles, _ in packed) and {k for _, k in packed} == {1, 2}
