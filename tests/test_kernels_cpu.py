"""What the kernel library's host side decides, and rules its sources keep: no GPU needed."""
import os
import re
import subprocess
import sys

import pytest

from mojo_linuxperiments_b200 import _build
from mojo_linuxperiments_b200.ops import _lib


@pytest.fixture(scope="module")
def lib():
    if not _lib._lib_path().exists():
        pytest.skip("kernel library not built")
    return _lib.lib()


@pytest.mark.parametrize("long_form", [0, 1])
@pytest.mark.parametrize("group", [1, 2, 4, 8, 16])
def test_decode_attention_asks_for_all_the_shared_memory_it_addresses(lib, group, long_form):
    """The parts of a CTA, one by one: ring, weights, queries, exchange, barriers, three words, page ids, rows of the heads, value and
    scores of the new token, largest values of the warps and of the cluster's CTAs, merge zone."""
    if group == 16 and long_form:
        assert lib.b200_attn_decode_tc_smem(group, long_form) < 0
        return
    nb = 9 if long_form else 4
    parts = 2 * 32768 + nb * 4096 + 4096 + 128 * 4 + (7 + 2 * nb) * 8
    parts = (parts + 3 * 4 + nb * 8 * 4 + 15) // 16 * 16
    parts += (group * 128 + 128 + 16 + 8 + 8 * 4) * 4 + (0 if long_form else 32 * 130 * 4)
    got = lib.b200_attn_decode_tc_smem(group, long_form)
    assert got >= parts + 1023                          # the start is moved to a multiple of 1,024
    assert 2 * (got + 1024) <= 228 * 1024               # two CTAs per SM


def test_cluster_barriers_are_reached_by_whole_warps():
    """``barrier.cluster`` with ``.aligned`` is defined for converged warps only: every one of them stands behind a ``__syncwarp``."""
    found = 0
    for path in sorted((_build.CSRC / "kernels").glob("*.cu*")):
        lines = path.read_text().splitlines()
        for i, line in enumerate(lines):
            if "barrier.cluster." in line and ".aligned" in line and "asm" in line:
                found += 1
                assert "__syncwarp();" in lines[i - 1], f"{path.name}:{i + 1}"
    assert found >= 3


# tensors that never change while a model runs: scales of weights, norm gains and shifts, gate biases, routing corrections, tables of
# embeddings, vectors of a step
SETTLED = {"gamma", "q_gain", "c_gain", "zb", "xb", "correction", "table", "add", "shift", "swp", "swg", "sw", "norm_w", "norm_b"}


def _arguments(text: str, call: str):
    for m in re.finditer(re.escape(call), text):
        depth, at = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        yield text.count("\n", 0, m.start()) + 1, text[m.end():at - 1]


def test_only_settled_tensors_are_read_through_the_non_coherent_path():
    """A kernel may be resident before its input is written, so a line that an older kernel left in L1 may be stale: activations are
    read with plain loads or past L1."""
    found = 0
    for path in sorted((_build.CSRC / "kernels").glob("*.cu*")):
        text = re.sub(r"//.*", "", path.read_text())
        for line, arg in _arguments(text, "__ldg("):
            found += 1
            assert SETTLED & set(re.findall(r"\w+", arg)), f"{path.name}:{line}: {arg}"
        assert "ld.global.nc" not in text and "__restrict" not in text, path.name      # a restricted parameter lets the compiler choose that path
    assert found >= 20


def test_the_kernels_that_open_a_step_wait_for_all_of_the_step_before():
    """Kernels of a step read lengths, positions and page tables before their dependency wait; what orders them behind the writers is
    that the first kernel (embedding rows, in each of its three forms) does not start early."""
    for name, kernel, starts in (("rope_kv.cu", "embed_gather_kernel", ("launch_first(",)), ("rotary_paged.cu", "embed_norm_kernel", ("launch_first(",)),
                                 ("stream_rows.cu", "launch_with(", ("launch_with(p.r.ids == nullptr,",))):
        text = (_build.CSRC / "kernels" / name).read_text()
        lines = [ln for ln in text.splitlines() if kernel in ln and "launch" in ln]
        assert lines and all(any(s in ln for s in starts) for ln in lines), name


@pytest.mark.parametrize("sms", [1, 3])
@pytest.mark.parametrize("name", ["w8a8_gemm", "bf16_gemm"])
def test_a_linear_told_of_a_single_multiprocessor_returns(lib, name, sms):
    """The linears of two CTAs per tile share tiles out to half the multiprocessors: one is a pair's worth, not none (which was a
    division by zero).  Without a driver the call ends at its first tensor map; in a process of its own, since it ended there."""
    code = f"""
import ctypes
from mojo_linuxperiments_b200.ops import _lib
a, L = 1 << 20, _lib.lib()
e = _lib.DenseEpilogue(mode=0, y=a, ldy=512)
rc = (L.b200_w8a8_gemm(a, a, a, a, a, None, 300, 512, 512, 512, 0, None, 0, None, 0, a, {sms}, -1, None) if "{name}" == "w8a8_gemm" else
      L.b200_bf16_gemm(a, 512, a, 512, 300, 512, 512, ctypes.byref(e), a, {sms}, 0, None))
print("rc", rc)
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=_build.PKG.parent, env={**os.environ, "CUDA_VISIBLE_DEVICES": ""})
    assert r.returncode == 0 and "rc -" in r.stdout, (r.returncode, r.stdout, r.stderr[-500:])


def test_prefill_split_only_where_a_few_heads_walk_far():
    """Measured on both sides of the line, with 148 multiprocessors."""
    from mojo_linuxperiments_b200.ops.attention import pick_prefill_kv_chunk as pick
    assert all(pick(*c) > 0 for c in ((1, 2, 700), (1, 2, 1024), (1, 2, 3000), (1, 4, 700), (1, 4, 1024), (2, 2, 1024)))
    assert all(pick(*c) == 0 for c in ((1, 2, 256), (1, 2, 512), (1, 4, 256), (1, 4, 512), (1, 4, 2048), (1, 4, 3000), (2, 4, 1024), (1, 8, 700), (1, 8, 2048), (1, 16, 512), (1, 32, 129), (1, 32, 512),
                                       (1, 32, 4096), (32, 32, 1024), (1, 1, 64)))
    assert pick(1, 2, 3000) == 4 and pick(1, 4, 1024) == 1
    # 144 KV tiles in all: one round of 148 or 144 multiprocessors, more than one of 140
    assert pick(1, 4, 1024, 144) == 1 and pick(1, 4, 1024, 140) == 0 and pick(2, 2, 1024, 144) == 1 and pick(2, 2, 1024, 132) == 0


def test_every_kernel_that_reports_a_status_has_a_name():
    import torch

    from mojo_linuxperiments_b200.ops.workspace import Workspace, _KERNEL_NAMES
    w = Workspace(torch.device("cpu"), ws_bytes=64, counters=16)
    numbers = set()
    for path in sorted((_build.CSRC / "kernels").glob("*.cu*")):
        text = re.sub(r"//.*", "", path.read_text())
        numbers |= {int(n) for n in re.findall(r"\((?:\w+(?:<\w+>)?\(?\w*\)? \| \()?(\d+) << 8\)", text)} | {int(n) for n in re.findall(r"\| \((\d+) << 8\)", text)}
        numbers |= {int(n) for n in re.findall(r"loop\.open\(\w+, [\w.]+, (\d+),", text)}
    assert {1, 2, 3, 20, 21, 22, 23} <= numbers and numbers <= set(_KERNEL_NAMES), numbers - set(_KERNEL_NAMES)
    for n in numbers:
        w.status[0] = 1 | n << 8
        with pytest.raises(RuntimeError, match=_KERNEL_NAMES[n]):
            w.check_status()
        assert int(w.status[0]) == 0


def test_token_scales_are_stored_before_the_sums_count_as_complete():
    """Split along K, the int8 decode linear's reduction runs on all six warps, its token scales are stored by the first of the epilogue's: the
    barrier that counts the partial sums counts the warps that store scales, and each arrives behind its stores."""
    text = (_build.CSRC / "kernels" / "w8a8_gemm_decode.cu").read_text()
    assert "mbar_init(xch_bar, 1 + SX_WARPS);" in text
    stores = [m.start() for m in re.finditer(r"sx_s\[\w+\] = ", text)]
    arrives = [m.start() for m in re.finditer(r"mbar_arrive\(xch_bar\)", text)]
    assert len(stores) == 3 and len(arrives) == 1 and max(stores) < arrives[0] < text.index("mbar_wait(xch_bar")


def test_the_experts_kernel_leaves_its_loop_with_all_epilogue_warps_or_none():
    """They meet at barriers: a warp whose bounded wait ran out takes the others along through the barrier that joins the verdicts, not through a
    flag that one thread may have read before."""
    text = (_build.CSRC / "kernels" / "w8a8_gemm_experts.cu").read_text()
    loop = text[text.index("tmem_ld_x16") - 1500:text.index("tmem_ld_x16")]
    assert "if (named_bar_or(1, 128, !ok)) break;" in loop and "verdict =" not in text


def test_f32_tensor_core_linear_takes_no_more_columns_than_its_grid_has(lib):
    assert lib.b200_f32_gemm_tc_takes(16, 65535 * 128, 2048) == 1 and lib.b200_f32_gemm_tc_takes(16, 65535 * 128 + 1, 2048) == 0


def test_decode_linears_of_up_to_64_tokens_fill_the_shared_memory_they_have(lib):
    """A grid of no more than a CTA per multiprocessor has the deep ring; a fuller one two CTAs with three stages.  Measured on both sides; clusters of
    1 .. 8 CTAs that 148 multiprocessors hold with one CTA each."""
    import ctypes
    one = (ctypes.c_int * 9)(0, 148, 74, 45, 33, 26, 22, 15, 15)

    def ring(n, k, tokens, splits, fixed=0):
        r = lib.b200_w8a8_gemm_decode_ring((n + 127) // 128, k // 128, tokens, splits, fixed, one)
        return r >> 1, r & 1
    assert ring(512, 14336, 33, 8) == (8, 1) and ring(1536, 2048, 64, 8) == (8, 1) and ring(18944, 4096, 40, 1) == (1, 1)
    assert ring(1024, 2048, 33, 8) == (8, 0) and ring(1920, 8192, 64, 8) == (8, 0) and ring(2048, 4096, 64, 8) == (8, 0)
    assert ring(18944, 1024, 64, 1) == (1, 0) and ring(28672, 4096, 64, 1) == (1, 0) and ring(8192, 4096, 64, 4) == (4, 0)
    assert ring(16384, 4096, 33, 2) == (1, 1) and ring(16384, 8192, 33, 2) == (2, 0) and ring(16384, 8192, 64, 2) == (1, 1)
    assert ring(10240, 1024, 33, 3) == (1, 1) and ring(10240, 2048, 33, 3) == (3, 0) and ring(10240, 4096, 64, 3) == (3, 0)
    assert ring(16384, 4096, 64, 2, fixed=1) == (2, 0)

    def bf(n, k, tokens, splits):
        return lib.b200_bf16_gemm_decode_ring((n + 127) // 128, k // 64, tokens, splits, 148)
    assert bf(512, 14336, 33, 8) == 1 and bf(1536, 1024, 64, 8) == 1 and bf(4096, 4096, 33, 4) == 1
    assert bf(4096, 1024, 33, 4) == 0 and bf(2048, 4096, 64, 8) == 0 and bf(6144, 4096, 64, 4) == 0 and bf(512, 4096, 64, 9) == 0
