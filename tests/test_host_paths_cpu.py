"""The library's host code without a GPU: its decisions and its error paths, run in child processes on the CUDA runtime of
fake_cuda.cpp, whose kernels do nothing, which logs every launch and wait and fails the call a test names."""
import json
import os
import re
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = """
import ctypes as C, json, sys
sys.path.insert(0, %r)
import numpy as np
from common import load_pkg
pkg = load_pkg()
fake = C.CDLL(None)
fake.fake_log.restype = C.c_char_p
for f in (fake.fake_device_bytes, fake.fake_pinned_bytes): f.restype = C.c_longlong
for f in (fake.fake_mallocs, fake.fake_host_allocs): f.restype = C.c_long
fake.fake_fail_malloc.argtypes = [C.c_long]
fake.fake_fail_kernel.argtypes = [C.c_char_p, C.c_long]
def log(): return fake.fake_log().decode().splitlines()
def launches(part): return sum(l.startswith("launch") and part in l for l in log())
def context(wave=2, **kw):
    ctx = pkg.Context(pkg.default_config(**kw), 0, wave)
    ctx.upload_model(np.zeros(pkg.model_bytes(ctx.cfg), np.int8))
    ctx.set_dataset(np.zeros(5000, np.uint8 if ctx.cfg.vocab_size == 256 else np.uint32))
    return ctx
def error(call):
    try: call()
    except pkg.EggError as e: return e.code
    return 0
def unjoined(main):
    # streams on which something was launched that `main` does not wait for afterwards
    lines, left = [l.split() for l in log()], []
    for st in {l[2] for l in lines if l[0] == "launch"} - {main}:
        last = max(i for i, l in enumerate(lines) if l[0] == "launch" and l[2] == st)
        marks = [(i, l[1]) for i, l in enumerate(lines) if l[0] == "record" and l[2] == st and i > last]
        if not any(l[0] == "wait" and l[1] == main and l[2] == ev and i > at for at, ev in marks for i, l in enumerate(lines)): left.append(st)
    return left
out = {}
""" % HERE


@pytest.fixture(scope="session")
def fake_cuda(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cuda.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "fake_cuda.cpp")], check=True)

    def run(code):
        r = subprocess.run([sys.executable, "-c", PRELUDE + code + "\nprint(json.dumps(out))"], capture_output=True, text=True, timeout=300,
                           env=dict(os.environ, LD_PRELOAD=so, EGG_NCCL_LIB=so))
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
        return json.loads(r.stdout.splitlines()[-1])
    return run


@pytest.mark.parametrize("kw,fused", [
    (dict(hidden_dim=512, seq_len=256), True),
    (dict(hidden_dim=896, seq_len=192, shift_out=11, fixed_point=6, sigma_shift=4), False),      # 21
    (dict(hidden_dim=384, seq_len=48, shift_mlp_down=14), False),
    (dict(hidden_dim=384, seq_len=48, shift_mlp_down=13), True),                                 # 20: the largest sum
])
def test_shifts_beyond_the_row_owning_form(fake_cuda, kw, fused):
    """Shifts that the row-owning projections cannot take go to the two-kernel form, unpadded, instead of being refused."""
    out = fake_cuda("""
ctx = context(n_layers=1, population_size=8, **%r)
ctx.eval_chunk(1, 0, 0, 8)
out["fused"], out["active"] = launches("gemm_fused_kernel"), ctx.fused_epilogues_active()
""" % kw)
    assert (out["fused"] > 0) == fused and (out["active"] > 0) == fused


@pytest.mark.parametrize("shift,prefill", [(13, True), (14, False)])
def test_sampling_takes_any_shift(fake_cuda, shift, prefill):
    """Given bytes are decoded one by one where the evaluation's kernels do not take the model's shifts."""
    out = fake_cuda("""
ctx = context(hidden_dim=128, n_layers=1, seq_len=64, population_size=8, shift_mlp_up=%d)
out["rc"] = error(lambda: ctx.generate(np.zeros(20, np.uint8), 4, 1))
out["prefill"], out["decode"] = launches("kv_gather"), launches("generate_kernel")
""" % shift)
    assert out == {"rc": 0, "prefill": int(prefill), "decode": 1}


@pytest.mark.parametrize("muon", [0, 1])
def test_update_survives_a_failed_change_of_sharding(fake_cuda, muon):
    """Out of memory while the update's buffers are replaced: the change is refused and the context goes on with the ones it has."""
    out = fake_cuda("""
ctx = context(hidden_dim=128, n_layers=2, seq_len=32, population_size=64, use_muon=%d)
ctx.comm_init(bytes(128), 0, 2)
out["steps"] = []
for target, fails in ((1, 1), (1, 0), (0, 1), (0, 0), (1, 1)):
    fake.fake_fail_malloc(0 if fails else -1)
    before = fake.fake_device_bytes()
    rc = error(lambda: ctx.set_update_sharding(target))
    same = fake.fake_device_bytes() == before
    fake.fake_clear()
    out["steps"].append([rc, same, error(lambda: ctx.apply_update(1, 0.1)), launches("upd_votes_kernel")])
""" % muon)
    nomem = out["steps"][0][0]
    assert nomem < 0
    assert [s[0] for s in out["steps"]] == [nomem, 0, nomem, 0, nomem]
    assert [s[1] for s in out["steps"]] == [True, False, True, False, True]
    assert all(s[2] == 0 and s[3] > 0 for s in out["steps"]), out


def test_update_follows_a_replaced_communicator(fake_cuda):
    """The shares of a sharded update belong to a communicator: alone again a rank steps every parameter, among more ranks fewer."""
    out = fake_cuda("""
ctx = context(hidden_dim=128, n_layers=4, seq_len=32, population_size=64)
def blocks():
    fake.fake_clear()
    ctx.apply_update(1, 0.1)
    return [l.split()[-1] for l in log() if "upd_adam_kernel" in l]
out["all"] = blocks()
ctx.comm_init(bytes(128), 0, 2)
ctx.set_update_sharding(True)
out["two"] = blocks()
ctx.comm_init(bytes(128), 0, 8)
out["eight"] = blocks()
ctx.comm_init(bytes(128), 0, 1)
out["alone"] = blocks()
""")
    n = {k: sum(int(g.split(",")[0]) for g in v) for k, v in out.items()}
    assert n["alone"] == n["all"] and n["eight"] < n["two"] < n["all"], n


@pytest.mark.parametrize("rows_per_member,offset,rpl", [(64, 0, 1), (64, 16, 1), (64, 4, 0), (64, 8, 0), (20, 0, 0), (20, 4, 0), (64, 2, None)])
@pytest.mark.parametrize("n", [256, 384, 4096])
def test_projection_into_unaligned_memory(fake_cuda, n, rows_per_member, offset, rpl):
    """The row-per-lane epilogue stores 16 bytes at a time: results elsewhere take the one that stores words, and what is not even
    word-aligned is refused on the host."""
    out = fake_cuda("""
ctx = context(hidden_dim=128, n_layers=1, seq_len=32, population_size=8)
rows, n, k, p = 2 * %d * 80, %d, 128, C.c_void_p()
fake.cudaMalloc(C.byref(p), C.c_size_t(rows * (n + k) + n * k + 64))
x, w = p.value, p.value + rows * k
fake.fake_clear()
out["rc"] = error(lambda: ctx.perturbed_projection(x, w, w + n * k + %d, rows, k, n, %d, 1, 200, 201, 7, 8, on_device=True))
out["kernels"] = [l.split()[1] for l in log() if l.startswith("launch") and "gemm_i8" in l]
""" % (rows_per_member, n, offset, rows_per_member))
    if rpl is None:
        assert out["rc"] < 0 and not out["kernels"]
    else:
        assert out["rc"] == 0 and len(out["kernels"]) == 1 and ("ELi0ELi%dE" % rpl) in out["kernels"][0], out


@pytest.mark.parametrize("optimizer", [0, 1])
@pytest.mark.parametrize("w_off,opt_off,copies", [(0, 0, 0), (4, 16, 0), (1, 0, 2), (2, 0, 2), (0, 4, None), (0, 8, None)])
def test_matrix_update_of_unaligned_weights(fake_cuda, optimizer, w_off, opt_off, copies):
    """Weights that are not word-aligned are stepped in an aligned copy; a state that is not 16-byte aligned is refused."""
    out = fake_cuda("""
ctx = context(hidden_dim=128, n_layers=1, seq_len=32, population_size=8)
p = C.c_void_p()
fake.cudaMalloc(C.byref(p), C.c_size_t(1 << 20))
w, opt, fit = p.value + %d, p.value + (1 << 16) + %d, p.value + (1 << 19)
update = lambda off: ctx.update_matrix(w + off, opt, 128, 128, 402, 403, 0, fit, 100, 1, 0.1, %d, False)
for off in (-%d, 0):                  # the first call leaves the scratch behind
    fake.fake_clear()
    out["rc"] = error(lambda: update(off))
    out.setdefault("copies", []).append(sum(l.startswith("copy") for l in log()))
out["kernels"] = launches("")
""" % (w_off, opt_off, optimizer, w_off))
    if copies is None:
        assert out["rc"] < 0 and out["kernels"] == 0
    else:
        assert out["rc"] == 0 and out["copies"][1] - out["copies"][0] == copies


@pytest.mark.parametrize("hidden,fixed,sigma,shift_out,merged", [
    (128, 4, 3, 9, True), (512, 4, 3, 9, True), (896, 4, 3, 9, True), (1024, 4, 3, 9, False),      # the default shifts
    (896, 4, 3, 12, False), (256, 5, 4, 4, False), (128, 5, 5, 4, False), (128, 5, 5, 0, False),   # 2^31 within the noise of three values of 15
])
def test_merged_shifts_cannot_overflow(fake_cuda, hidden, fixed, sigma, shift_out, merged):
    """The output projection shifts once instead of twice only where its accumulator times 2^t, the largest rank-1 term (Gaussian
    noise reaches three times the mask) and the shifted bias together fit 32 bits."""
    largest = hidden * 127 * 128 * 2 ** (fixed + sigma) + hidden * 127 * 45 * 45 + 256 * 2 ** (fixed + sigma + shift_out)
    assert (largest < 2 ** 31) == merged
    out = fake_cuda("""
ctx = context(hidden_dim=%d, n_layers=1, seq_len=128, population_size=8, fixed_point=%d, sigma_shift=%d, shift_out=%d, shift_mlp_down=0, sigma_shift_vector=8,
              device_gaussian=1)
ctx.eval_chunk(1, 0, 0, 8)
out["kernels"] = [l.split()[1] for l in log() if l.startswith("launch") and "gemm_fused" in l]
""" % (hidden, fixed, sigma, shift_out))
    # <blocks a tile, tile width, mode (1: output projection), members across tiles, merged>
    got = [k.split("gemm_fused_kernelI")[1].split("EEEv")[0] for k in out["kernels"]]
    assert any(k.endswith("Lb%d" % merged) for k in got if "ELi1E" in k), got
    assert merged or not any(k.endswith("Lb1") for k in got if "ELi1E" in k), got


@pytest.mark.parametrize("kernel,after", [(None, 0), ("gru_scan_kernel", 0), ("gru_scan_kernel", 5), ("gru_rows_kernel", 7), ("gemm_i8_kernel", 11), ("gru_loss_rows", 1)])
def test_recurrent_windows_are_joined_also_when_a_launch_fails(fake_cuda, kernel, after):
    """Whatever was enqueued on the window streams is waited for by the context's stream, on which the next call works."""
    out = fake_cuda("""
cfg = pkg.default_gru_config(hidden_dim=128, n_layers=4, population_size=32, seq_len=4096)
ctx = pkg.GruContext(cfg, 0)
ctx.upload_model(np.zeros(pkg.gru_model_bytes(cfg), np.int8))
ctx.set_dataset(np.zeros(9000, np.uint8))
kernel, after = %r, %d
if kernel: fake.fake_fail_kernel(kernel.encode(), after)
fake.fake_clear()
out["rc"] = error(lambda: ctx.generation(1, 0, 4000, True))
main = next(l.split()[2] for l in log() if "gru_noise_kernel" in l)
out["streams"], out["left"] = len({l.split()[2] for l in log() if l.startswith("launch")}), unjoined(main)
""" % (kernel, after))
    assert (out["rc"] < 0) == (kernel is not None) and out["streams"] > 1 and out["left"] == [], out


@pytest.mark.parametrize("kernel,after", [(None, 0), ("muon_split", 0), ("muon_split", 2), ("ns_gemm", 0), ("ns_gemm", 13), ("muon_apply", 0), ("muon_apply", 1)])
def test_muon_streams_are_joined_also_when_a_launch_fails(fake_cuda, kernel, after):
    out = fake_cuda("""
ctx = context(hidden_dim=128, n_layers=2, seq_len=32, population_size=64, use_muon=1)
kernel, after = %r, %d
if kernel: fake.fake_fail_kernel(kernel.encode(), after)
fake.fake_clear()
out["rc"] = error(lambda: ctx.apply_update(1, 0.1))
main = next(l.split()[2] for l in log() if "upd_table_kernel" in l)
out["streams"], out["left"] = len({l.split()[2] for l in log() if l.startswith("launch")}), unjoined(main)
""" % (kernel, after))
    assert (out["rc"] < 0) == (kernel is not None) and out["left"] == [], out
    assert out["streams"] > 1 or (kernel, after) == ("muon_split", 0)


def test_as_many_contexts_as_memory_holds(fake_cuda):
    """The pinned pool bounds what copies hold, not how many contexts there are, and returns everything with the last of them."""
    out = fake_cuda("""
cfg = pkg.default_config(hidden_dim=128, n_layers=1, seq_len=16, population_size=2)
all = [pkg.Context(cfg, 0, 2) for _ in range(600)]
for c in all: c.upload_model(np.zeros(pkg.model_bytes(cfg), np.int8))
out["pinned"] = fake.fake_pinned_bytes()
for c in all[1:]: c.close()
kept = fake.fake_pinned_bytes()
again = [pkg.Context(cfg, 0, 2) for _ in range(599)]
out["reused"] = fake.fake_pinned_bytes() == kept
for c in again + all[:1]: c.close()
out["left"] = [fake.fake_pinned_bytes(), fake.fake_device_bytes()]
""")
    assert out["pinned"] <= 600 * (128 << 10) and out["reused"] and out["left"] == [0, 0]


@pytest.mark.parametrize("call,most", [
    ("ctx.perturbed_projection(p, p, p, 2048, 256, 256, 32, 1, 200, 201, 7, 8, on_device=True)", 0),
    ("ctx.perturbed_projection(p, p, p, 32768, 4096, 4096, 32, 1, 200, 201, 7, 8, on_device=True)", 1),
    ("ctx.perturbed_projection(h(65536), h(65536), h(65536), 256, 256, 256, 32, 1, 200, 201, 7, 8)", 0),
    ("ctx.update_matrix(p, p, 256, 256, 402, 403, 0, p, 1000, 1, 0.1, 0, False)", 0),
    ("ctx.update_matrix(p, p, 256, 256, 402, 403, 0, p, 1000, 1, 0.1, 1, True)", 0),
    ("ctx.update_matrix(p + 1, p, 1024, 1024, 402, 403, 0, p, 1000, 1, 0.1, 1, True)", 1),
    ("ctx.update_reconstruct(h(4000).view(np.int32), 1000, 256, 256, 402, 403, 0, 1, h(1 << 18))", 0),
    ("ctx.generate(np.zeros(40, np.uint8), 20, 1)", 0),
])
def test_first_calls_allocate_once_at_most(fake_cuda, call, most):
    """Scratch comes from the context's own memory where the work is small, in one allocation where it is not, and then stays."""
    out = fake_cuda("""
ctx = context(hidden_dim=512, n_layers=4, seq_len=256, population_size=8, device_mask=3)
p = C.c_void_p()
fake.cudaMalloc(C.byref(p), C.c_size_t(1 << 30))
p, h = p.value, lambda n: np.zeros(n, np.int8)
n = [fake.fake_mallocs()]
for _ in range(3):
    %s
    n.append(fake.fake_mallocs())
ctx.close()
out["n"] = [b - a for a, b in zip(n, n[1:])]
""" % call)
    assert out["n"] == [most, 0, 0]


@pytest.mark.parametrize("kw,two_kernel", [(dict(seq_len=16), True), (dict(seq_len=32), False), (dict(seq_len=48, shift_out=14), True)])
def test_memory_of_the_two_kernel_form_is_asked_for_where_it_is_chosen(fake_cuda, kw, two_kernel):
    """At creation for shapes that take it, else by the call that switches to it; an evaluation allocates nothing and runs out of nothing."""
    out = fake_cuda("""
ctx = context(hidden_dim=256, n_layers=1, population_size=64, **%r)
def evaluate():
    fake.fake_fail_malloc(0)
    rc = error(lambda: (ctx.eval_chunk(1, 0, 0, 64), ctx.read_losses(0, 64)))
    fake.fake_fail_malloc(-1)
    return rc
out["first"] = evaluate()
fake.fake_fail_malloc(0)
out["refused"] = error(lambda: ctx.set_fused_epilogues(0))
fake.fake_fail_malloc(-1)
out["again"] = [evaluate(), ctx.fused_epilogues_active()]
out["switched"] = [error(lambda: ctx.set_fused_epilogues(0)), evaluate(), launches("aqn_kernel")]
""" % kw)
    assert out["first"] == 0 and out["again"][0] == 0 and out["switched"][:2] == [0, 0] and out["switched"][2] > 0, out
    assert (out["refused"] < 0) == (not two_kernel) and (out["again"][1] > 0) == (not two_kernel), out


def test_recurrent_generation_without_memory_for_windows(fake_cuda):
    """Token by token where the windows' buffers cannot be had, in windows again when they can."""
    out = fake_cuda("""
cfg = pkg.default_gru_config(hidden_dim=128, n_layers=2, population_size=32, seq_len=4096)
ctx = pkg.GruContext(cfg, 0)
ctx.upload_model(np.zeros(pkg.gru_model_bytes(cfg), np.int8))
ctx.set_dataset(np.zeros(9000, np.uint8))
def generation(tokens, fails):
    fake.fake_fail_malloc(0 if fails else -1)
    fake.fake_clear()
    rc = error(lambda: ctx.generation(1, 0, tokens, True))
    fake.fake_fail_malloc(-1)
    return [rc, launches("gru_scan_kernel") > 0, any(l.startswith("graph") for l in log())]
out["g"] = [generation(100, True), generation(100, False), generation(4096, True), generation(100, False)]
""")
    assert out["g"] == [[0, False, True], [0, True, False], [0, False, True], [0, True, False]]


def test_owner_costs_are_those_of_the_update():
    """The sharded update deals parameters by cost: a vector element takes the time of 37 to 56 matrix weights."""
    from common import load_pkg
    pkg = load_pkg()
    cfg = pkg.default_config(hidden_dim=256, n_layers=4)
    _, costs, _, weights = pkg.update_owner_plan(cfg, 8, spans=True)
    vector = weights <= 4 * 256
    assert (costs[~vector] == weights[~vector]).all() and set(costs[vector] // weights[vector]) <= set(range(37, 57))


@pytest.mark.parametrize("seqs,mode,kernel", [
    ((128, 512), 0, "attention_tm_kernel"), ((528, 1024), 0, "attention_kernel"),
    ((128, 512), 1, "attention_tc_kernel"), ((128, 512), 2, "attention_hy_kernel"),
])
def test_first_launches_of_two_threads(fake_cuda, seqs, mode, kernel):
    """Two threads whose first evaluations need different amounts of shared memory for one kernel: neither lowers the other's limit."""
    out = fake_cuda("""
import threading
fake.fake_meet(%r)
ctxs = [context(hidden_dim=128, n_layers=1, seq_len=s, population_size=2) for s in %r]
if %d:
    for c in ctxs: c.set_attention_tensor_core(%d)
rcs = [None, None]
def go(i): rcs[i] = error(lambda: ctxs[i].eval_chunk(1, 0, 0, 2))
ts = [threading.Thread(target=go, args=(i,)) for i in (0, 1)]
[t.start() for t in ts]; [t.join() for t in ts]
out["rcs"], out["launched"] = rcs, launches(%r)
""" % (kernel.encode(), seqs, mode, mode, kernel))
    assert out == {"rcs": [0, 0], "launched": 2}


def forms(names, kernel):
    """Template arguments of the launches of one kernel."""
    found = [re.search(kernel + r"I((?:L[ib]\d+E)+)E", n) for n in names]
    return [tuple(map(int, re.findall(r"\d+", f[1]))) for f in found if f]


def test_sizes_of_the_pair_tests_take_pairs(fake_cuda):
    """Of every product that test_pair_tiles_gpu.py compares with single blocks, one side is formed by pairs and the other is not."""
    from test_pair_tiles_gpu import EVALUATIONS, MATRIX_UPDATES, MODEL_UPDATES, NEWTON_SCHULZ, PROJECTIONS, RECONSTRUCTIONS, small_chunk
    out = fake_cuda("""
def names(): return [l.split()[1] for l in log() if l.startswith("launch")]
for key in ("eval", "small", "projection", "aside", "votes", "update", "model", "muon"): out[key] = []
for hidden, layers, seq, pop, other, small in %r:
    ctx = context(wave=pop, hidden_dim=hidden, n_layers=layers, seq_len=seq, population_size=pop, **other)
    for key, count in (("eval", pop), ("small", small)):
        fake.fake_clear()
        ctx.eval_chunk(1, 0, 0, count)
        out[key].append(names())
    ctx.close()
p = C.c_void_p()
fake.cudaMalloc(C.byref(p), C.c_size_t(1 << 30))
p = p.value
ctx = context(hidden_dim=128, n_layers=1, seq_len=32, population_size=8, device_mask=3)
for rows, k, n in %r:
    for key, offset in (("projection", 64), ("aside", 68)):
        fake.fake_clear()
        ctx.perturbed_projection(p, p, p + offset, rows, k, n, 32, 7, 200, 201, 7, 8, on_device=True)
        out[key].append(names())
for rows, cols, pairs, _ in %r:
    fake.fake_clear()
    ctx.update_reconstruct(p, pairs, rows, cols, 402, 403, 1000, 2, p, on_device=True)
    out["votes"].append(names())
for rows, cols, pairs, split in %r:
    fake.fake_clear()
    ctx.update_matrix(p, p, rows, cols, 402, 403, 1000, p, pairs, 2, 2.5, 0, split)
    out["update"].append(names())
for rows, cols, _ in %r:
    fake.fake_clear()
    ctx.update_matrix(p, p, rows, cols, 402, 403, 0, p, 32, 7, 1.0, 1, False)
    out["muon"].append(names())
for hidden, layers, pairs, _ in %r:
    ctx = context(hidden_dim=hidden, n_layers=layers, seq_len=16, population_size=2 * pairs, device_mask=15)
    fake.fake_clear()
    ctx.apply_update(1, 0.4)
    out["model"].append(names())
    ctx.close()
""" % ([e + (small_chunk(e[0], e[2]),) for e in EVALUATIONS], PROJECTIONS, RECONSTRUCTIONS, MATRIX_UPDATES, NEWTON_SCHULZ, MODEL_UPDATES))

    def fused(names, mode):                      # blocks a tile, width of the sub-tiles, last argument
        return {(f[0], f[1], f[4]) for f in forms(names, "gemm_fused_kernel") if f[2] == mode}

    def gemm(names, epi):
        return {f[3] for f in forms(names, "gemm_i8_kernel") if f[1] == epi}

    QKV, RES, RES_LN, CLIP8, GELU, VOTE = 0, 1, 2, 0, 1, 7
    for (hidden, layers, seq, pop, other), names, small in zip(EVALUATIONS, out["eval"], out["small"]):
        one_member = seq % 128 == 0
        width = 256 if hidden in (256, 512, 1024) and one_member else 128
        wide = 2 if hidden <= 512 and one_member else 1
        assert fused(names, QKV) == {(wide, width, 0)}
        assert fused(names, RES) == {(wide if hidden == 512 else 1, width, 0 if other or hidden == 1024 else 1)}
        if hidden > 256:
            assert fused(names, RES_LN) == {(2, width, 0), (2, width, 1)}
            assert gemm(names, GELU) == {2}
        for mode in (QKV, RES, RES_LN):
            assert {f[0] for f in fused(small, mode)} == {1}
        assert gemm(small, GELU) == {1}
    assert [gemm(n, CLIP8) for n in out["projection"]] == [{2}] * 2 and [gemm(n, CLIP8) for n in out["aside"]] == [{1}] * 2
    assert [gemm(n, VOTE) for n in out["votes"]] == [{2 if r[3] else 1} for r in RECONSTRUCTIONS]
    assert [gemm(n, VOTE) for n in out["update"]] == [{2}] * len(MATRIX_UPDATES)
    assert [{f[1] for f in forms(n, "ns_gemm_kernel")} for n in out["muon"]] == [{2 if r[2] else 1} for r in NEWTON_SCHULZ]
    assert [set(forms(n, "upd_votes_kernel")) for n in out["model"]] == [{(2 if u[3] else 1,)} for u in MODEL_UPDATES]


@pytest.mark.parametrize("call,kernel,blocks", [
    # votes of one matrix: the contraction of one item
    ("ctx.update_matrix(p, p, 2048, 2048, 402, 403, 0, p, 1024, 1, 0.1, 0, False)", "gemm_i8_kernel", 1),          # 384
    ("ctx.update_matrix(p, p, 512, 512, 402, 403, 0, p, 16384, 1, 0.1, 0, False)", "gemm_i8_kernel", 1),           # 512
    ("ctx.update_matrix(p, p, 2048, 2048, 402, 403, 0, p, 2000, 1, 0.1, 0, False)", "gemm_i8_kernel", 2),          # 683
    ("ctx.update_reconstruct(p, 512, 2048, 3072, 402, 403, 0, 1, p, on_device=True)", "gemm_i8_kernel", 1),
    ("ctx.update_reconstruct(p, 513, 2048, 3072, 402, 403, 0, 1, p, on_device=True)", "gemm_i8_kernel", 2),
    # projections: rows and contraction
    ("ctx.perturbed_projection(p, p, p, 296 * 128, 384, 2048, 64, 7, 200, 201, 7, 8, on_device=True)", "gemm_i8_kernel", 1),
    ("ctx.perturbed_projection(p, p, p, 148 * 128, 512, 2048, 64, 7, 200, 201, 7, 8, on_device=True)", "gemm_i8_kernel", 1),
    ("ctx.perturbed_projection(p, p, p, 222 * 128, 512, 2048, 64, 7, 200, 201, 7, 8, on_device=True)", "gemm_i8_kernel", 2),
    ("ctx.perturbed_projection(p, p, p, 198 * 128, 768, 768, 64, 7, 200, 201, 7, 8, on_device=True)", "gemm_i8_kernel", 1),
    ("ctx.perturbed_projection(p, p, p, 148 * 128, 1024, 1024, 64, 7, 200, 201, 7, 8, on_device=True)", "gemm_i8_kernel", 2),
    # votes of a model
    ("context(hidden_dim=256, n_layers=2, seq_len=32, population_size=64).apply_update(1, 0.1)", "upd_votes_kernel", 1),
    ("context(hidden_dim=896, n_layers=1, seq_len=32, population_size=738).apply_update(1, 0.1)", "upd_votes_kernel", 1),
    ("context(hidden_dim=896, n_layers=1, seq_len=32, population_size=740).apply_update(1, 0.1)", "upd_votes_kernel", 2),
])
def test_pairs_of_blocks_where_they_gain(fake_cuda, call, kernel, blocks):
    out = fake_cuda("""
ctx = context(hidden_dim=128, n_layers=1, seq_len=32, population_size=8, device_mask=3)
p = C.c_void_p()
fake.cudaMalloc(C.byref(p), C.c_size_t(1 << 30))
p = p.value
fake.fake_clear()
%s
out["names"] = [l.split()[1] for l in log() if l.startswith("launch")]
""" % call)
    at = {"gemm_i8_kernel": 3, "upd_votes_kernel": 0}[kernel]
    assert {f[at] for f in forms(out["names"], kernel)} == {blocks}
