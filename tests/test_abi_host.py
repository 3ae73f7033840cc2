"""CPU-only checks of the C-ABI library: it loads, exports every symbol the header declares, and its
host-side logic (file reader, planner, helpers) agrees with the oracle. No kernel runs here."""

import ctypes as C
import pathlib
import re

import numpy as np
import pytest

import oracle as O
from oracle import brasa_format as BF

ROOT = pathlib.Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def B():
    import brasa_b200
    from brasa_b200 import build
    build.build()
    return brasa_b200


def test_library_exports_every_declared_symbol(B):
    header = (ROOT / "include" / "brasa_cuda.h").read_text()
    declared = sorted(set(re.findall(r"\b(brasa_[a-z0-9_]+)\s*\(", header)))
    assert len(declared) > 60
    L = B.lib()
    missing = [n for n in declared if not hasattr(L, n)]
    assert not missing, missing


def test_helpers_match_reference_formulas(B):
    assert B.decode_partials_len(32, 1) == 32 * 130
    assert B.decode_partials_len(32, 129) == 32 * 2 * 130
    assert B.norm_partials(2560) == 10 and B.norm_partials(2561) == 11
    assert [B.gqa_supported(h, 8) for h in (8, 16, 32, 64, 24, 40)] == [True, True, True, True, False, False]
    assert not B.gqa_supported(8, 0)
    assert B.qtype_nbytes(B.WeightType.Q4_0, 64) == 36
    assert B.qtype_nbytes(B.WeightType.Q6_0, 64) == 52
    assert B.qtype_nbytes(B.WeightType.Q8_0, 64) == 68
    assert B.KvType.F16.bytes(256) == 512 and B.KvType.Q8_0.bytes(256) == 272 and B.KvType.F32.bytes(32) == 128
    assert B.KvType.parse("q8") == B.KvType.Q8_0 and B.KvType.parse("nope") is None
    assert (B.DECODE_CHUNK, B.KV_ALIGN, B.NORM_PREP_TG) == (128, 64, 256)


def test_rope_table_is_the_oracles(B):
    cos, sin = B.rope_table(1e6, 128, 300)
    oc, os_ = O.rope_table(1e6, 128, 300)
    assert np.array_equal(cos, oc) and np.array_equal(sin, os_)


def test_file_reader_accepts_the_reference_file_and_detects_damage(B, golden_dir, tmp_path):
    path = golden_dir / "tiny" / "model.brasa"
    B.file_check(path, verify=True)
    shape, cfg = B.model_shape(path)
    assert (cfg["layers"], cfg["hidden"], cfg["heads"], cfg["kv_heads"], cfg["head_dim"], cfg["ffn"], cfg["vocab"]) == (2, 256, 4, 2, 128, 512, 512)
    assert cfg["tied"] == 1 and abs(cfg["eps"] - 1e-6) < 1e-12 and cfg["rope_theta"] == 1e6
    f = BF.BrasaFile(path)
    assert shape.weight_bytes == sum(B.planner.buffer_bytes(t["nbytes"]) for t in f.meta["tensors"])
    raw = bytearray(path.read_bytes())
    # a flipped data byte passes the structure check and fails verification
    bad = bytearray(raw)
    bad[f.tensors["model.norm.weight"]["offset"] + 5] ^= 0x40
    (tmp_path / "flip.brasa").write_bytes(bad)
    B.file_check(tmp_path / "flip.brasa", verify=False)
    with pytest.raises(B.BrasaError) as e:
        B.file_check(tmp_path / "flip.brasa", verify=True)
    assert e.value.code == B.EIO and "sha256" in str(e.value)
    # truncation, bad magic, bad version
    (tmp_path / "short.brasa").write_bytes(raw[: len(raw) // 2])
    (tmp_path / "magic.brasa").write_bytes(b"XXXX" + raw[4:])
    (tmp_path / "version.brasa").write_bytes(raw[:4] + (2).to_bytes(4, "little") + raw[8:])
    (tmp_path / "tiny.brasa").write_bytes(raw[:10])
    for name in ("short", "magic", "version", "tiny"):
        with pytest.raises(B.BrasaError) as e:
            B.file_check(tmp_path / f"{name}.brasa", verify=False)
        assert e.value.code == B.EIO
    with pytest.raises(B.BrasaError):
        B.file_check(tmp_path / "does-not-exist.brasa")


def test_hand_built_file_alignment_rules(B, tmp_path):
    cfg = BF.tiny_config(layers=1)
    w = BF.synth_weights(cfg, seed=3)
    meta = BF.write_brasa(tmp_path / "m.brasa", cfg, w)
    B.file_check(tmp_path / "m.brasa", verify=True)
    assert all(t["offset"] % 16384 == 0 for t in meta["tensors"])
    # an offset that is not page aligned is rejected by the structure check (same header length)
    raw = (tmp_path / "m.brasa").read_bytes()
    off = meta["tensors"][0]["offset"]
    old, new = f'"offset":{off}'.encode(), f'"offset":{off + 1}'.encode()
    assert len(old) == len(new) and raw.count(old) >= 1
    (tmp_path / "unaligned.brasa").write_bytes(raw.replace(old, new, 1))
    with pytest.raises(B.BrasaError) as e:
        B.file_check(tmp_path / "unaligned.brasa", verify=False)
    assert "aligned" in str(e.value)


def test_planner_arithmetic(B, golden_dir):
    shape, cfg = B.model_shape(golden_dir / "tiny" / "model.brasa")
    lim = B.Limits(ctx=300, max_tokens=64, max_logit_rows=2, kv=B.KvType.F16)
    p = B.planner.plan(shape, lim)
    bb = B.planner.buffer_bytes
    cap = 320  # ctx rounded up to KV_ALIGN
    assert p["kv"] == 2 * bb(2 * (2 * cap * 2 * 128))
    f = lambda n: bb(4 * n)
    t, h, qd, kvd, ffn = 64, 256, 512, 256, 512
    want_ws = (3 * f(t * h) + 2 * f(t * qd) + 2 * f(t * kvd) + 2 * f(t * ffn) + bb(2 * t * 512) + f(t) + f(1)
               + f(4 * 3 * 130) + f(2 * 512) + 2 * f(300 * 64))
    assert p["workspace"] == want_ws
    assert p["weights"] == shape.weight_bytes and p["overhead"] == 256 << 20
    assert p["total"] == p["weights"] + p["kv"] + p["workspace"] + p["overhead"]
    q8 = B.planner.plan(shape, B.Limits(ctx=300, max_tokens=64, max_logit_rows=2, kv=B.KvType.Q8_0))
    assert q8["kv"] == 2 * bb((2 * cap * 2 * 128) // 128 * 136)
    # budget check without a device: explicit budget
    ok, plan, mx = B.planner.check(None, shape, lim, budget=p["total"])
    assert ok and mx == 300
    ok, plan, mx = B.planner.check(None, shape, lim, budget=p["total"] - 1)
    assert not ok and 0 < mx < 300
    smaller = B.planner.plan(shape, B.Limits(ctx=mx, max_tokens=min(64, mx), max_logit_rows=2, kv=B.KvType.F16))
    assert smaller["total"] <= p["total"] - 1
    ok, _, mx0 = B.planner.check(None, shape, lim, budget=1000)
    assert not ok and mx0 == 0


def test_no_cpu_fallback_without_a_device(B):
    import torch
    if torch.cuda.is_available():
        pytest.skip("a CUDA device is present")
    with pytest.raises(B.BrasaError) as e:
        B.Context(0)
    assert e.value.code == B.ECUDA


def test_batch_planner_arithmetic_and_largest_batch(B):
    """The paged pool's plan (crates/memory/src/planner.rs:57-95 retargeted): every buffer of a batch at the allocation
    granularity, and the largest batch that fits a budget (planner.rs:237-281 for sequences): one more sequence than
    the answer does not fit, the answer does."""
    shape = B._ModelShape(0, 36, 2560, 32, 8, 128, 9728, 151936)  # the Qwen3-4B architecture
    bb = B.planner.buffer_bytes
    p = B.planner.plan_batch(shape, 64, 2048 // 16 + 64 * 97, 3600, B.KvType.F16)
    row = 8 * 128 * 2
    assert p["kv_pages"] == 2 * bb(36 * (128 + 64 * 97) * 16 * row)
    assert p["tables"] == bb(64 * 225 * 4) + 3 * bb(64 * 4) + bb(64 * 16)
    assert p["logits"] == bb(64 * 151936 * 4) and p["sampler"] == bb(64 * 2 * 151936 * 4)
    assert p["attention_partials"] == bb(64 * 32 * ((225 * 16 + 127) // 128) * 130 * 4)
    assert p["total"] == sum(v for k, v in p.items() if k != "total")
    q8 = B.planner.plan_batch(shape, 64, 2048 // 16 + 64 * 97, 3600, B.KvType.Q8_0)
    assert q8["kv_pages"] == 2 * bb(36 * (128 + 64 * 97) * 16 * 8 * 136)
    # 64 sequences of 3 600 positions behind a 2 048-token shared prefix: 13.9 GiB of pages; 31.5 GiB without sharing
    assert abs(p["kv_pages"] / 2**30 - 13.92) < 0.05
    budget = 40 << 30
    n, pages, plan = B.planner.max_batch(None, shape, B.KvType.F16, 2048, 3600, budget=budget)
    assert n > 64 and plan["total"] <= budget and pages == 128 + n * 97
    more = B.planner.plan_batch(shape, n + 1, 128 + (n + 1) * 97, 3600, B.KvType.F16)
    assert more["total"] > budget
    n0, _, _ = B.planner.max_batch(None, shape, B.KvType.F16, 2048, 3600, budget=1 << 20)
    assert n0 == 0
    n_cap, _, _ = B.planner.max_batch(None, shape, B.KvType.F16, 2048, 3600, budget=budget, cap=10)
    assert n_cap == 10
    # a tensor-parallel shard (an eighth of the lm_head's rows): two more full-width logits buffers for the sampled choice
    sh = B.planner.plan_batch(shape, 16, 2048 // 16 + 16 * 97, 3600, B.KvType.F16, head_rows=151936 // 8)
    assert sh["logits"] == bb(16 * (151936 // 8) * 4)
    assert sh["sampler"] == bb(16 * 2 * 151936 * 4) + 2 * bb(16 * 151936 * 4)


def test_few_token_gemm_partition(B):
    """The cut of a few-token GEMM over the SMs (`brasa_gemm_few_tokens_plan`): the runs tile the units exactly, every
    unit's owner is the block whose run holds it, the blocks that share a tile are consecutive and never more than
    `max_parts`, and the scratch holds one 64 x 128 f32 tile per (tile, part). Shapes: the Qwen3-4B layer at 148 SMs
    (qkv, o, gate + up, down), a shard's, tiny ones, and one too large for 32-bit unit arithmetic."""
    L = B.lib()
    L.brasa_gemm_few_tokens_plan.argtypes = [C.c_uint32, C.c_uint32, C.c_uint32, C.POINTER(C.c_uint32), C.POINTER(C.c_uint32), C.POINTER(C.c_uint64)]
    L.brasa_gemm_few_tokens_plan.restype = C.c_int32
    L.brasa_gemm_few_tokens_owner.argtypes = [C.c_uint32, C.c_uint32, C.c_uint32]
    L.brasa_gemm_few_tokens_owner.restype = C.c_uint32
    for sms, tiles, stages in [(148, 48, 40), (148, 20, 64), (148, 152, 40), (148, 20, 152), (148, 1, 4), (148, 3, 4), (148, 1, 1), (132, 25, 38),
                               (148, 200, 4), (7, 5, 9)]:
        blocks, parts, scratch = C.c_uint32(), C.c_uint32(), C.c_uint64()
        assert L.brasa_gemm_few_tokens_plan(sms, tiles, stages, C.byref(blocks), C.byref(parts), C.byref(scratch)) == 0
        nb, units = blocks.value, tiles * stages
        assert 1 <= nb <= min(sms, units) and (nb == sms or nb == max(1, units // 4))
        beg = [b * units // nb for b in range(nb + 1)]
        assert beg[0] == 0 and beg[-1] == units and all(beg[b] < beg[b + 1] for b in range(nb))  # no empty run
        owner = [L.brasa_gemm_few_tokens_owner(units, nb, u) for u in range(units)]
        for u, b in enumerate(owner):
            assert beg[b] <= u < beg[b + 1], (u, b)
        worst = 0
        for t in range(tiles):
            own = owner[t * stages:(t + 1) * stages]
            assert own == sorted(own) and set(own) == set(range(own[0], own[-1] + 1))  # consecutive blocks, in K order
            worst = max(worst, own[-1] - own[0] + 1)
        assert parts.value == worst
        assert scratch.value == tiles * worst * 64 * 128 * 4
    blocks, parts, scratch = C.c_uint32(), C.c_uint32(), C.c_uint64()
    assert L.brasa_gemm_few_tokens_plan(148, 1 << 20, 1 << 6, C.byref(blocks), C.byref(parts), C.byref(scratch)) != 0
    assert L.brasa_gemm_few_tokens_plan(148, 0, 4, C.byref(blocks), C.byref(parts), C.byref(scratch)) != 0
    assert L.brasa_gemm_few_tokens_owner(100, 10, 100) == 0xFFFFFFFF


def test_token_ring_is_one_the_kernel_can_index(B):
    """The weight ring of the whole-token kernel on integer products over models up to vocabularies of 2^23: none, or at least two slots (one
    would make the kernel's reciprocal of their number 2^32, which its 32-bit word holds as 0: every slot but the first would lie behind
    the ring), never more for a larger vocabulary; and that reciprocal gives the list index of every slot exactly."""
    L = B.lib()
    L.brasa_token_ring_slots.argtypes = [C.c_uint32] * 7 + [C.c_int32] * 2
    L.brasa_token_ring_slots.restype = C.c_uint32
    SMS, SMEM, Q4, Q6 = 148, 232448, int(B.WeightType.Q4_0), int(B.WeightType.Q6_0)
    f16, q8, f32 = int(B.KvType.F16), int(B.KvType.Q8_0), int(B.KvType.F32)
    assert L.brasa_token_ring_slots(SMS, SMEM, 2560, 32, 8, 9728, 151936, Q6, f16) >= 4  # the 4B architecture
    assert L.brasa_token_ring_slots(SMS, SMEM, 2560, 32, 8, 9728, 151936, Q6, f32) == 0  # decode_token.cu's
    assert L.brasa_token_ring_slots(SMS, SMEM, 512, 8, 2, 1536, 1024, Q6, f16) == 0
    seen = set()
    for hidden, heads, ffn in [(768, 6, 1024), (1024, 16, 3072), (1024, 40, 10240), (1536, 8, 4096), (2048, 16, 6144), (2560, 32, 9728), (3072, 24, 8192), (3072, 80, 10240)]:
        for head in (Q4, Q6):
            for kv in (f16, q8):
                last = 1 << 30
                for vocab in [*range(1 << 17, (1 << 23) + 1, 1 << 17)]:
                    ring = L.brasa_token_ring_slots(SMS, SMEM, hidden, heads, heads // 2, ffn, vocab, head, kv)
                    assert ring != 1 and ring <= last, (hidden, vocab, ring)
                    last = ring
                    seen.add(ring)
    assert 0 in seen and 2 in seen and max(seen) >= 7
    for ring in seen - {0}:
        mul = ((1 << 32) + ring - 1) // ring
        assert mul < 1 << 32
        k = np.concatenate([np.arange(4096, dtype=np.uint64), np.random.default_rng(1).integers(0, 1 << 24, 4096).astype(np.uint64)])
        assert np.array_equal((k * np.uint64(mul)) >> np.uint64(32), k // np.uint64(ring)), ring


@pytest.mark.parametrize("name", ["decode_token.cu", "decode_token_mma.cu"])
def test_token_kernels_keep_the_output_scale_in_a_word_of_its_own(name):
    """Behind the rows' barrier every warp of a whole-token kernel reads the scale of the operation's outputs; a warp without rows of the lm_head
    then stores its best logit with no barrier in between. So no word of that store, whatever the warp, may be the scale's. Read from the source:
    the window is some hundred cycles."""
    words = dict(TK_WARPS=16)
    for a, b in re.findall(r"\b(RED_\w+) = ([^,;]+)", (ROOT / "brasa_b200" / "csrc" / "token_device.cuh").read_text()):
        words[a] = eval(b, {}, words)
    text = (ROOT / "brasa_b200" / "csrc" / name).read_text()
    stores = [(i, [eval(i, {}, dict(words, warp=w)) for w in range(16)] if "warp" in i else [eval(i, {}, words)])
              for i in re.findall(r"\bred(?:\(\))?\[([^\]&]+)\] = ", text)]
    best, scale = [w for i, ws in stores if "warp" in i and i != "warp" for w in ws], [ws[0] for i, ws in stores if "warp" not in i]
    assert len(best) == 64 and len(scale) == 1  # a block's best, the choice among the blocks: logit and index each
    assert scale[0] not in best and scale[0] >= 16 and max(best + scale) < words["RED_WORDS"]
    assert re.findall(r"gemv_epilogue\(c, op, bo, c\.red(?:\(\))?\[(\w+)\]", text) == ["RED_SCALE"]


def test_token_kernel_that_gave_up_waits_for_every_copy_it_asked_for():
    """A block of the whole-token kernel on integer products has two kinds of bulk copies in flight, ring slots and the next norm weight. Once a
    wait has given up, nobody waits for either any more, so neither may be asked for again (its barrier may be armed still), and the block
    waits for both before it leaves: shared memory that a copy still writes is the next block's. Read from the source, since no wait is made
    to run out on a GPU here."""
    text = re.sub(r"//[^\n]*", "", (ROOT / "brasa_b200" / "csrc" / "decode_token_mma.cu").read_text())
    asks = re.findall(r"\b(issue_slot|stage_norm)\((?!const)", text)
    assert asks.count("issue_slot") == 2 and asks.count("stage_norm") == 2  # the first ones; one refill, one norm an operation
    refill = text.index("issue_slot(c, c.sdesc()")
    assert "!*c.abort_flag()" in text[text.rindex("if (", 0, refill):refill]
    norm = text[text.index("auto stage_norm = "):]
    assert norm.index("if (*c.abort_flag()) return;") < norm.index("*c.norms_asked() = *c.norms_asked() + 1;") < norm.index("mbar_expect_tx")
    leave = text[text.index("gemv_epilogue(c, op, bo, c.red()"):text.index("if (b == 0)")]
    leave = leave[leave.index("if (*c.abort_flag()"):]
    assert "mbar_wait(c.full(tid), *c.gen(tid) & 1)" in leave and "mbar_wait(c.nw_full(), (*c.norms_asked() - 1) & 1)" in leave


def test_dp4a_token_kernel_that_gave_up_waits_for_its_ring():
    """The same of decode_token.cu, whose only bulk copies are the ring's: no refill once a wait has given up, and the last copy of every slot is
    waited for in the phase that the slot's refills have come to."""
    text = re.sub(r"//[^\n]*", "", (ROOT / "brasa_b200" / "csrc" / "decode_token.cu").read_text())
    assert len(re.findall(r"\bissue_slot\((?!const)", text)) == 2 and len(re.findall(r"\bbulk_g2s\(", text)) == text[text.index("void issue_slot("):text.index("gemv_input(")].count("bulk_g2s(")
    refill = text.index("issue_slot(c, c.sdesc[j], rs)")
    ask = text[text.rindex("atomicAdd(&c.done[rs], 1u)", 0, refill):refill]
    assert "!*c.abort_flag()" in ask and "c.done[rs] = (c.done[rs] & DONE_PARITY) ^ DONE_PARITY;" in ask
    leave = text[text.index("gemv_epilogue(c, op, bo, c.red["):text.index("if (b == 0)")]
    assert "if (*c.s_abort)" in leave and "mbar_wait(&c.full[s], c.done[s] >> 31)" in leave


@pytest.mark.parametrize("name,kernels", [("flash_tc.cu", 2), ("window_attn.cu", 1)])
def test_row_warps_of_the_attention_kernels_leave_together(name, kernels):
    """The two warps that hold the same query rows meet at counted barriers, and each may give up a wait on its own. So a meeting has to tell
    both whether they go on (tc_pair_agree), and neither may leave between a wait for scores and the meeting behind it: the other would
    stand at a barrier that never fills, and the block would never end. Read from the source, since a GPU is not made to hang for it."""
    text = re.sub(r"//[^\n]*", "", (ROOT / "brasa_b200" / "csrc" / name).read_text())
    assert not re.search(r"\bbar(rier)?\.(cta\.)?sync", text)  # every meeting of fewer than all threads carries the verdict
    score_waits = list(re.finditer(r"ok = (wait_s\(j\)|wait\(&s_ready\[x\]|wait\(&bar_s\[j & 1\])", text))
    meetings = [m.start() for m in re.finditer(r"ok = tc_pair_agree\(", text)]
    followed = [w for w in score_waits if any(w.start() < m < w.start() + 2500 for m in meetings)]
    assert len(followed) == kernels
    for w in followed:
        between = text[w.end():min(m for m in meetings if m > w.start())]
        assert not re.search(r"\b(break|return|continue)\b", between)
