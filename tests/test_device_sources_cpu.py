"""Rules of the device code that no single run can show: read from the sources."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "velox_voice_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name,kernel", [("vx_gemm_ln.cu", "bsgemm_residual_ln_kernel("), ("vx_gemm.cu", "bsgemm_kernel("),
                                         ("vx_attn.cu", "relpos_attn_kernel("), ("vx_mel.cu", "power_mel_log_dense_kernel("),
                                         ("vx_mel.cu", "power_mel_log_kernel(")])
def test_waits_before_warp_wide_tensor_memory_accesses_end_in_a_vote(name, kernel):
    """tcgen05.ld, .st and .wait are warp-wide.  A poll of an mbarrier can answer lane by lane, so the lanes of a warp can leave
    a waiting loop on different turns: before such an access they have to be brought together (a vote or __syncwarp).  Held
    for every wait by all lanes from which such an access can be reached without one."""
    text = source(name)
    text = text[text.index(kernel):]
    end = re.search(r"\n}\n", text)
    text = text[:end.end()]
    aligned = re.compile(r"\btc_(ld|st|wait)\w*\(")
    wait = re.compile(r"\bmbar_wait\w*(<\w+>)?\(")
    gather = re.compile(r"__all_sync|__syncwarp|__shfl\w*_sync|__any_sync|__syncthreads|__ballot_sync")
    role = re.compile(r"\n  } else\b")  # the next role of a warp-specialised kernel: other warps
    event = re.compile("|".join(f"(?:{r.pattern})" for r in (aligned, wait, gather, role)))
    open_wait = None
    for m in event.finditer(text):
        t = m.group(0)
        if wait.fullmatch(t):
            line = text[text.rfind("\n", 0, m.start()):m.start()]
            if "__all_sync" not in line:
                open_wait = text[m.start():m.start() + 60]
        elif gather.fullmatch(t) or role.fullmatch(t):
            open_wait = None
        else:
            assert open_wait is None, f"{name}: {t} can be reached by a part of a warp behind {open_wait!r}"


@pytest.mark.parametrize("name,kernel", [("vx_gemm_ln.cu", "bsgemm_residual_ln_kernel("), ("vx_pass.cu", "conformer_pass_kernel(")])
def test_no_lane_of_a_warp_stays_behind_when_a_limit_runs_out(name, kernel):
    """The kernels of clusters end in a barrier that every thread has to reach.  A limit that runs out for some lanes of a warp while
    the barrier completes for the others must not part them at a __syncwarp: each wait is one thread's, or a vote, or its
    outcome ends no loop (no MMA is issued for a lane that gave up, and it waits for nothing more)."""
    text = source(name)
    text = text[text.index(kernel):]
    text = text[:re.search(r"\n}\n", text).end()]
    start, end = text.index("elect_one()"), text.rindex("  } else {\n", 0, text.index("const int row_in"))
    mma = text[start:end]
    together = "__syncwarp" in mma
    if together:
        assert "break" not in mma and not re.search(r"for \([^\n]*\bok\b", mma)
        assert len(re.findall(r"if \(leader && ok\)", mma)) == mma.count("if (leader")
    for m in re.finditer(r"\bmbar_wait\w*\(", text):
        line = text[text.rfind("\n", 0, m.start()):text.index("\n", m.start())]
        role = text[text.rindex("if (warp == ", 0, m.start()):m.start()]
        alone = re.match(r"[^{]*{\s*if \((lane == 0\b[^\n]*|elect_one\(\)\)) {", role)
        assert alone or "__all_sync" in line or (together and start < m.start() < end), f"{name}: {line.strip()}"


@pytest.mark.parametrize("name,kernel", [("vx_mel.cu", "power_mel_log_kernel("), ("vx_mel.cu", "power_mel_log_dense_kernel("),
                                         ("vx_attn.cu", "relpos_attn_kernel("), ("vx_gemm.cu", "bsgemm_kernel(")])
def test_lanes_that_meet_at_a_syncwarp_agree_on_their_waits(name, kernel):
    """A lane of an MMA warp that gave up a wait leaves its loop.  Either the lanes meet nowhere in it, or whether the limit ran out is a
    vote."""
    text = source(name)
    text = text[text.index(kernel):]
    text = text[text.index("elect_one()"):]
    mma = text[:re.search(r"\n  } else {\n", text).start()]
    waits = [mma[mma.rfind("\n", 0, m.start()):m.start()] for m in re.finditer(r"\bmbar_wait\w*(<\w+>)?\(", mma)]
    assert len(waits) >= 2 and ("__syncwarp" not in mma or all("__all_sync" in w for w in waits))


@pytest.mark.parametrize("name", ["vx_gemm_ln.cu", "vx_gemm.cu"])
def test_stores_are_complete_before_a_kernel_ends(name):
    """Writes of a bulk store are ordered by waiting for its group, not by the end of the thread that issued it; the `.read`
    form says only that shared memory may be reused.  The last wait before the tear-down is the full one."""
    text = source(name)
    waits = [m.group(1) for m in re.finditer(r"tma_store_wait_(read|all)<0>\(\)", text)]
    assert text.count("tma_store_commit()") >= 1 and waits[-1] == "all"
    last = text.rindex("tma_store_wait_all<0>()")
    assert text.rindex("tma_store_commit()") < last < text.index("tmem_dealloc(tmem_base", last)


@pytest.mark.parametrize("name,kernel,storers", [("vx_gemm_ln.cu", "bsgemm_residual_ln_kernel(", 2), ("vx_gemm.cu", "bsgemm_kernel(", 1)])
def test_every_role_that_stores_waits_for_its_writes(name, kernel, storers):
    """Each role that hands blocks to the TMA ends with the full wait for them, not with that of another role."""
    text = source(name)
    text = text[text.index(kernel):]
    text = text[:re.search(r"\n}\n", text).end()]
    roles = [r for r in re.split(r"\n  } else\b[^\n]*{|\n  if \(warp == 0\) {", text) if "tma_store_commit()" in r]
    assert len(roles) == storers
    for role in roles:
        role = role[:role.find("tmem_dealloc")]
        assert role.rindex("tma_store_commit()") < role.rindex("tma_store_wait_all<0>()")


@pytest.mark.parametrize("name,kernel,waits", [("vx_gemm.cu", "bsgemm_kernel(", r"warp != 0 \|\| my_tiles == 0"),
                                               ("vx_gemm_ln.cu", "bsgemm_residual_ln_kernel(", "!producer_thread"),
                                               ("vx_pass.cu", "conformer_pass_kernel(", "warp != PS_WARP_B")])
def test_a_gemm_triggers_the_next_launch_only_behind_its_own_wait(name, kernel, waits):
    """One thread that triggers counts for its CTA.  A loader reads weights ahead of its wait, so the trigger must not be reachable for
    it, nor for any thread, without the wait in front."""
    text = source(name)
    text = text[text.index(kernel):]
    text = text[:re.search(r"\n}\n", text).end()]
    assert text.count("pdl_launch_dependents()") == 1
    assert re.search(r"if \(%s\) {\s*pdl_wait\(\);\s*pdl_launch_dependents\(\);\s*}" % waits, text)
    if name == "vx_gemm_ln.cu":
        assert "const bool producer_thread = (warp == 0 || warp == 18) && lane == 0 && my_tiles > 0;" in text


@pytest.mark.parametrize("name,barrier", [("vx_gemm.cu", "empty"), ("vx_gemm_ln.cu", "empty"), ("vx_gemm_ln.cu", "hb_empty"),
                                          ("vx_pass.cu", "b_empty")])
def test_loaders_that_run_ahead_wait_for_the_previous_launch_before_a_bounded_wait(name, barrier):
    """A ring that is full empties only when the MMAs start, behind the previous launch: the limit of a wait is for this kernel's
    own progress, so whoever loads constant weights ahead waits for that launch once before waiting for a slot to be free."""
    text = source(name)
    wait = re.search(r"mbar_wait\w*(<\w+>)?\(&sm\.%s\[" % barrier, text).start()
    role = text[text.rindex("if (warp == ", 0, wait):wait]
    waits = re.findall(r"if \(([^\n]*)\) (?:\{ )?pdl_wait\(\)", role)
    assert "p.b_const" in waits or any(w in ("ph && !waited", "!par && !waited") for w in waits), (name, waits)


def test_the_wait_for_the_other_ctas_sums_acquires_at_cluster_scope():
    """st.async of the peer completes the exchange barrier with a release at cluster scope; a wait that acquires at the default
    scope, the CTA, does not pair with it."""
    text = source("vx_gemm_ln.cu")
    assert re.findall(r"mbar_wait\w*\(&sm\.xch", text) == ["mbar_wait_spin_cluster(&sm.xch"]
    assert "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64" in source("vx_ptx.cuh")


def test_what_writes_weights_does_not_trigger_the_next_launch():
    """A GEMM may read a constant weight and its scale factors ahead of its wait, and the launches between may all have triggered
    before their own: the kernels that write them must not.  (Scale factors of a single operand are a weight's: PackedLinear, or
    a C caller before VX_GEMM_CONST_B.)"""
    text = source("vx_quant.cu")
    body = text[text.index("sf_relayout_kernel(RelayoutSide"):]
    body = body[:body.index("pdl_wait()")]
    assert re.findall(r"[^\n]*pdl_launch_dependents\(\);", body) == ["  if (early) pdl_launch_dependents();"]
    pair = text[text.index("int vx_sf_from_natural_pair("):]
    assert re.search(r"launch_dependent\(sf_relayout_kernel.*?side\[1\]\.words != 0 \? 1 : 0\)\)", pair, re.S)
    assert "vx_sf_from_natural_pair(fmt, scales, R, scales_sf, fmt, nullptr, 0, nullptr, K, stream)" in pair


@pytest.mark.parametrize("name,kernel", [("vx_quant.cu", "ln_quant_kernel(const QuantParams p) {"), ("vx_quant.cu", "rows2_kernel(const QuantParams p) {"),
                                         ("vx_gemm_ln.cu", "bsgemm_residual_ln_kernel("), ("vx_mel.cu", "power_mel_log_kernel("),
                                         ("vx_mel.cu", "power_mel_log_dense_kernel("), ("vx_rowscale.cu", "rowscale_small_kernel(const RsParams p) {")])
def test_parameters_are_read_behind_the_wait(name, kernel):
    """A library GEMM may have written a bias, a LayerNorm parameter or a filterbank, and triggers the launch behind it early: no address
    of one is formed ahead of that launch's wait."""
    text = source(name)
    text = text[text.index(kernel):]
    text = text[:re.search(r"\n}\n", text).end()]
    ahead = text[:text.index("pdl_wait()")]
    assert not re.search(r"\bp\.(bias|gamma2?|beta2?|mel)\b(?! \? 2 : 1)", ahead), (name, kernel)
