"""Rules that every kernel of booster_b200/csrc keeps and that no run shows reliably when one is broken: read from the source."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "booster_b200" / "csrc"
WAIT = re.compile(r"\b(um_wait|um_wait_asleep|mbar_wait|mbar_wait_limited)\(")
ARRIVE = re.compile(r"if \(lane == 0\).*\bmbar_arrive\(|\bmbar_arrive_if\(")      # one lane of the warp
JOINED = re.compile(r"__syncwarp\(\)|__syncthreads\(\)|tmem_ld_wait\(\)|tmem_st_wait\(\)|\.sync\b")


def _code(path):
    return [line.split("//")[0] for line in path.read_text().splitlines()]


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cuh")))
def test_a_warp_is_whole_before_one_lane_arrives_for_it(name):
    """All lanes of a warp wait for a barrier's phase, one lane arrives for the warp. Were it let on while another lane still looks for that phase, the barrier could complete the
    next one, whose parity that lane then waits out. Between the wait and the arrival the lanes have to meet."""
    code, bad = _code(CSRC / name), []
    for i, line in enumerate(code):
        if not ARRIVE.search(line) or "__device__" in line:
            continue
        for back in range(i, max(-1, i - 80), -1):
            text = code[back]
            if back == i:
                text = text[:ARRIVE.search(text).start()]
            if JOINED.search(text) or "__device__" in text or "__global__" in text:
                break
            if WAIT.search(text):
                bad.append(f"{name}:{i + 1} (waits at {back + 1})")
                break
    assert not bad, bad


def test_every_call_that_runs_products_reads_their_error_flag():
    """a product whose bounded wait runs out stores nothing and raises a flag: each entry point that runs one and synchronises looks at it before it reports success"""
    text = (CSRC / "engine.cu").read_text()
    calls, bad = re.split(r'(?m)^(?=extern "C" )', text)[1:], []
    for call in calls:
        body = "\n".join(line.split("//")[0] for line in call.splitlines())
        name = re.search(r"(b200_\w+)\(", body).group(1)
        runs = re.search(r"\b(enqueue_forward|enqueue_stage_step|cudaGraphLaunch|launch_matvec|pb_matmul)\(", body)
        if runs and "cudaStreamSynchronize(" in body and "pb_check(" not in body[body.rindex("cudaStreamSynchronize("):]:
            bad.append(name)
    assert not bad, bad


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu")))
def test_shared_memory_limits_are_kept_per_device(name):
    """a kernel's limit of dynamic shared memory holds on the device it was set on: what remembers that it was raised is an array over devices"""
    once = [line.strip() for line in _code(CSRC / name) if re.search(r"static (const )?(bool|size_t) \w+ = ", line) and ("cudaFuncSetAttribute" in line or "attr" in line)]
    assert not once, once


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cuh")))
def test_accumulators_are_read_behind_the_wait_for_them(name):
    """tcgen05.ld returns before its registers hold anything: only what depends on tcgen05.wait::ld is safe from being moved in front of it. The wait has the registers as operands, or the
    statement behind it has"""
    text = "\n".join(_code(CSRC / name))
    bad = [text[:m.start()].count("\n") + 1 for m in re.finditer(r"asm volatile\(\"tcgen05\.wait::ld[^;]*;\"([^;]*);", text)
           if '"+r"' not in m.group(1) and "void tmem_ld_wait()" not in text[text.rfind("\n", 0, m.start()):m.start()]]
    bad += [text[:m.start()].count("\n") + 1 for m in re.finditer(r"\btmem_ld_wait\(\);(\s*)(?!tmem_ld\d+_ready\()\S", text)]
    assert not bad, bad


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("stack_kernels*.cuh")))
def test_a_warp_loads_accumulators_whole(name):
    """tcgen05.ld is an instruction of the whole warp. A bounded wait may run out for some of its lanes and not for others: what decides by it whether accumulators are loaded is the same for
    all lanes, and a loop that lanes leave early in (continue) meets before the next load"""
    text = "\n".join(_code(CSRC / name))
    bad = [m.group(0) for m in re.finditer(r"const bool \w+ = [^;]*mbar_wait_limited\([^;]*;", text) if "__all_sync(" not in m.group(0)]
    for m in re.finditer(r"continue;", text):
        head = text.rfind("#pragma unroll 1", 0, m.start())
        loop = text[head:m.start()]
        if head >= 0 and "tcgen05.ld" in loop and "__syncwarp();" not in loop[:loop.index("tcgen05.ld")]:
            bad.append(text[:m.start()].count("\n") + 1)
    assert not bad, bad


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("stack_kernels*.cuh")))
def test_stack_kernels_wait_for_the_kernel_before_them(name):
    """a pass's kernels become resident while the one before still runs: each waits before it reads what another wrote, and reads that coherently (no __ldg, no read-only pointer of
    what a pass computes: the compiler may take such a load for one of a constant and move it ahead of the wait)"""
    text = "\n".join(_code(CSRC / name))
    bodies = re.split(r"__global__", text)[1:]
    weights = {"embed", "w_post", "w_next", "cnorm", "qnorm", "W2", "w0", "coef", "sink", "dt_bias", "A_log", "w", "bias", "r1v", "r2v", "Wdt", "bdt"}
    bad = []
    for b in bodies:
        kernel = re.search(r"\b(k_\w+)\s*\(", b).group(1)
        signature = b[:b.index("{")]
        if "pdl_enter()" not in b and "pdl_wait()" not in b:
            bad.append(f"{kernel} does not wait")
        bad += [f"{kernel}: {m}" for m in re.findall(r"\*\s*__restrict__\s*(\w+)", signature) if m not in weights]
        bad += [f"{kernel}: __ldg of {m}" for m in re.findall(r"__ldg\((.*)", b) if "(w + i)" not in m]
    assert not bad, bad


# pointers that a kernel of a pass names ahead of its (last) wait. Weights: read. "st" and "tokens": the step's header, written before the pass's first launch, which is launched
# whole; so are cached rows below pos0 ("cache" of the two attention kernels) and the state of the delta rule ("S"). The others give addresses, or are used behind a wait further up
# (k_post_norm_add's `waited`, k_gemv_ring's indexed batch, k_gemm_bf16_pair's segments), or are another thing of that name (a tile's part).
EARLY = {
    "k_post_norm_add": {"w_post", "w_next", "Y", "X", "Hn", "H16"}, "k_gemv_ring": {"W", "w_index"}, "k_latent_prep": {"cnorm", "st", "P", "cache"}, "k_latent_attn_staged": {"st", "cache"},
    "k_causal_conv_rows": {"w", "bias"}, "k_delta_gates": {"CV"}, "k_delta_scan": {"S"}, "k_gqa_prep": {"st", "P", "cache"}, "k_gqa_attn_group": {"st", "cache", "pool"},
    "k_moe_route": {"Wr", "w_sg", "Hn", "z"}, "k_side_in": {"tokens", "table", "Wg"}, "k_side_out": {"Wp"}, "k_gemm_bf16_pair": {"seg", "part"},
}


def test_what_stack_kernels_name_ahead_of_their_wait():
    """EARLY, kernel by kernel: a pointer that joins the names ahead of a wait is looked at before it joins this table"""
    known = {"X", "W", "Y", "Yb", "bias", "seg", "w_index", "x_scale", "QK", "cache", "sink", "st", "OL", "part", "ml", "P", "A", "hist", "w", "Q", "Vv", "S", "O", "ab", "den", "Wg", "Wp", "pool", "r1", "r2",
             "Wr", "w_sg", "Hn", "z", "Ya", "Yb", "Yk", "wt", "slot_of", "nw", "H16", "keep", "coef", "XS", "counter", "table", "proj", "gate", "norm", "sel", "sg", "fw", "scratch"}
    found = {}
    for path in sorted(CSRC.glob("stack_kernels*.cuh")):
        for body in re.split(r"__global__", "\n".join(_code(path)))[1:]:
            kernel, start = re.search(r"\b(k_\w+)\s*\(", body).group(1), body.index("{")
            ends = re.search(r"\n}\n", body).end()
            early = body[start:max(m.start() for m in re.finditer(r"pdl_(enter|wait)\(\)", body[:ends]))]
            names = {p for p in re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)\s*[,)=]", body[:start]) if re.search(rf"\b{p}\b", early)}
            names |= {f for f in re.findall(r"\b[as]\.(\w+)", early) if f in known}
            if names:
                found[kernel] = names
    assert found == EARLY, {k: (found.get(k), EARLY.get(k)) for k in set(found) | set(EARLY) if found.get(k) != EARLY.get(k)}
