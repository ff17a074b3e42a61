"""Rules of the kernels that cannot be shown by running them without hanging a GPU: read from their sources."""
import glob
import os
import random
import re

import pytest

import helpers

CSRC = os.path.join(helpers.PKG_DIR, "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def plain(path):
    """The source without comments."""
    text = re.sub(r"//[^\n]*", "", open(path).read())
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
        at, depth = text.index("{", m.end()), 0
        for i in range(at, len(text)):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            if depth == 0:
                yield m.group(1), text[at:i]
                break


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_tensor_memory_is_taken_before_successors_may_start(path):
    """A successor that is placed beside a CTA without its columns yet could take them and wait for this grid for good. A trigger
    before the allocation is allowed where the CTA leaves right after it."""
    for name, body in kernels(plain(path)):
        alloc = re.search(r"\btmem_alloc\w*\(", body)
        for m in re.finditer(r"\bpdl_trigger\(\);", body[:alloc.start()] if alloc else ""):
            assert "return;" in body[m.end():body.index("}", m.end())], name


def test_unbounded_barriers_do_not_hang_on_a_wait_that_ran_out():
    """A warp whose bounded wait ran out must not leave others in a named barrier, which has no bound: the prompt kernel has none,
    and in the CTA-pair kernel the warps that trade columns walk all units whatever their waits gave. What went wrong is reported
    once no thread can find out any more, and copies in flight are waited for then, whoever gave up."""
    (prompt,) = [b for _, b in kernels(plain(os.path.join(CSRC, "attention_prefill_tc.cu")))]
    assert "bar.sync" not in prompt
    (pair,) = [b for _, b in kernels(plain(os.path.join(CSRC, "gemm_tc_pair.cu")))]
    epilogue = pair[pair.index("setmaxnreg.inc"):]
    units = re.search(r"for \(uint32_t u = pair; u < a\.units([^;]*);", epilogue)
    assert units.group(1) in ("", " && (PAIRED || ok)") and "if (!ok) break;" not in epilogue
    for body in (prompt, pair):
        end = body.rindex("__syncthreads();")
        assert re.search(r"if \(abort_flag\b", body[end:]) and "_full[i]" in body[end:] or "&full[s]" in body[end:]
    assert "a.status" not in pair[:pair.rindex("__syncthreads();")]


def expression(text):
    """A C expression of unsigned names and numbers as a Python one."""
    return re.sub(r"\b(\d+)u\b", r"\1", text).replace("a.stages", "stages").replace("/", "//").replace("&&", "and")


def statements(text):
    """Comma-separated C assignments and increments as Python ones."""
    return [re.sub(r"\+\+(\w+)", r"\1 += 1", re.sub(r"^uint32_t ", "", expression(part.strip()))) for part in text.split(",")]


def test_ring_of_the_few_rows_kernel():
    """Four warps write every fourth k-block of the activation operand and wait by parity for the stage's last use only. The first stage, the
    parity waited for and the way on are taken from the kernel. Any order in which the warps and the issuing one may run, on every ring that the
    launch allows: no stage is overwritten early, none waits for good."""
    source = plain(os.path.join(CSRC, "gemm_tc_rows.cu"))
    low, high = (int(re.search(rf"{n} = (\d+)", source).group(1)) for n in ("MIN_STAGES", "MAX_STAGES"))
    assert "a.stages < MIN_STAGES" in source
    maker = source[source.index("void make_operand("):source.index("gemm_tc_rows_kernel(")]
    start = statements(re.search(r"(uint32_t s = [^;]*, round = [^;]*);", maker).group(1))
    waits, parity = re.search(r"if \(half == 0 && (.*?)\) ok = __all_sync\(0xffffffffu, !\*abort_flag && mbar_wait\(&empty\[s\], (.*?)\)\);", maker).groups()
    step, wraps, wrap = re.search(r"if \(lane == 0\) mbar_arrive\(&x_full\[s\]\);\s*(s \+= [^;]*);\s*if \((.*?)\) (s -= [^;]*);", maker).groups()
    # the k-block that is converted at stage s of the round is w + 4 i: as the columns are fetched and the trips counted
    assert "(kb0 + w + t / UNITS * 4u) * BLOCK_K" in maker and "(n_kb - w + 3u) / 4u * UNITS" in maker
    issuer = source[source.index("} else if (warp == 1) {"):]
    assert re.search(r"uint32_t s = 0, phase = 0;", issuer) and "mbar_wait(&x_full[s], phase)" in issuer
    assert re.search(r"if \(\+\+s == a\.stages\) s = 0, phase \^= 1u;", issuer)

    def run(stages, blocks, rng):
        freed, filled, holds, done = [0] * stages, [0] * stages, {}, 0
        makers = [{"w": w, "stages": stages} for w in range(4)]
        for m in makers:
            for line in start:
                exec(line, {}, m)
        at = list(range(4))  # each warp's next k-block
        while done < blocks:
            ready = [w for w, m in enumerate(makers) if at[w] < blocks and
                     (not eval(expression(waits), {}, m) or freed[m["s"]] % 2 != eval(expression(parity), {}, m))]
            if filled[done % stages] % 2 != done // stages % 2:
                ready.append(4)
            assert ready, (stages, blocks, done)
            w = rng.choice(ready)
            if w == 4:
                assert holds[done % stages] == done
                freed[done % stages] += 1
                done += 1
            else:
                m = makers[w]
                assert at[w] - stages < done and m["s"] == at[w] % stages
                holds[m["s"]] = at[w]
                filled[m["s"]] += 1
                at[w] += 4
                exec(expression(step), {}, m)
                if eval(expression(wraps), {}, m):
                    for line in statements(wrap):
                        exec(line, {}, m)

    rng = random.Random(1)
    for stages in range(low, high + 1):
        for blocks in (1, 2, 3, 4, 5, 7, 11, 13, 28, 56):
            for _ in range(20):
                run(stages, blocks, rng)
