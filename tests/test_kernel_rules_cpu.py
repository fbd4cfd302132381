"""Rules of the CUDA sources that no run can show to be broken (what they guard against is a race), checked on the text."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "deepseek-v4.1-flash-pro6000_b200", "csrc")


def source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def braced(text, start):
    """What stands between the first brace from `start` on and the brace that closes it."""
    at = begin = text.index("{", start) + 1
    depth = 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
    return text[begin:at - 1]


def kernels():
    """(file, kernel, parameters, body) of every __global__ function."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = source(name)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            at, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            parameters = text[m.end():at - 1]
            yield name, m.group(1), parameters, braced(text, at)


def test_every_kernel_is_found():
    found = {k for _, k, _, _ in kernels()}
    assert len(found) >= 22 and {"row_kernel", "head_fp8_kernel", "verify_rows_fast_kernel", "flat_mass_kernel"} <= found
    assert sum(source(n).count("__global__") for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh"))) == len(list(kernels()))


REMOTE = re.compile(r"map_shared_rank|\bexchange\(c,|\bexchange_by_reading\(|\brow_body\s*<|cluster\.sync\(|\bdraw_region\(|"
                    r"\bnucleus_row\(|\bfast_small_support\(|\bgeneral_search\(|\bpeer_(?:load|store)_\w+\(|\bpeer_addr\(|"
                    r"\bmbar_arrive_leader\(|\btma_load_pair\(|\bumma_f8_pair\b|\bumma_commit_pair\(")
PLAIN_PTX = {"flat_front_kernel", "head_fp8_pair_kernel"}    # clusters by csrc/cluster.cuh


def test_cluster_kernels_wait_until_every_cta_has_started():
    """Another CTA's shared memory is touched only behind a barrier of the whole cluster, without which that CTA need not have
    started: announced, then awaited, in the same block and without a way around it, before the first access."""
    seen = set()
    for name, kernel, _, body in kernels():
        if not re.search(r"make_ctx\(|this_cluster\(|\bcluster_rank\(", body):
            assert not REMOTE.search(body), (name, kernel)
            continue
        seen.add(kernel)
        if kernel == "row_kernel" or kernel in PLAIN_PTX:
            continue                     # the next tests
        assert body.count("cluster_announce();") == 1 and body.count("cluster_await();") == 1, (name, kernel)
        announced, awaited = body.index("cluster_announce();"), body.index("cluster_await();")
        assert announced < awaited < REMOTE.search(body).start(), (name, kernel)
        between = body[announced:awaited]
        assert "return" not in between and between.count("{") == between.count("}"), (name, kernel)
        if kernel == "verify_kernel":    # inside the branch that a rejection takes, which holds every access
            branch = body.index("if (walk.status >= 0 && walk.rejected && !greedy)")
            assert branch < announced and not REMOTE.search(body.replace(braced(body, branch), "")), kernel
        else:
            assert "{" not in body[:announced] and "return" not in body[:announced], (name, kernel)
    assert seen == {"row_kernel", "verify_kernel", "verify_rows_fast_kernel", "probability_rows_kernel", "score_kernel"} | PLAIN_PTX


def enclosing(text, at):
    """Where the blocks begin that hold the place `at`, the outermost first."""
    open_ = []
    for i, ch in enumerate(text[:at]):
        if ch == "{":
            open_.append(i)
        elif ch == "}":
            open_.pop()
    return open_


def test_barriers_of_the_cluster_stand_around_the_accesses_in_plain_ptx():
    """Kernels that use csrc/cluster.cuh: before an access to another CTA's shared memory, and behind the last one, every thread of the
    cluster passes a barrier: one in the same block or in a block around it, and no block of a barrier depends on more than the variant."""
    seen = set()
    for name, kernel, _, body in kernels():
        if kernel not in PLAIN_PTX:
            continue
        seen.add(kernel)
        assert "return" not in without_lambdas(body), kernel
        barriers = [m.start() for m in re.finditer(r"\bcluster_barrier\(\);", body)]
        variants = [i for i in (body.find("if constexpr (kKnown) {"),) if i >= 0]
        variants = [i + len("if constexpr (kKnown) {" + braced(body, i) + "} else ") for i in variants]
        assert all(set(enclosing(body, b)) <= set(variants) for b in barriers), kernel
        accesses = [m.start() for m in REMOTE.finditer(body)]
        assert len(accesses) >= 5, kernel
        for at in accesses:
            around = enclosing(body, at)
            assert any(b < at and enclosing(body, b) == around[:len(enclosing(body, b))] for b in barriers), (kernel, body[at:at + 60])
        last = [b for b in barriers if b > accesses[-1] and not enclosing(body, b)]
        assert last, kernel
        given_back = body.find("tcgen05.dealloc.cta_group::2")       # the pair's tensor memory: by both, neither gone
        assert given_back < 0 or last[0] < given_back < last[-1], kernel
    assert seen == PLAIN_PTX
    users = {n for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh")) and '#include "cluster.cuh"' in open(os.path.join(CSRC, n)).read()}
    assert users == {"flat.cu", "head_fp8.cu"}


def test_an_early_arrival_at_the_clusters_barrier_is_completed():
    """The CTA that ends a row alone arrives early, behind its last access to another CTA's shared memory, and completes that barrier
    before its next row; the others pass it as the row's end.  Nowhere else is a barrier of the cluster taken apart."""
    fast, row = source("row_fast.cuh"), source("row_kernel.cuh")
    text = braced(fast, fast.index("FastOutcome fast_small_support("))
    assert text.count("cluster_arrive();") == 1 and "if (release) cluster_arrive();" in text
    ahead, behind = text.split("if (release) cluster_arrive();")
    assert "out.applicable = 1;\n  if (c.rank != 0) return out;" in ahead      # one CTA, and its row is decided
    assert not enclosing(text, text.index("cluster_arrive();"))
    assert not REMOTE.search(behind) and "lists" not in behind and "return out;" in behind and behind.count("return out;") == 1
    body = braced(row, row.index("bool row_body("))
    call, complete = body.index("fast_small_support("), body.index("cluster_complete();")
    branch = "if (f.applicable) {"
    assert body.count("cluster_complete();") == 1 and call < body.index(branch) < complete
    taken = braced(body, body.index("if (release && c.rank == 0)"))
    assert re.sub(r"\s+", " ", taken).strip() == "cluster_complete(); __syncthreads(); closed = true;"
    assert body.rindex("return closed;") > complete
    assert "if (!row_body<kMode, kPerSm>(a, c, s, row)) c.cluster.sync();" in row
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh")):
            text = re.sub(r"__device__ __forceinline__ void cluster_(?:arrive|complete)\(\)[^\n]*", "", source(name))
            uses = len(re.findall(r"\bcluster_(?:arrive|complete)\(\)", text))
            assert uses == {"row_fast.cuh": 1, "row_kernel.cuh": 1}.get(name, 0), name


def test_first_exchange_of_a_row_reads():
    """row_kernel has no barrier of the cluster in front of its rows: a row begins with an exchange in which every CTA writes to
    its own memory and reads the others' behind the barrier, or, with the head's record, with a plain barrier."""
    text = source("row_kernel.cuh")
    body = braced(text, text.index("bool row_body("))
    calls = [m.group(0) for m in REMOTE.finditer(body)]
    assert calls[:2] == ["exchange_by_reading(", "cluster.sync("], calls
    barrier = "if (known && (status != 0 || a.top_p >= 1.0 || !s->map.ok)) c.cluster.sync();"
    assert body.index("exchange_by_reading(") < body.index(barrier) < body.index("nucleus_row(")
    assert body.rindex("if (!known) {", 0, body.index("exchange_by_reading(")) > 0
    text = source("row_nucleus.cuh")     # with a cut, the row's range usable: the histogram's barrier comes first
    body = braced(text, text.index("NucleusOut nucleus_row("))
    first = REMOTE.search(body)
    assert first.group(0) == "cluster.sync(" and "return" not in body[:first.start()].replace("if (!s->map.ok) return out;", "")
    text = source("row_core.cuh")
    body = braced(text, text.index("Slot exchange_by_reading("))
    assert body.index("*at = mine") < body.index("cluster.sync(") < body.index("map_shared_rank")


WAIT = "cudaGridDependencySynchronize();"
ROLES = {"head_fp8_kernel": 3, "head_fp8_decode_kernel": 3, "head_fp8_pair_kernel": 4}   # kernels of specialised warps: their roles


def early_kernels():
    """The kernels that are launched before the one in front of them has finished (csrc/launch.h)."""
    names = set()
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            names |= set(re.findall(r"\blaunch_early\(\s*(\w+)|\blaunch_clusters<(\w+)>|cudaLaunchKernelEx\(&cfg, (\w+)", source(name)))
    return {n for group in names for n in group if n} - {"kernel", "score_kernel"}   # (a template's parameter; launched plainly)


def without_lambdas(text):
    """What a text runs by itself: definitions `auto name = [...](...) {...};` are taken out, whose calls stay."""
    while (m := re.search(r"auto \w+ = \[", text)):
        text = text[:m.start()] + text[text.index("{", m.start()) + len(braced(text, m.start())) + 2:]
    return text


def test_early_kernels_wait_before_they_touch_global_memory():
    early = early_kernels()
    assert {"row_kernel", "head_fp8_kernel", "flat_mass_kernel", "verify_rows_fast_kernel", "replay_sample_kernel"} <= early
    assert PLAIN_PTX | {"head_fp8_decode_kernel"} <= early
    seen = {}
    for name, kernel, parameters, body in kernels():
        if kernel not in early:
            continue
        seen[kernel] = name
        text = without_lambdas(body)
        assert WAIT in text, (name, kernel)
        pointers = re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)\s*(?:,|$)", parameters)
        touch = r"__ldg\(|__ldc|load_input\(|tma_load|cp\.async\.c|copy4_async\(|\bfetch(?:_scales)?\(|stage_begin\(|\brow_body|\b[ap]\.\w+\["
        touch += "".join(rf"|\b{p}\[|(?<!prefetch_l2\()\b{p} \+" for p in pointers)
        parts = [text]
        if kernel in ROLES:              # (the warps go separate ways, each with a wait of its own)
            parts = [part for part in re.split(r"\} else (?:if \([^{]*)?\{", text) if WAIT in part]
            assert len(parts) == text.count(WAIT) == ROLES[kernel], kernel
        for part in parts:
            before = part[:part.index(WAIT)]
            assert not re.search(touch, before), (name, kernel, re.search(touch, before))
    assert set(seen) == early, early - set(seen)


def test_no_read_only_loads_of_what_the_kernel_in_front_may_write():
    """The read-only path is for data that nobody writes while the kernel runs: constants, and the inputs of kernels that are not
    launched early (the score, the streaming path, the compact head whose activations fill the shared memory)."""
    early = early_kernels()
    plain_files = {"score.cu", "stream.cuh"}
    for name, kernel, parameters, _ in kernels():
        if kernel in early:
            assert name not in plain_files and "__restrict__" not in parameters, (name, kernel)
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".h")) or name in plain_files:
            continue
        text = source(name)
        for _, kernel, _, body in (k for k in kernels() if k[0] == name and k[1] not in early):
            text = text.replace(body, "")
        assert set(re.findall(r"__ldg\(([^)]*)\)", text)) <= {"&kExp2Table[n & 63]"}, name
        assert "ld.global.nc" not in text, name


def test_only_the_clearing_kernel_signals_before_its_wait():
    """csrc/launch.h says which kernels let their successor start when: after their own wait, but for one."""
    before = set()
    for _, kernel, _, body in kernels():
        signal = "cudaTriggerProgrammaticLaunchCompletion();"
        if signal in body and body.index(signal) < body.index(WAIT):
            before.add(kernel)
    assert before == {"clear_stats_kernel"}


def test_waits_for_another_ctas_arrivals_have_the_clusters_scope():
    """A barrier that another CTA arrives at with the cluster's scope is waited on with that scope, and the wait has the order that the
    arrival has (relaxed: the tensor memory's accesses are ordered by the tcgen05 fences around both)."""
    text = source("head_fp8.cu")
    arrival = braced(text, text.index("void mbar_arrive_leader("))
    assert "mbarrier.arrive.relaxed.cluster.shared::cluster" in arrival
    probe = braced(text, text.index("bool mbar_try("))
    wide = probe[probe.index("if constexpr (kCluster)"):probe.index("else")]
    assert "mbarrier.try_wait.parity.relaxed.cluster.shared::cta" in wide
    waits = braced(text, text.index("bool mbar_wait("))
    assert set(re.findall(r"mbar_try(<\w+>)?\(", waits)) == {"<kCluster>"}
    seen = []
    for name, kernel, _, body in kernels():
        for address in set(re.findall(r"\bmbar_arrive_leader\((\w+)", body)):
            barrier = re.search(rf"\b{address} = peer_addr\((\w+), 0\);", body).group(1)
            found = re.findall(rf"mbar_wait(<true>)?\(&{barrier}\[", body)
            assert found and set(found) == {"<true>"}, (kernel, barrier)
            seen.append((kernel, barrier))
    assert seen == [("head_fp8_pair_kernel", "acc_empty")]
