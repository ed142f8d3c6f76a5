"""The chunk-wise delta rule's hand-overs, read from its source: what each role waits for, loads, hands
over and reads, as a graph of what comes before what.  A buffer may only be copied over once every read of it
lies before, and a wait for a phase of a barrier must lie before that barrier's next phase can end (a wait
knows a phase's parity only)."""

import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parent.parent / "mini_llm_stack_b200" / "csrc" / "delta_chunk.cu"
CHUNKS = 6
ROLES = ("copies", "products", "columns 0", "columns 1")     # two warps of columns stand for all eight


def programs(text):
    """Per role its steps (what, barrier or buffer, chunk), all chunks one after the other."""
    walk = text[text.index("delta_chunk_scan_kernel(const"):]
    copies, rest = walk.split("} else if (warp == 9) {")
    products, columns = rest.split("} else if (warp < 8) {")
    out = {r: [] for r in ROLES}
    # what is loaded ahead of the loop, then the loop
    ahead, loop = copies[copies.index("load_k(0);"):].split("for (int c = 0; c + 1 < w.chunks; ++c) {")
    for buf, c in re.findall(r"load_(\w)\((\d)\)", ahead):
        out["copies"].append(("load", buf.upper(), int(c)))
    loop = loop[:loop.index("if (timed_out) break;")]
    steps = re.findall(r"mbar_wait\(bar\((\w+)\)|load_(\w)\(c \+ (\d)\)", loop)
    for c in range(CHUNKS - 1):
        for bar, buf, ahead in steps:
            if bar:
                out["copies"].append(("wait", bar, c))
            elif c + int(ahead) < CHUNKS:
                out["copies"].append(("load", buf.upper(), c + int(ahead)))
    body = products[products.index("for (int c = 0; c < w.chunks; ++c)"):]
    steps = re.findall(r"wait\((\w+)(?: \+ ph)?, [^)]|umma_commit\(bar\((\w+)\)", body)
    for c in range(CHUNKS):
        out["products"] += [("wait", w, c) if w else ("end", e, c) for w, e in steps]
    body = columns[columns.index("for (int c = 0; c < w.chunks; ++c)"):]
    body = body[:body.index("store(w.chunks - 1);")]
    body = re.sub(r"const float\* factors = .*", "", body)
    steps = re.findall(r"[^_]wait\((\w+)(?: \+ ph)?, |hand_over\((\w+)\)|(factors(?:_s)?)\b", body)
    for role in ROLES[2:]:
        for c in range(CHUNKS):
            for wait, put, read in steps:
                out[role].append(("wait", wait, c) if wait else ("put", put, c) if put else ("read", "factors", c))
    return out


def faults(text):
    progs = programs(text)
    after = {}                                               # node -> nodes that come after it
    ends = {}                                                # (barrier, chunk) -> node at which that phase ends

    def edge(a, b):
        after.setdefault(a, set()).add(b)

    for role, steps in progs.items():
        for i, (what, name, c) in enumerate(steps):
            node = (role, i)
            if i:
                edge((role, i - 1), node)
            if what == "load":
                ends[(name + "_FULL", c)] = node
            elif what == "end":
                ends[(name, c)] = node
            elif what == "put":                              # all warps of columns meet, then one arrives
                edge(node, ("met", name, c))
                edge(("met", name, c), (role, i + 1))
                ends[(name, c)] = ("met", name, c)
    waits = [((role, i), name, c) for role, steps in progs.items() for i, (what, name, c) in enumerate(steps)
             if what == "wait"]
    for node, name, c in waits:
        edge(ends[(name, c)], node)

    def reaches(a, b):
        seen, todo = {a}, [a]
        while todo:
            x = todo.pop()
            if x == b:
                return True
            for y in after.get(x, ()):
                if y not in seen:
                    seen.add(y)
                    todo.append(y)
        return False

    found = []
    for node, name, c in waits:
        apart = 2 if name == "K_FULL" else 1                 # (two barriers that take turns)
        later = ends.get((name, c + apart))
        if later and not reaches(node, later):
            found.append(f"{node[0]} may see {name} of chunk {c} two phases late")
    for role, steps in progs.items():
        for i, (what, name, c) in enumerate(steps):
            if what == "read":
                later = ends.get(("K_FULL", c + 2))          # the factors come with the keys, two buffers
                if later and not reaches((role, i), later):
                    found.append(f"{role} may read the factors of chunk {c} under their overwriting")
    # operands that products read from shared memory: done once the products' own barrier has ended
    for buf, bar, apart in (("K", "KU", 2), ("Q", "QS2", 1), ("T", "TR", 1), ("P", "PU", 1)):
        for c in range(CHUNKS - apart):
            if not reaches(ends[(bar, c)], ends[(buf + "_FULL", c + apart)]):
                found.append(f"{buf} of chunk {c} may be copied over under its product")
    return sorted(set(found))


def test_every_read_lies_before_its_overwriting_and_no_wait_is_lapped():
    text = SOURCE.read_text()
    progs = programs(text)
    # the extraction sees the whole protocol
    assert {n for w, n, _ in progs["products"] if w == "end"} == {"KS", "QS", "TR", "QS2", "KU", "PU"}
    assert {n for w, n, _ in progs["columns 0"] if w == "put"} == {"S_PUT", "R_PUT", "O_READ", "Z_PUT", "U_PUT"}
    assert sum(w == "read" and c == 0 for w, _, c in progs["columns 0"]) >= 5
    assert {n for w, n, _ in progs["copies"] if w == "load"} == {"K", "Q", "T", "P"}
    assert faults(text) == []


def test_the_graph_finds_planted_mistakes():
    text = SOURCE.read_text()
    # the copies look at the state's product instead of the chunk's last one
    early = text.replace("if (!mbar_wait(bar(PU), c & 1)) timed_out = true;",
                         "if (!mbar_wait(bar(KU), c & 1)) timed_out = true;")
    assert early != text
    assert any("factors" in f for f in faults(early)) and any("two phases" in f for f in faults(early))
