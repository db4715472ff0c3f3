"""Generated register passes run on the CPU: the text of each launch
(qs_jit_pass_source) with its parameter block (qs_jit_pass_params), as numpy
statements over all threads of all tiles, in the pass's own precision."""
import ctypes as C
import re

import numpy as np


def plan_launches(ops, n, esize, knobs):
    """(launches, matrix table): (source, parameter block) of every launch of
    the fused passes of `ops`, in order; knobs = (tile bits, low bits, merge bits)."""
    from quict_b200 import _native as N
    from quict_b200.simulation.fusion import MatrixTable, Pass, emit, iter_plan, relabel_swaps
    lib = N.load()
    steps = list(iter_plan(relabel_swaps(ops, n), n, knobs[0], knobs[1], merge_bits=knobs[2]))
    assert all(isinstance(s, Pass) for s in steps)
    table = MatrixTable()
    cps, npass, cops, nops = emit([s for s in steps if s.ops], table)
    host = table.array().astype(np.complex128 if esize == 16 else np.complex64)
    out = []
    for i in range(npass):
        li = 0
        while True:
            head = (n, N.QS_C128 if esize == 16 else N.QS_C64, C.byref(cps[i]), cops, nops,
                    C.c_void_p(host.ctypes.data), host.size, li)
            ln = C.c_int64(0)
            src, par = C.create_string_buffer(1 << 22), np.zeros(1 << 16, dtype=np.uint8)
            rc = lib.qs_jit_pass_source(*head, src, len(src), C.byref(ln))
            if rc != 0:
                assert rc == N.QS_EINVAL and li > 0, N.load().qs_last_error()
                break
            assert lib.qs_jit_pass_params(*head, C.c_void_p(par.ctypes.data), par.nbytes, C.byref(ln)) == 0
            out.append((src.value.decode(), par[:ln.value].copy()))
            li += 1
    return out, host


def sources(circuit, n, esize, knobs):
    from quict_b200.simulation.lowering import lower_circuit
    return [s for s, _ in plan_launches(lower_circuit(circuit.gates, n), n, esize, knobs)[0]]


def params(src, block):
    """The parameter block's fields by name."""
    fields = re.search(r"struct __align__\(16\) P \{(.*?)\};", src).group(1)
    cd = "c16" if "typedef double2 V;" in src else "c8"
    out, at = {}, 0
    for typ, name, cnt in re.findall(r"(V|u64|u32) (\w+)(?:\[(\d+)\])?;", fields):
        d = np.dtype({"V": cd, "u64": "u8", "u32": "u4"}[typ])
        k = int(cnt or 1)
        out[name] = block[at:at + k * d.itemsize].view(d)
        at += k * d.itemsize
    return out


def _python(e):
    """A C expression of the generated text as a numpy expression."""
    e = re.sub(r"\b(\d+)u(?:ll)?\b", r"\1", e)
    e = e.replace("u32(", "(").replace("&&", "&")
    return re.sub(r"p\.(\w+)\[", r"p['\1'][", e)


def run_launch(vec, src, block, norms=None):
    """One launch on `vec` (in place).  norms: list that gets the vector's 2-norm
    at every relayout, i.e. between the stages."""
    p = params(src, block)
    head = re.search(r"n=(\d+) K=(\d+) L=(\d+) R=(\d+)", src)
    n, K, L, R = (int(x) for x in head.groups())
    H, ntiles, threads = K - L, 1 << (n - K), 1 << (K - R)
    t = np.arange(ntiles, dtype=np.int64) << L
    hib = p["hibit"][:H].astype(np.int64)
    for b in hib:
        t = ((t & ~(b - 1)) << 1) | (t & (b - 1))
    base = t[:, None]
    e = np.arange(1 << K)
    hoff = np.zeros(1 << H, dtype=np.int64)
    for i, b in enumerate(hib):
        hoff |= np.where((np.arange(1 << H) >> i) & 1, b, 0)
    tid = np.arange(threads, dtype=np.int64)
    cur = vec[base | hoff[e >> L] | (e & ((1 << L) - 1))]
    T, F = vec.dtype, vec.real.dtype.type
    dsm = np.zeros(1 << 13, dtype=T)

    def cmul(a, b):
        return np.multiply(a, b, dtype=T)

    def of(a, x):  # a real factor times both components
        out = np.empty(np.broadcast(a, x).shape, dtype=T)
        out.real, out.imag = a * x.real, a * x.imag
        return out

    def imul(b, x):
        out = np.empty(np.broadcast(b, x).shape, dtype=T)
        out.real, out.imag = -b * x.imag, b * x.real
        return out

    env = dict(p={k: (v.astype(np.int64) if v.dtype == np.uint64 else v) for k, v in p.items()}, base=base, tid=tid,
               dsm=dsm, np=np, cmul=cmul, cfma=lambda a, b, c: cmul(a, b) + c, cadd=lambda a, b: a + b,
               cneg=lambda a: -a, rmul=of, rfma=lambda a, x, c: of(a, x) + c, imul=imul,
               ifma=lambda b, x, c: imul(b, x) + c, csel=lambda c, a, b: np.where(c, a, b),
               zero=np.zeros((1, 1), dtype=T), cur=cur, vec=vec)
    env["gthr"] = sum(np.where((tid >> i) & 1, int(p["gthr"][i]), 0) for i in range(K - R))
    shape = (ntiles, threads)
    for line in src.split("\n"):
        line = line.strip()
        if m := re.match(r"for \(u32 q = tid; q < (\d+)u; q \+= \d+u\) dsm\[(\d+) \+ q\] = p\.m\[(\d+) \+ q\];", line):
            k, d, s = (int(x) for x in m.groups())
            dsm[d:d + k] = p["m"][s:s + k]
        elif m := re.match(r"const (?:u32|bool) (RD\d+|WR\d+|TH\d+|h\d+|c\d+) = (.*);", line):
            env[m.group(1)] = eval(_python(m.group(2)), env)
        elif m := re.match(r"const V (v\d+) = (.*);", line):
            x = m.group(2)
            x = re.sub(r"make_(?:float|double)2\(0, 0\)", "zero", x)
            x = re.sub(r"cur\[(.*)\]", r"cur[:, \1]", x)
            x = x.replace("].x", "].real").replace("].y", "].imag")
            if c := re.match(r"(c\d+) \? (.*) : (v\d+)$", x):
                x = f"np.where({c.group(1)}, {c.group(2)}, {c.group(3)})"
            env[m.group(1)] = np.broadcast_to(eval(_python(x), env), shape)
        elif m := re.match(r"cur\[(.*)\] = (v\d+);", line):
            cur[:, eval(_python(m.group(1)), env) + 0 * tid] = env[m.group(2)]
        elif m := re.match(r"vec\[(base .*)\] = (v\d+);", line):
            vec[eval(_python(m.group(1)), env)] = env[m.group(2)]
        elif line == "__syncthreads();" and norms is not None:
            norms.append(float(np.linalg.norm(cur.astype(np.complex128))))
    return vec


def run(circuit, n, esize, knobs, norms=None):
    """The circuit from |0...0> through its generated passes (complex64 for
    esize 8, complex128 for 16)."""
    from quict_b200.simulation.lowering import lower_circuit
    launches, host = plan_launches(lower_circuit(circuit.gates, n), n, esize, knobs)
    vec = np.zeros(1 << n, dtype=host.dtype)
    vec[0] = 1
    with np.errstate(all="ignore"):
        for src, block in launches:
            run_launch(vec, src, block, norms)
    return vec
