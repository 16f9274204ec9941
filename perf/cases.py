"""The work this framework is used for, as measurable cases.

Every case goes through the public Python entry points (b2lstm.Net, LstmLayer, train_epoch, matrix_multiply) with the
inputs, the batch shapes and the options of a training or synthesis program.  Kinds of case:

  train   one minibatch of training: load, forward, error, BPTT, weight gradients, update.  "host": the minibatch comes
          from pinned host memory and the error goes back (Net.train_step); otherwise it is resident on the GPU
          (Net.train_step_dev)
  infer   forward pass and error of one fraction (validation, or the synthesis of one utterance with "P" 1)
  layer   one (b)lstm layer, forward and backward, on the caller's own device buffers (the drop-in boundary)
  epoch   one pass of training over a data file in the toolkit's .nc layout (data loader, copies and all steps)
  gemm    one matrix product through the GEMM wrapper

A stack is described by "in" inputs, "ff" feed-forward layers of "ff_size" units, "rec" recurrent layers of "units"
units per direction ("bi": both directions) and "out" outputs; "P" parallel sequences with lengths between "lo" and "hi"
frames, sorted (a data set sorts by length).  Sizes are those of the benchmark configurations, of the tests and of the
example logs quoted with them.
"""
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "project-currennt-public_b200"))
import b2lstm  # noqa: E402


def listed():
    return [
        # the smallest training step: one unidirectional layer, 4 short sequences; launches and host work count
        dict(name="train lstm128 4x200", kind="train", **{"in": 64}, binary=0, ff=0, ff_size=0, act="tanh", rec=1, units=128, bi=False,
             out=32, P=4, lo=200, hi=200, host=False, option=0),
        # the acoustic model of speech synthesis: 2 feed-forward + 2 blstm layers, 32 utterances of 300..1200 frames
        dict(name="train acoustic 32", kind="train", **{"in": 382}, binary=350, ff=2, ff_size=512, act="tanh", rec=2, units=256, bi=True,
             out=187, P=32, lo=300, hi=1200, host=False, option=0),
        # the same model with few utterances a step, minibatch from host memory, error read back after every step
        dict(name="train acoustic 4 host", kind="train", **{"in": 382}, binary=350, ff=2, ff_size=512, act="tanh", rec=2, units=256,
             bi=True, out=187, P=4, lo=300, hi=1200, host=True, option=0),
        # wide and deep: 4 blstm layers of 1024 units per direction, 64 sequences of one length
        dict(name="train deep 1024 64x1000", kind="train", **{"in": 512}, binary=0, ff=0, ff_size=0, act="tanh", rec=4, units=1024,
             bi=True, out=256, P=64, lo=1000, hi=1000, host=False, option=0),
        # online learning on one very long sequence: nothing but dependent steps
        dict(name="train online 1x8000", kind="train", **{"in": 128}, binary=0, ff=0, ff_size=0, act="tanh", rec=2, units=512, bi=True,
             out=80, P=1, lo=8000, hi=8000, host=False, option=0),
        # large-batch training, and the share of it that one of eight data-parallel processes has
        dict(name="train batch 256", kind="train", **{"in": 382}, binary=350, ff=0, ff_size=0, act="tanh", rec=3, units=512, bi=True,
             out=187, P=256, lo=600, hi=1000, host=False, option=0),
        dict(name="train share 32", kind="train", **{"in": 382}, binary=350, ff=0, ff_size=0, act="tanh", rec=3, units=512, bi=True,
             out=187, P=32, lo=600, hi=1000, host=False, option=0),
        # sizes off the powers of two, the AdaGrad option
        dict(name="train odd 160 8", kind="train", **{"in": 382}, binary=350, ff=1, ff_size=300, act="logistic", rec=2, units=160, bi=True,
             out=187, P=8, lo=300, hi=1200, host=False, option=1),
        # an epoch over a small corpus, one utterance at a time (the example log's network and its two utterances)
        dict(name="epoch blstm128 2 files", kind="epoch", **{"in": 382}, binary=350, ff=1, ff_size=512, act="tanh", rec=1, units=128,
             bi=True, out=259, P=1, lo=570, hi=946, nseq=2),
        # synthesis of one utterance with the acoustic model
        dict(name="infer acoustic 1x700", kind="infer", **{"in": 382}, binary=350, ff=2, ff_size=512, act="tanh", rec=2, units=256, bi=True,
             out=187, P=1, lo=700, hi=700),
        # a unidirectional layer inside another program, on that program's buffers
        dict(name="layer lstm512 50x300", kind="layer", **{"in": 512}, units=512, bi=False, P=50, lo=100, hi=300),
        # one product of the GEMM wrapper, ragged in all three sizes
        dict(name="gemm 187x9001x509 tn", kind="gemm", m=187, n=9001, k=509, ta=True, tb=False),
    ]


# ---- drawn cases -----------------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _units(rng, lo=16, hi=1024):
    """units per direction: powers of two, round numbers, or any number; but not 4 modulo 8, which earlier builds, the ones
    to compare with, do not run (their weight-gradient product starts its TMA boxes off the 16-byte boundary there)"""
    kind = rng.random()
    if kind < 0.4:
        return 2 ** rng.randint(int(math.log2(lo)), int(math.log2(hi)))
    u = _log_int(rng, lo, hi)
    if kind < 0.7 and u >= 20:
        u = u // 10 * 10
        return u + 10 if u % 8 == 4 else u
    return u + 1 if u % 8 == 4 else u


def draw(rng):
    kind = rng.choices(["train", "infer", "layer", "epoch", "gemm"], [0.55, 0.15, 0.12, 0.08, 0.10])[0]
    if kind == "gemm":
        while True:
            c = dict(kind="gemm", m=_log_int(rng, 16, 4096), n=_log_int(rng, 64, 100000), k=_log_int(rng, 16, 4096), ta=rng.random() < 0.5,
                     tb=False)
            if not c["ta"]:
                c["tb"] = rng.random() < 0.5
            if c["m"] * c["n"] * c["k"] <= 5e11 and c["n"] * (c["m"] + c["k"]) <= 3e8:
                return c
    if kind == "epoch":
        units = _units(rng, 16, 256)
        hi = _log_int(rng, 100, 800)
        return dict(kind="epoch", **{"in": rng.randint(60, 400)}, binary=0, ff=rng.randint(0, 1), ff_size=rng.randint(64, 512), act="tanh",
                    rec=rng.randint(1, 2), units=units, bi=rng.random() < 0.75, out=rng.randint(20, 260), P=_log_int(rng, 1, 16), lo=max(20, hi // 3),
                    hi=hi, nseq=rng.randint(2, 24))
    while True:
        units = _units(rng)
        hi = _log_int(rng, 50, 2000)
        c = dict(kind=kind, **{"in": rng.randint(32, 512)}, units=units, bi=rng.random() < 0.75, P=_log_int(rng, 1, 256),
                 lo=hi if rng.random() < 0.3 else max(1, int(hi * rng.uniform(0.2, 0.9))), hi=hi)
        if kind != "layer":
            c.update(binary=0, ff=rng.randint(0, 2), ff_size=rng.randint(64, 1024), act=rng.choice(["tanh", "logistic"]), rec=rng.randint(1, 3),
                     out=rng.randint(20, 260))
        if kind == "train":
            c.update(host=rng.random() < 0.25, option=rng.choice([0, 0, 0, 1, 2]))
        frames = c["P"] * c["hi"]
        # bounded by the largest listed case: work, memory, and dependent steps (which cost time whatever their work)
        if frames <= 256000 and work(c)["flops"] <= 6e12 and c["hi"] * c.get("rec", 1) <= 4000 and frames * _floats_per_frame(c) <= 6e9:
            return c


# ---- the stack of a case ------------------------------------------------------------------------------------------------
def _layers(c):
    L = [dict(type="input", size=c["in"])]
    L += [dict(type="feedforward_" + c["act"], size=c["ff_size"], bias=1.0) for _ in range(c["ff"])]
    L += [dict(type="blstm" if c["bi"] else "lstm", size=c["units"] * (2 if c["bi"] else 1), bias=1.0) for _ in range(c["rec"])]
    return L + [dict(type="feedforward_identity", size=c["out"], bias=1.0), dict(type="sse", size=c["out"])]


def _floats_per_frame(c):
    """what a net keeps per frame, roughly (states, activations, errors and the operand copies of the GEMMs)"""
    ls = c["units"] * (2 if c["bi"] else 1)
    return c["in"] * 3 + c.get("out", 0) * 4 + c.get("ff", 0) * c.get("ff_size", 0) * 2 + c.get("rec", 1) * ls * 21 + 5 * ls


def _lengths(c, n):
    """n sequence lengths between lo and hi, both met, longest first; the same for every seed (inputs differ, shapes do not)"""
    r = random.Random(c["lo"] * 100003 + c["hi"] * 101 + n)
    lens = [r.randint(c["lo"], c["hi"]) for _ in range(n)]
    lens[0] = c["hi"]
    if n > 1:
        lens[-1] = c["lo"]
    return np.array(sorted(lens, reverse=True), np.int32)


def _rate(c, frames):
    """a learning rate that neither diverges nor stands still: gradients are sums over frames (option 0), averages otherwise"""
    return 1e-3 if c.get("option", 0) else 0.02 / frames


def _frames(gen, T, P, size, binary, lens_dev):
    """[T, P, size] on the GPU: `binary` 0/1 entries (a tenth of them set), the rest N(0, 1); zero behind a sequence's end"""
    x = torch.randn((T, P, size), generator=gen, device="cuda")
    if binary:
        x[:, :, :binary] = (torch.rand((T, P, binary), generator=gen, device="cuda") < 0.1).float()
    x *= (torch.arange(T, device="cuda")[:, None] < lens_dev[None, :]).float()[:, :, None]
    return x


class _View:
    """a buffer of a net, as an array of the device; holds the net as long as somebody holds the array"""

    def __init__(self, net, ptr, shape):
        self.net = net
        self.__cuda_array_interface__ = dict(data=(int(ptr), False), shape=tuple(shape), typestr="<f4", version=3)


def _view(net, ptr, *shape):
    return torch.as_tensor(_View(net, ptr, shape), device="cuda")


def _net(c, seed, T):
    b2lstm.lib().b2_config_set_weights_uniform(-0.05 if c["units"] > 512 else -0.08, 0.05 if c["units"] > 512 else 0.08)
    layers = _layers(c)
    net = b2lstm.Net(layers, c["P"], T, seed=seed)
    if c.get("option", 0):
        net.set_optimizer(c["option"])
    return layers, net


def prepare(case, seed):
    c = dict(case)
    seed = int(seed) & 0x7FFFFFFF
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = {"case": c, "kind": c["kind"]}
    if c["kind"] == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        s["A"] = torch.randn(m * k, generator=gen, device="cuda")
        s["B"] = torch.randn(k * n, generator=gen, device="cuda")
        s["C"] = torch.zeros((n, m), device="cuda")
        s["lda"], s["ldb"] = (k if c["ta"] else m), (n if c["tb"] else k)
        return s
    if c["kind"] == "epoch":
        return _prepare_epoch(c, seed, s)
    lens = _lengths(c, c["P"])
    T, P = int(lens.max()), c["P"]
    lens_dev = torch.from_numpy(lens).cuda()
    s.update(T=T, lens=lens)
    if c["kind"] == "layer":
        ls = c["units"] * (2 if c["bi"] else 1)
        layer = b2lstm.LstmLayer(P, T, c["in"], ls, c["bi"])
        t = torch.arange(T, device="cuda")[:, None]
        pat = torch.full((T, P), 2, device="cuda", dtype=torch.int8)      # 0 padding, 1 first, 2 inside, 3 last
        pat[0] = 1
        pat[(t == lens_dev[None, :] - 1) & (t > 0)] = 3
        pat[t >= lens_dev[None, :]] = 0
        s.update(layer=layer, pat=pat.contiguous(), Tmin=int(lens.min()),
                 w=(torch.rand(layer.num_weights, generator=gen, device="cuda") - 0.5) * 0.16,
                 x=_frames(gen, T, P, c["in"], 0, lens_dev), dy=_frames(gen, T, P, ls, 0, lens_dev) * 0.1,
                 y=torch.zeros((T, P, ls), device="cuda"), dx=torch.zeros((T, P, c["in"]), device="cuda"),
                 dw=torch.zeros(layer.num_weights, device="cuda"))
        torch.cuda.synchronize()
        return s
    layers, net = _net(c, seed, T)
    x = _frames(gen, T, P, c["in"], c["binary"], lens_dev)
    tg = _frames(gen, T, P, c["out"], 0, lens_dev)
    s.update(net=net, layers=layers, rate=_rate(c, int(lens.sum())))
    if c.get("host"):
        hx, ht = torch.empty(x.shape, pin_memory=True), torch.empty(tg.shape, pin_memory=True)
        hx.copy_(x)
        ht.copy_(tg)
        s.update(hold=(hx, ht), x=hx.numpy(), tg=ht.numpy())
    else:
        s.update(x=x, tg=tg)
    torch.cuda.synchronize()
    s["out"] = _results(s)
    return s


def _prepare_epoch(c, seed, s):
    rng = np.random.Generator(np.random.PCG64(seed))
    lens = _lengths(c, c["nseq"])
    n = int(lens.sum())
    x = rng.standard_normal((n, c["in"]), dtype=np.float32)
    if c["binary"]:
        x[:, :c["binary"]] = rng.random((n, c["binary"]), dtype=np.float32) < 0.1
    tg = rng.standard_normal((n, c["out"]), dtype=np.float32)
    fd, path = tempfile.mkstemp(suffix=".nc")
    os.close(fd)
    try:
        b2lstm.write_nc(path, ["s%03d" % i for i in range(len(lens))], [int(v) for v in lens], x, tg)
        s["data"] = b2lstm.DataSet(path, c["P"])
    finally:
        os.unlink(path)   # the data set has mapped it
    s["layers"], s["net"] = _net(c, seed, int(lens.max()))
    s.update(T=int(lens.max()), rate=_rate(c, n // (2 if len(lens) > c["P"] else 1)))
    s["out"] = _results(s)
    return s


def _results(s):
    """device views of what a pass leaves behind: the last layer's outputs, in training the gradients and the weights"""
    c, net, layers, lib = s["case"], s["net"], s["layers"], b2lstm.lib()
    last = len(layers) - 2
    out = {}
    if c["kind"] != "epoch":
        out["outputs"] = _view(net, lib.b2_net_outputs_dev(net.h, last), s["T"], c["P"], c["out"])
    if c["kind"] != "infer":
        for i in range(1, last + 1):
            out["gradient%d" % i] = _view(net, lib.b2_net_weight_updates_dev(net.h, i), net.num_weights(i))
            out["weights%d" % i] = _view(net, lib.b2_net_weights_dev(net.h, i), net.num_weights(i))
    return out


def run(s):
    c, kind = s["case"], s["kind"]
    if kind == "train":
        if c["host"]:
            return s["net"].train_step(s["lens"], s["x"], s["tg"], s["rate"], 0.9), s["out"]
        s["net"].train_step_dev(s["lens"], s["T"], s["x"], s["tg"], s["rate"], 0.9)
        return s["out"]
    if kind == "infer":
        s["net"].load_fraction_dev(s["lens"], s["T"], s["x"], s["tg"])
        return s["net"].forward(), s["out"]
    if kind == "epoch":
        error, frames = b2lstm.train_epoch(s["net"], s["data"], s["rate"], 0.9)
        return error, frames, s["out"]
    if kind == "layer":
        layer = s["layer"]
        layer.load_sequences(s["T"], s["Tmin"], s["pat"])
        layer.forward(s["w"], s["x"], s["y"])
        layer.backward(s["w"], s["x"], s["y"], s["dy"], s["dx"], s["dw"])
        return s["y"], s["dx"], s["dw"]
    b2lstm.matrix_multiply(s["C"], c["m"], s["A"], s["lda"], c["ta"], s["B"], s["ldb"], c["tb"], c["m"], c["n"], c["k"])
    return s["C"]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------
def work(case):
    """flops of the dense products on the real frames (a fused multiply-add is two); bytes of inputs, targets, outputs, weights"""
    c = case
    if c["kind"] == "gemm":
        return {"bytes": 4.0 * (c["m"] * c["k"] + c["k"] * c["n"] + c["m"] * c["n"]), "flops": 2.0 * c["m"] * c["n"] * c["k"]}
    n = int(_lengths(c, c.get("nseq", c["P"])).sum())
    D = 2 if c["bi"] else 1
    ls = c["units"] * D
    rec_w = lambda prev: ls * (4 * (prev + 1) + 4 * c["units"] + 3)  # noqa: E731
    if c["kind"] == "layer":
        w = rec_w(c["in"])
        proj, rec = 8.0 * ls * c["in"], 8.0 * ls * c["units"]
        return {"bytes": 4.0 * (n * (2 * c["in"] + 2 * ls) + 2 * w), "flops": 3.0 * n * (proj + rec)}
    sizes = [c["in"]] + [c["ff_size"]] * c["ff"] + [ls] * c["rec"] + [c["out"]]
    fwd, first, weights = 0.0, 0.0, 0
    for i in range(1, len(sizes)):
        recurrent = c["ff"] < i <= c["ff"] + c["rec"]
        dense = (8.0 if recurrent else 2.0) * sizes[i] * sizes[i - 1]
        fwd += dense + (8.0 * ls * c["units"] if recurrent else 0.0)
        weights += rec_w(sizes[i - 1]) if recurrent else sizes[i] * (sizes[i - 1] + 1)
        if i == 1:
            first = dense     # nobody needs the error of the input
    data = n * (c["in"] + 2 * c["out"])
    if c["kind"] == "infer":
        return {"bytes": 4.0 * (data + weights), "flops": n * fwd}
    # weights, gradients and momentum: read and written at the update
    steps = -(-c["nseq"] // c["P"]) if c["kind"] == "epoch" else 1
    return {"bytes": 4.0 * (data + 5 * weights * steps), "flops": n * (3.0 * fwd - first)}


def tolerance(case):
    """fp32 throughout, sums of up to some 10^5 terms and chains of up to thousands of dependent steps in between; two orders of
    summation differ by a few 1e-6 of a tensor's norm on outputs and gradients, single small entries by more."""
    if case["kind"] == "gemm":
        return {"rel": 2e-6, "max": 2e-5}
    return {"rel": 3e-5, "max": 2e-3}
