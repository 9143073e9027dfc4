"""Performance cases of the attention path: what programs have this library do, as data.

A case describes one step through the public entry points (boat_b200.host over the C API):

  kind     "layer"  forward (and backward, update) of one attention layer
           "graph"  x + attention(x) recorded and differentiated through variables
           "block"  training step of a pre-LN encoder block, mean-squared-error loss
  step     "forward"        inference
           "backward"       forward and backward to dq, dk, dv and all parameter gradients
           "sgd" / "adam"   forward, mean-squared-error gradient, backward, update
  B S d nh causal           the problem: batch, sequence, model width, heads
  dtype    "fp32" (exact, the default arithmetic of FP32 tensors), "tf32", "bf16"
  place    "cuda" or "host": where the program's tensors and the layer's parameters live
  inputs   1: query, key and value are one tensor (self-attention), 3: three tensors

Inputs follow the benchmark's distributions: X ~ N(0,1), W ~ N(0, 1/sqrt(d)) (0.02 in the block), upstream
gradient or target ~ N(0,1), biases ~ N(0, 0.1).
"""
import ctypes as C
import math

import numpy as np
import torch

import boat_b200
from boat_b200 import capi
from boat_b200.host import Adam, Attention, EncoderBlock, Tensor, Variable, lincomb


def _case(name, kind, step, B, S, d, nh, causal, dtype, place="cuda", inputs=1):
    return dict(name=name, kind=kind, step=step, B=B, S=S, d=d, nh=nh, causal=causal, dtype=dtype, place=place, inputs=inputs)


def listed():
    return [
        # the reference's own training test: a handful of tokens, host tensors, SGD; all latency
        _case("first_program", "layer", "sgd", 2, 4, 32, 4, False, "fp32", place="host"),
        # the benchmark's smallest configuration (2 x 64 tokens of width 64), tensors kept on the GPU
        _case("small_fp32", "layer", "backward", 2, 64, 64, 4, False, "fp32"),
        # FP32 program written with variables: residual attention, causal, a length that fits no tile
        _case("graph_fp32_ragged", "graph", "backward", 4, 250, 256, 8, True, "fp32"),
        # FP32 storage on the tensor cores (benchmark configuration 2)
        _case("tf32_train", "layer", "backward", 8, 512, 512, 8, False, "tf32"),
        # one short prompt: inference latency
        _case("short_prompt", "layer", "forward", 1, 128, 1024, 16, True, "bf16"),
        # long prompts, head size 128: inference throughput
        _case("long_prompt", "layer", "forward", 2, 4096, 2048, 16, True, "bf16"),
        # a batch of documents cut at a length that is no multiple of a tile, key and value from elsewhere
        _case("ragged_train", "layer", "backward", 8, 1000, 1024, 16, True, "bf16", inputs=3),
        # benchmark configuration 3 with the Adam step behind it
        _case("adam_train", "layer", "adam", 16, 2048, 1024, 16, True, "bf16"),
        # benchmark configuration 4: long sequences, head size 128 - the largest single-GPU step
        _case("long_train", "layer", "backward", 4, 8192, 2048, 16, True, "bf16"),
        # encoder block on a small ragged batch
        _case("block_small", "block", "backward", 4, 333, 768, 12, False, "bf16"),
        # encoder block at benchmark configuration 5
        _case("block_train", "block", "backward", 32, 1024, 1024, 16, False, "bf16"),
        # tensors and layer on the host, as programs written for the reference keep them
        _case("host_train", "layer", "backward", 4, 2048, 1024, 16, True, "bf16", place="host"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A sequence length: half of them whole 128-row tiles, half anything."""
    s = _log_int(rng, lo, hi)
    return max(128, s // 128 * 128) if rng.random() < 0.5 else s


def draw(rng):
    what = rng.choice(["small", "fp32", "tf32", "bf16", "bf16", "bf16", "block", "host"])
    causal = rng.random() < 0.6
    if what == "small":
        # test-sized programs: host or CUDA tensors, widths and lengths of the tests
        hs, nh, S = rng.choice([8, 16, 32]), rng.choice([1, 2, 4, 8]), _log_int(rng, 4, 100)
        place = rng.choice(["host", "cuda"])
        return _nameless("layer", rng.choice(["sgd", "backward"]), rng.randint(1, 8), S, hs * nh, nh, causal, "fp32", place,
                         rng.choice([1, 3]))
    if what == "fp32":
        hs, nh = rng.choice([16, 32, 64]), rng.choice([2, 4, 8])
        S = _length(rng, 32, 1024)
        B = rng.randint(1, max(1, min(16, 4096 // S)))
        kind = rng.choice(["graph", "layer"])
        return _nameless(kind, "backward", B, S, hs * nh, nh, causal, "fp32", "cuda", 1 if kind == "graph" else rng.choice([1, 3]))
    if what == "tf32":
        nh, S = rng.choice([4, 8, 16]), _length(rng, 64, 1024)
        return _nameless("layer", "backward", rng.randint(1, max(1, min(16, 8192 // S))), S, 64 * nh, nh, causal, "tf32", "cuda", 1)
    if what == "bf16":
        step = rng.choice(["forward", "backward", "backward", "adam"])
        hs, nh = rng.choice([64, 128]), rng.choice([8, 12, 16])
        S = _length(rng, 64, 8192)
        if S % 128:                                       # batches of shorter, uneven texts
            S = min(S, _log_int(rng, 64, 3000))
        T = 16384 if S % 128 == 0 else 8192
        return _nameless("layer", step, rng.randint(1, max(1, min(16, T // S))), S, hs * nh, nh, causal, "bf16", "cuda",
                         1 if step == "adam" else rng.choice([1, 1, 3]))
    if what == "block":
        nh, S = rng.choice([4, 8, 12, 16]), _length(rng, 100, 2048)
        return _nameless("block", "backward", rng.randint(1, max(1, min(32, 8192 // S))), S, 64 * nh, nh, causal, "bf16", "cuda", 1)
    nh, S = rng.choice([8, 16]), _length(rng, 128, 2048)
    return _nameless("layer", "backward", rng.randint(1, max(1, min(8, 8192 // S))), S, 64 * nh, nh, causal, "bf16", "host", 1)


def _nameless(*a):
    c = _case("", *a)
    del c["name"]
    return c


# ---- tensors -------------------------------------------------------------------------------------------------

def _boat(t, bf16, device):
    """A boat tensor on `device` with the values of the FP32 torch tensor `t` (on the GPU)."""
    src = t.to(torch.bfloat16) if bf16 else t
    dtype = capi.DTYPE_BFLOAT16 if bf16 else capi.DTYPE_FLOAT32
    out = Tensor.create(tuple(t.shape), dtype, device)
    _fill(out, src)
    return out


def _fill(tensor, src):
    """Overwrite a boat tensor with the bytes of a torch tensor of the same storage type."""
    host = tensor.device == capi.DEVICE_CPU
    src = (src.cpu() if host else src).contiguous()
    here = capi.DEVICE_CPU if host else capi.DEVICE_CUDA
    assert src.nbytes == tensor.nbytes
    torch.cuda.current_stream().synchronize()
    capi.load().boat_memory_copy(tensor.data_ptr, C.c_void_p(src.data_ptr()), src.nbytes, here, here)


class _Memory:
    """Array interface over memory that `owner` keeps alive."""

    def __init__(self, ptr, shape, typestr, cuda, owner):
        desc = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}
        self.owner = owner
        if cuda:
            self.__cuda_array_interface__ = desc
        else:
            self.__array_interface__ = desc


def _torch(ptr, shape, bf16, cuda, owner):
    m = _Memory(ptr, shape, "<i2" if bf16 else "<f4", cuda, owner)
    t = torch.as_tensor(m, device="cuda") if cuda else torch.from_numpy(np.asarray(m))
    return t.view(torch.bfloat16) if bf16 else t


def _result(tensor, shape, bf16, cuda):
    """The caller's view of a result tensor: no copy."""
    return _torch(tensor.data_ptr, shape, bf16, cuda, tensor)


def _param_view(tensor, owner):
    return _torch(tensor.data_ptr, tensor.shape, False, tensor.device == capi.DEVICE_CUDA, owner)


def _bucket(layer, cuda):
    """The layer's parameter gradients: one FP32 array dWq dWk dWv dWo dbq dbk dbv dbo."""
    p, n = C.POINTER(C.c_float)(), C.c_size_t()
    capi.load().boat_attention_grad_bucket(layer.h, C.byref(p), C.byref(n))
    return _torch(C.cast(p, C.c_void_p).value, (n.value,), False, cuda, layer)


# ---- one step ------------------------------------------------------------------------------------------------

class _LayerStep:
    def __init__(self, c, normal):
        self.c = c
        self.cuda = c["place"] == "cuda"
        self.bf16 = c["dtype"] == "bf16"
        self.shape = (c["B"], c["S"], c["d"])
        d, device = c["d"], capi.DEVICE_CUDA if self.cuda else capi.DEVICE_CPU
        self.layer = layer = Attention(d, c["nh"], causal=c["causal"])
        if self.cuda:
            layer.to_device(device)
        for n in Attention.PARAMS:
            _fill(layer.param(n), normal(d, d) / math.sqrt(d) if n.startswith("weight") else normal(d) * 0.1)
        if c["dtype"] == "tf32":
            layer.set_precision(capi.MMA_TF32)
        self.x = [_boat(normal(*self.shape), self.bf16, device) for _ in range(c["inputs"])] * (3 // c["inputs"])
        self.dout = self.target = self.opt = self.params = self.grads = None
        if c["step"] in ("sgd", "adam"):
            self.target = _boat(normal(*self.shape), self.bf16, device)
            self.params = [_param_view(layer.param(n), layer) for n in Attention.PARAMS]
        elif c["step"] == "backward":
            self.dout = _boat(normal(*self.shape), self.bf16, device)
        if c["step"] == "adam":
            self.opt = Adam(1e-4)
            self.opt.add_attention(layer)

    def run(self):
        c = self.c
        if c["kind"] == "graph":
            x = Variable(self.x[0])
            r = x.attention(self.layer) + x
            r.backward(self.dout)
            out, gin = r.data, [x.grad]
            owners = (r, x)
        else:
            out = self.layer.forward(*self.x)
            if c["step"] == "forward":
                return [_result(out, self.shape, self.bf16, self.cuda)]
            dout, gin = self.dout, None
            if self.target is not None:
                n = 2.0 / (c["B"] * c["S"] * c["d"])
                if self.cuda:
                    dout = lincomb(out, n, self.target, -n)
                else:                                    # the host program computes its loss gradient itself
                    dout = Tensor.create(self.shape)
                    dout.host_view()[...] = (out.host_view() - self.target.host_view()) * n
            gin = self.layer.backward(dout)
            if c["step"] == "adam":
                self.opt.step()
            elif c["step"] == "sgd":
                self.layer.update(0.1)
            owners = None
        if self.grads is None:
            self.grads = _bucket(self.layer, self.cuda)
        res = [_torch(t.data_ptr, self.shape, self.bf16, self.cuda, owners or t) for t in (out, *gin)]
        return res + [self.grads] + (self.params or [])


class _BlockStep:
    def __init__(self, c, normal):
        self.c, d = c, c["d"]
        lib = capi.load()
        self.block = b = EncoderBlock(d, c["nh"], causal=c["causal"])
        self.dense = [Tensor(f(l.h), own=False) for l in (b.fc1, b.fc2)
                      for f in (lib.boat_dense_layer_get_weight, lib.boat_dense_layer_get_bias)]
        for t in self.dense:
            _fill(t, normal(*t.shape) * 0.02)
        for n in Attention.PARAMS:
            t = b.attn.param(n)
            _fill(t, normal(*t.shape) * 0.02)
        for l in (b.ln1, b.ln2):
            _fill(Tensor(lib.boat_layernorm_get_weight(l.h), own=False), 1.0 + 0.1 * normal(d))
            _fill(Tensor(lib.boat_layernorm_get_bias(l.h), own=False), 0.1 * normal(d))
        self.shape = (c["B"], c["S"], d)
        self.x, self.target = (_boat(normal(*self.shape), True, capi.DEVICE_CUDA) for _ in range(2))
        self.grads = None

    def run(self):
        b, lib = self.block, capi.load()
        b.zero_dense_grads()
        out, dx = b.step(self.x, self.target)
        if self.grads is None:
            ts = [f(l.h) for l in (b.fc1, b.fc2) for f in (lib.boat_dense_layer_get_grad_weight, lib.boat_dense_layer_get_grad_bias)]
            ts += [f(l.h) for l in (b.ln1, b.ln2) for f in (lib.boat_layernorm_get_grad_weight, lib.boat_layernorm_get_grad_bias)]
            self.grads = [_param_view(Tensor(t, own=False), b) for t in ts] + [_bucket(b.attn, True)]
        return [_result(out, self.shape, True, True), _result(dx, self.shape, True, True)] + self.grads


# ---- the interface -------------------------------------------------------------------------------------------

def prepare(case, seed):
    lib = boat_b200.load()
    if lib.boat_cuda_init(0):
        raise RuntimeError(lib.boat_cuda_last_error())
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    return (_BlockStep if case["kind"] == "block" else _LayerStep)(case, normal)


def run(state):
    return state.run()


def work(case):
    """Each input, parameter and result once; FLOPs of the products (nothing recomputed, masked half not counted)."""
    B, S, d, T = case["B"], case["S"], case["d"], case["B"] * case["S"]
    es = 2 if case["dtype"] == "bf16" else 4
    seen = 0.5 * (S + 1) / S if case["causal"] else 1.0
    act, par = T * d * es, 4 * (4 * d * d + 4 * d)
    if case["step"] == "forward":
        return {"bytes": (case["inputs"] + 1) * act + par, "flops": 8.0 * T * d * d + 4.0 * seen * B * S * S * d}
    flops = 24.0 * T * d * d + 12.0 * seen * B * S * S * d
    if case["kind"] == "block":                          # x, target, out, dx; parameters read, gradients written
        par = 4 * (12 * d * d + 13 * d)
        return {"bytes": 4 * act + 2 * par, "flops": flops + 48.0 * T * d * d}
    results = 2 if case["kind"] == "graph" else 4        # out and dx, or out and dq, dk, dv
    nbytes = (case["inputs"] + 1 + results) * act + 2 * par
    if case["step"] == "sgd":
        nbytes += par
    elif case["step"] == "adam":                         # weights written, both moments read and written
        nbytes += 5 * par
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "block":                          # a dozen BF16 roundings between input and gradient
        return {"rel": 2e-2}
    return {"rel": {"fp32": 1e-5, "tf32": 2e-3, "bf16": 1e-2}[case["dtype"]]}
