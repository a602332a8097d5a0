"""Parameters that change between calls: written through ``p.data`` (no version counter moves), given new storage, replaced;
and what a generation keeps while it runs and after it."""
import copy
import gc

import pytest
import torch

from _util import rel_l2

pytestmark = pytest.mark.gpu


def _block(M, cplx=False, dim=64, chunk=64, **kw):
    torch.manual_seed(11)
    args = dict(efficient_attn=True, rel_pos_bias='rotary')
    args.update(kw)
    blk = M.MovingAverageGatedAttention(dim, 64, 2 * dim, 16, chunk_size=chunk, moving_layer='cema' if cplx else 'ema',
                                        moving_act='silu', **args)
    return _other(blk).cuda().bfloat16().eval()


def _other(module, seed=12):
    """New values for every parameter, written behind autograd's back."""
    gen = torch.Generator().manual_seed(seed)
    for p in module.parameters():
        p.data.copy_((torch.randn(p.shape, generator=gen) * (0.5 if p.dim() != 2 else 0.1)).to(p.device))
    return module


def _fresh(module):
    """The module with its present parameters and nothing else."""
    new = copy.deepcopy(module)
    for m in new.modules():
        for name in ("_coeffs", "_decode_cache", "_step_plan", "_block_plan", "_qk_fp32", "_prep"):
            if m.__dict__.get(name) is not None:
                m.__dict__[name] = None
    return new


def _generate(blk, x, inc=None):
    inc = {} if inc is None else inc
    return torch.cat([blk(x[:, :5].contiguous(), incremental_state=inc)[0]]
                     + [blk(x[:, t:t + 1].contiguous(), incremental_state=inc)[0] for t in range(5, x.size(1))], 1)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("call", ["block", "generate", "norm_ema", "step"])
def test_writes_between_evaluations(cplx, call):
    """Evaluate, train with an optimiser that writes through p.data, evaluate again."""
    import fairseq_apollo_b200 as M
    blk = _block(M, cplx)
    x = torch.randn(2, 12, 64, device="cuda").bfloat16()

    def run(b):
        with torch.no_grad():
            if call == "block":
                return b(x)[0]
            if call == "generate":
                return _generate(b, x)
            if call == "norm_ema":
                return torch.cat(M.timestep_norm_ema(b.norm, b.move, x, None, {}, "silu", True))
            inc = {}
            return torch.cat([M.timestep_norm_ema(b.norm, b.move, x[:, t:t + 1].contiguous(), None, inc) for t in range(3)])

    first = run(blk)
    blk.train()
    _other(blk, 13)
    blk.eval()
    second = run(blk)
    assert torch.equal(second, run(_fresh(blk)))
    assert rel_l2(second, first) > 0.1


@pytest.mark.parametrize("cplx", [False, True])
def test_query_key_affine_and_norm_are_read_on_each_call(cplx):
    """Without train() in between: the block's own affine parameters are read when they are used."""
    import fairseq_apollo_b200 as M
    blk = _block(M, cplx)
    x = torch.randn(2, 64, 64, device="cuda").bfloat16()
    with torch.no_grad():
        blk(x)
        own = [blk.gamma, blk.beta] + ([blk.norm.weight] if cplx else [])
        for p in own:
            p.data.mul_(-1.5).add_(0.25)
        assert torch.equal(blk(x)[0], _fresh(blk)(x)[0])


@pytest.mark.parametrize("how", ["data", "moved", "assigned", "in place"])
def test_storage_replaced_during_a_generation(how):
    import fairseq_apollo_b200 as M
    blk = _block(M)
    x = torch.randn(2, 8, 64, device="cuda").bfloat16()
    ref = copy.deepcopy(blk).float()
    a, b = {}, {}
    got, want = [], []
    with torch.no_grad():
        for t in range(8):
            if t == 4:
                for m in (blk, ref):
                    if how == "data":
                        for p in m.parameters():
                            p.data = p.data.clone() * 1.5
                    elif how == "moved":
                        for p in m.parameters():
                            p.mul_(1.5)
                        m.cpu()
                        m.cuda()
                    elif how == "assigned":
                        m.v_proj.weight = torch.nn.Parameter(m.v_proj.weight * 1.5)
                        m.h_proj = copy.deepcopy(m.h_proj)
                    else:
                        m.v_proj.weight.mul_(1.5)
                junk = [torch.full_like(p, float("nan")) for p in blk.parameters()]   # (takes what was given back)
            got.append(blk(x[:, t:t + 1].contiguous(), incremental_state=a)[0])
            want.append(ref(x[:, t:t + 1].float().contiguous(), incremental_state=b)[0])
    del junk
    assert rel_l2(torch.cat(got, 1).float(), torch.cat(want, 1)) < 2e-2


def test_generation_gives_its_buffers_back():
    import fairseq_apollo_b200 as M
    blk = _block(M, chunk=1024)
    x = torch.randn(8, 8, 64, device="cuda").bfloat16()
    with torch.no_grad():
        _generate(blk, x)
        gc.collect()
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        inc = {}
        _generate(blk, x, inc)
        assert torch.cuda.memory_allocated() > before
        del inc
        assert torch.cuda.memory_allocated() - before < 1 << 16


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_two_generations_in_turn(dtype):
    """Two requests answered token by token in turn: each as by itself, and neither sets the other's step up again."""
    import fairseq_apollo_b200 as M
    blk = _block(M).to(dtype)
    xs = [torch.randn(2, 40, 64, device="cuda").to(dtype) for _ in range(2)]
    with torch.no_grad():
        want = [_generate(blk, x) for x in xs]
        incs = [{}, {}]
        got = [[blk(x[:, :5].contiguous(), incremental_state=i)[0]] for x, i in zip(xs, incs)]
        for t in range(5, 40):
            before = M.launch_count()
            for k in range(2):
                got[k].append(blk(xs[k][:, t:t + 1].contiguous(), incremental_state=incs[k])[0])
            if t > 5:
                assert M.launch_count() - before == 10
    for k in range(2):
        assert torch.equal(torch.cat(got[k], 1), want[k])


def test_copies_and_files_of_a_block_in_the_middle_of_a_generation(tmp_path):
    """A copied or loaded block and state go on as the original does; a state's file holds tensors alone."""
    import fairseq_apollo_b200 as M
    blk = _block(M)
    x = torch.randn(2, 12, 64, device="cuda").bfloat16()
    with torch.no_grad():
        want = _generate(blk, x)[:, 8:]
        inc = {}
        _generate(blk, x[:, :8], inc)
        torch.save(inc, tmp_path / "state.pt")
        torch.save(blk, tmp_path / "block.pt")
        copies = [(copy.deepcopy(blk), copy.deepcopy(inc)),
                  (torch.load(tmp_path / "block.pt", weights_only=False), torch.load(tmp_path / "state.pt", weights_only=True)),
                  (blk, {k: {n: t if t is None else t.clone() for n, t in v.items()} for k, v in inc.items()}), (blk, inc)]
        for b, i in copies:
            got = torch.cat([b(x[:, t:t + 1].contiguous(), incremental_state=i)[0] for t in range(8, 12)], 1)
            assert torch.equal(got, want)


@pytest.mark.parametrize("shift", [1, 4])
def test_token_at_any_address(shift):
    """A token that is a slice of a larger tensor, aligned to its elements only."""
    import fairseq_apollo_b200 as M
    blk = _block(M)
    x = torch.randn(2, 12, 64, device="cuda").bfloat16()
    with torch.no_grad():
        want = _generate(blk, x)
        inc = {}
        got = [blk(x[:, :5].contiguous(), incremental_state=inc)[0]]
        for t in range(5, 12):
            buf = torch.empty(2 * 64 + 8, device="cuda", dtype=x.dtype)
            tok = buf[shift:shift + 128].view(2, 1, 64)
            tok.copy_(x[:, t:t + 1])
            got.append(blk(tok, incremental_state=inc)[0])
    assert torch.equal(torch.cat(got, 1), want)


def test_chunk_is_laid_out_as_it_fills():
    """Buffers for at most 256 positions, or twice those there are; tokens across the doublings as without a chunk's end."""
    import fairseq_apollo_b200 as M
    blk = _block(M, chunk=4096)
    x = torch.randn(8, 600, 64, device="cuda").bfloat16()
    with torch.no_grad():
        gc.collect()
        _generate(blk, x[:, :8])
        before = torch.cuda.memory_allocated()
        inc = {}
        got = [_generate(blk, x[:, :8], inc)]
        assert torch.cuda.memory_allocated() - before < 8 * 300 * (64 + 64 + 128) * 2
        got += [blk(x[:, t:t + 1].contiguous(), incremental_state=inc)[0] for t in range(8, 600)]
        want = blk(x)[0]
    assert rel_l2(torch.cat(got, 1), want) < 1e-2


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("length", [1, 24])
def test_graph_outlives_what_a_layer_keeps(cplx, length):
    """A captured call replayed after another generation and a change of mode, with what they gave back taken by others."""
    import fairseq_apollo_b200 as M
    blk = _block(M, cplx)
    x = torch.randn(2, length, 64, device="cuda").bfloat16()

    def call(inc):
        return M.timestep_norm_ema(blk.norm, blk.move, x, None, inc, "silu", True)

    with torch.no_grad():
        want, inc = {}, {}
        for _ in range(2):
            call(want)
            call(inc)
        state = {key: dict(own) for key, own in inc.items()}   # (what the graph starts from is the caller's to keep)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = call(inc)
        for _ in range(2):
            call({})
        blk.train()
        blk.eval()
        gc.collect()
        junk = [torch.full((n,), float("nan"), device="cuda") for n in (16, 64, 128, 1024, 2048, 4096) for _ in range(16)]
        graph.replay()
        ref = call(want)
    torch.cuda.synchronize()
    del junk, state
    for a, b in zip(got, ref):
        assert torch.equal(a, b)
    for name in want:
        for key, t in want[name].items():
            assert torch.equal(inc[name][key], t), key


def test_what_a_graph_reads_goes_with_the_state():
    import fairseq_apollo_b200 as M
    blk = _block(M)
    x = torch.randn(2, 1, 64, device="cuda").bfloat16()
    with torch.no_grad():
        M.timestep_norm_ema(blk.norm, blk.move, x, None, {})
        gc.collect()
        before = torch.cuda.memory_allocated()
        inc = {}
        M.timestep_norm_ema(blk.norm, blk.move, x, None, inc)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            M.timestep_norm_ema(blk.norm, blk.move, x, None, inc)
        M.timestep_norm_ema(blk.norm, blk.move, x, None, {})
        held = torch.cuda.memory_allocated()
        graph.reset()
        del graph, inc
        gc.collect()
        assert torch.cuda.memory_allocated() < held and torch.cuda.memory_allocated() <= before
