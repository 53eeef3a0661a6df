"""GPU parity at the sizes where a kernel's split or a rule of the dispatch changes: edges of tiles, remainders, the smallest
and largest of a range. The walk generator bit-exactly and the loss + gradient against the oracle, as in the other suites."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import multigputrainmlp_b200 as mgt  # noqa: E402
from helpers import rel_l2  # noqa: E402
from oracle import MlpShape  # noqa: E402
from oracle.binding import WALK_META_DTYPE  # noqa: E402

DEV = "cuda:0"


def random_puzzle(state_len, move_count, seed):
    """Random permutations (they do not commute, so the order of the moves shows) on `state_len` positions."""
    rng = np.random.default_rng(seed)
    moves = np.zeros((18, 80), np.uint8)
    for i in range(move_count):
        moves[i, :state_len] = rng.permutation(state_len)
    target = np.zeros(80, np.uint8)
    target[:state_len] = np.arange(state_len)
    return moves, target


# samples around a CTA's 32 and the step to 128 (4 736), depths around a drawing round's 32 moves, record lengths that end inside a word
@pytest.mark.parametrize("n,k_min,k_max,state_len,move_count", [(1, 1, 1, 72, 18), (31, 1, 2, 72, 18), (32, 31, 32, 72, 18), (33, 32, 33, 70, 18),
                                                                 (4737, 1, 29, 72, 18),
                                                                 (200, 1, 64, 71, 3), (130, 60, 65, 17, 2), (100, 90, 200, 72, 18)])
def test_walk_rounds_and_edges(oracle, n, k_min, k_max, state_len, move_count):
    moves, target = random_puzzle(state_len, move_count, n)
    d_states = torch.full((n, 80), 255, dtype=torch.uint8, device=DEV)
    labels, meta = torch.zeros(n, device=DEV), torch.zeros(n, 16, dtype=torch.uint8, device=DEV)
    cfg = mgt.RandomWalkKernelConfig(n, k_min, k_max, move_count, state_len, 80)
    assert mgt.launch_random_walk_kernel(cfg, 77, 1, 5, 3, torch.from_numpy(moves).to(DEV), torch.from_numpy(target).to(DEV), d_states, labels, meta) == 0
    st, want, depth, want_meta = oracle.random_walks(moves, target, seed=77, epoch=1, step=5, rank=3, k_min=k_min, k_max=k_max, samples=n,
                                                     move_count=move_count, state_len=state_len)
    assert st == 0
    assert np.array_equal(d_states.cpu().numpy(), want) and np.array_equal(labels.cpu().numpy(), depth)
    assert np.array_equal(meta.cpu().numpy().view(WALK_META_DTYPE).reshape(-1), want_meta)


def loss_grad_case(oracle, dims, n, *, seed=1, scale=0.03, mirror=True, options=None, flags=(True, True), tol=1e-3, section_tol=3e-3, forks=None, slices=None):
    """One loss + gradient launch on a walk batch against the oracle's model of the same data flow, whole and by section. The last
    of four calls has a callback, which keeps all work on the caller's stream; the first three may use a second one (`forks`: have to, may not).
    slices: the oracle, which adds the samples one after the other, gets that many at a time and its results are added in double."""
    shape = MlpShape(*dims)
    length, values = shape.state_len, shape.state_value_pad
    moves, target = random_puzzle(length, 18, seed)
    target[:length] = np.arange(length) * values // length
    _, states, depth, _ = oracle.random_walks(moves, target, seed=seed, epoch=0, step=0, rank=0, k_min=1, k_max=29, samples=n, state_len=length)
    labels = np.ascontiguousarray(np.repeat(depth.reshape(-1, 1), shape.output_dim, axis=1).astype(np.float32))
    w = (np.random.default_rng(seed).standard_normal(shape.param_count) * scale).astype(np.float32)
    c = mgt.CudaMlpShape(*dims)
    half_ig, half_lin = flags
    engine = mgt.Engine(0)
    try:
        if options:
            assert engine.set_train_options(**options) == 0
        dw = torch.from_numpy(w).to(DEV)
        loss = torch.zeros(1, device=DEV)
        grad = torch.full((shape.param_count,), float("nan"), device=DEV)
        floats = mgt.mlp_loss_grad_workspace_floats(c, n, 1, half_ig, half_lin)
        ws = torch.full((floats,), float("nan"), device=DEV)
        results = []
        for callback in (None, None, None, lambda *a: 0):  # the same call again must give the same bits, whatever the library keeps between calls
            grad.fill_(float("nan"))
            before = engine.launch_count
            st = engine.launch_mlp_loss_grad(c, dw, dw.half() if mirror else None, torch.from_numpy(states).to(DEV), torch.from_numpy(labels).to(DEV), n, loss, grad,
                                             ws, floats, use_half_input_grad=half_ig, use_half_linear=half_lin, gradient_ready=callback)
            assert st == 0 and engine.check()[0] == 0
            launches = engine.launch_count - before
            results.append((float(loss.item()), grad.cpu().numpy()))
        assert forks is None or engine.fork_count == (3 if forks else 0)
    finally:
        engine.close()
    for other in results[1:]:
        assert other[0] == results[0][0] and np.array_equal(other[1], results[0][1])
    got_loss, got = results[0]
    if options or flags == (False, True):
        st, want_loss, want, _ = oracle.loss_grad_ex(shape, w, states, labels, half_linear=half_lin, half_input_grad=half_ig, **(options or {}))
    elif half_lin:
        st, want_loss, want = oracle.loss_grad_mixed(shape, w, states, labels)
    elif slices:
        st, want_loss, want = 0, 0.0, np.zeros(shape.param_count)
        for lo in range(0, n, slices):
            some, some_loss, some_grad = oracle.loss_grad(shape, w, states[lo:lo + slices], labels[lo:lo + slices])
            share = min(slices, n - lo) / n
            st, want_loss, want = st | some, want_loss + share * some_loss, want + share * some_grad.astype(np.float64)
    else:
        st, want_loss, want = oracle.loss_grad(shape, w, states, labels)
    assert st == 0 and np.isfinite(got).all()
    assert abs(got_loss - want_loss) <= tol * abs(want_loss)
    assert rel_l2(got, want) <= tol, rel_l2(got, want)
    table = length * values * shape.hd1
    hidden = table + shape.hd1
    tower = hidden + shape.hd1 * shape.hd2 + shape.hd2
    head = shape.param_count - shape.hd2 * shape.output_dim - shape.output_dim
    for name, lo, hi in (("table", 0, table), ("input bias", table, hidden), ("hidden", hidden, tower), ("tower", tower, head), ("head", head, shape.param_count)):
        if hi > lo and np.abs(want[lo:hi]).max() > 0:
            assert rel_l2(got[lo:hi], want[lo:hi]) <= section_tol, (name, rel_l2(got[lo:hi], want[lo:hi]))
    return launches


# widths of the fused residual tower that are not multiples of its 32-column chunks, with and without the caller's fp16 copy
@pytest.mark.parametrize("hd2,n,mirror", [(8, 130, True), (31, 127, False), (33, 129, False), (72, 300, True), (200, 257, True), (250, 128, False), (255, 400, True)])
def test_residual_tower_widths(oracle, hd2, n, mirror):
    loss_grad_case(oracle, (72, 72, 48, hd2, 3, 1), n, mirror=mirror)


# fp32 linear layers: the three tile sizes of the products, K splits, sizes that are no multiples of four, several outputs
@pytest.mark.parametrize("dims,n", [((72, 72, 40, 24, 2, 1), 70), ((72, 72, 37, 19, 1, 1), 33), ((20, 6, 200, 136, 3, 1), 1500), ((72, 72, 132, 68, 2, 3), 517),
                                     ((30, 30, 64, 40, 0, 5), 300), ((12, 5, 516, 260, 1, 1), 9700)])
def test_fp32_linears_over_tiles(oracle, dims, n):
    loss_grad_case(oracle, dims, n, flags=(False, False), tol=1e-5, section_tol=2e-5)


# The fp32 tower as it is cut for different batches and widths: one warp of 32, 64, 128, 224 or 256 columns, up to four of 32 and of 64
# side by side and two of 128; stages of 8, 16 and 32; one round of the chip and more; ends of tiles, matrices that have to be padded. Blocks that
# hand their signs, the ring of weights and the column sums' two places on to one another. And layer by layer, the widths of 129 to 256
# too: with few samples, and where the products' tiles fill the chip better than another round of the tower's.
@pytest.mark.parametrize("hd2,n,blocks", [(4, 70, 3), (9, 64, 3), (40, 300, 3), (72, 301, 3), (117, 1021, 3), (60, 12001, 2), (128, 2999, 2), (136, 2600, 2), (200, 3301, 2), (5, 20001, 2), (96, 16390, 2),
                                          (16, 40001, 2), (160, 7001, 2), (224, 4201, 2), (224, 8201, 1), (250, 4100, 2), (250, 8190, 1), (136, 9500, 1), (200, 1021, 2), (250, 2499, 2), (224, 9501, 1), (301, 700, 2)])
def test_fp32_tower_cuts(oracle, hd2, n, blocks):
    loss_grad_case(oracle, (6, 4, 16, hd2, blocks, 1), n, flags=(False, False), tol=1e-5, section_tol=2e-5, slices=1000)


# ... and which widths and batches take it: a block more is then no launch more, else it is four products more
@pytest.mark.parametrize("hd2,n,fused", [(8, 33, True), (128, 70, True), (129, 2499, False), (129, 2500, True), (160, 9500, True), (160, 12000, False), (224, 8200, True), (224, 9500, False), (224, 20000, True),
                                         (256, 2500, True), (257, 2600, False)])
def test_fp32_tower_or_layers(hd2, n, fused):
    states, labels, loss = torch.zeros(n, 80, dtype=torch.uint8, device=DEV), torch.ones(n, device=DEV), torch.zeros(1, device=DEV)
    launches = []
    engine = mgt.Engine(0)
    try:
        for blocks in (1, 2):
            c = mgt.CudaMlpShape(4, 4, 16, hd2, blocks, 1)
            w, floats = torch.zeros(c.param_count, device=DEV), mgt.mlp_loss_grad_workspace_floats(c, n, 1, False, False)
            before = engine.launch_count
            assert engine.launch_mlp_loss_grad(c, w, None, states, labels, n, loss, torch.empty_like(w), torch.empty(floats, device=DEV), floats, use_half_input_grad=False,
                                               use_half_linear=False, gradient_ready=lambda *a: 0) == 0
            launches.append(engine.launch_count - before)
    finally:
        engine.close()
    assert launches[1] - launches[0] == (0 if fused else 4)


# A weight without bound behind a unit that no sample opens: its products with the samples are NaN before a ReLU that closes on
# them and before masks that are zero, so that all gradients are those of the same model with that weight 0. Nor may the rows of the tower's
# last tile that are no samples bring it into the bias gradients: there the unit would be open.
@pytest.mark.parametrize("hd2,n", [(24, 61), (128, 1003), (224, 4099)])
def test_fp32_tower_rows_past_the_batch(hd2, n):
    c = mgt.CudaMlpShape(6, 4, 16, hd2, 2, 1)
    rng = np.random.default_rng(hd2)
    w = (rng.standard_normal(c.param_count) * 0.03).astype(np.float32)
    hidden = 24 * 16 + 16
    w[hidden + 16 * hd2:hidden + 17 * hd2] = 1.0  # hidden bias: every activation positive
    first = hidden + 17 * hd2                     # W1_0, b1_0, W2_0, b2_0
    second = first + hd2 * hd2 + hd2
    w[first:first + hd2 * hd2].reshape(hd2, hd2)[:, 0] = -1.0
    w[first + hd2 * hd2] = 0.5                    # unit 0 of the first block: open where the activations are zero, and only there
    w[second + hd2 * hd2 + 3] = -1000.0           # unit 3 behind it: closed
    states = torch.from_numpy(rng.integers(0, 4, (n, 80), dtype=np.uint8)).to(DEV)
    labels, loss = torch.ones(n, device=DEV), torch.zeros(1, device=DEV)
    floats = mgt.mlp_loss_grad_workspace_floats(c, n, 1, False, False)
    ws = torch.empty(floats, device=DEV)
    grads = []
    engine = mgt.Engine(0)
    try:
        for value in (0.0, np.inf):
            w[second + 3] = value                 # from unit 0 to unit 3
            grad = torch.full((c.param_count,), float("nan"), device=DEV)
            assert engine.launch_mlp_loss_grad(c, torch.from_numpy(w).to(DEV), None, states, labels, n, loss, grad, ws, floats, use_half_input_grad=False,
                                               use_half_linear=False) == 0
            assert engine.check()[0] == 0
            grads.append(grad.cpu().numpy())
    finally:
        engine.close()
    assert np.isfinite(grads[0]).all() and np.array_equal(grads[1], grads[0])


def multiply_in_order(x, w):
    """x w in fp32, one multiply-add after the other along k (the product of two floats is exact in double)."""
    acc = np.zeros((x.shape[0], w.shape[1]), np.float32)
    x, w = x.astype(np.float64), w.astype(np.float64)
    for k in range(w.shape[0]):
        acc = (x[:, k:k + 1] * w[k] + acc).astype(np.float32)
    return acc


# The forward products of the fp32 path add in the order of k whatever their tile: another order opens or closes a ReLU here and
# there, and with it the path of a whole gradient. With a batch of one sample every activation can be read back to the bit: a
# weight's gradient is the rounded product of the activation below it and of its unit's bias gradient.
@pytest.mark.parametrize("dims", [(18, 6, 64, 48, 6, 1), (18, 6, 200, 33, 3, 1), (72, 72, 1032, 230, 2, 1), (5, 3, 17, 300, 1, 1), (5, 3, 16, 8, 1, 1)])
def test_fp32_forward_adds_in_order(oracle, dims):
    shape = MlpShape(*dims)
    length, values, h1, h2, blocks = dims[:5]
    c = mgt.CudaMlpShape(*dims)
    floats = mgt.mlp_loss_grad_workspace_floats(c, 1, 1, False, False)
    ws, loss, grad = torch.empty(floats, device=DEV), torch.zeros(1, device=DEV), torch.zeros(shape.param_count, device=DEV)
    std = [0.8 / length ** 0.5, 0.05, (2 / h1) ** 0.5, 0.05] + [(2 / h2) ** 0.5, 0.05, (2 / h2) ** 0.5, 0.02] * blocks + [h2 ** -0.5, 0.1]
    sizes = [(length * values, h1), (h1,), (h1, h2), (h2,)] + [(h2, h2), (h2,)] * (2 * blocks) + [(h2,), (1,)]

    def split(flat):
        ends = np.cumsum([int(np.prod(size)) for size in sizes])
        return [part.reshape(size) for part, size in zip(np.split(flat, ends[:-1]), sizes)]
    engine = mgt.Engine(0)
    try:
        for seed in range(4):
            moves, target = random_puzzle(length, 18, seed)
            target[:length] = np.arange(length) * values // length
            _, state, depth, _ = oracle.random_walks(moves, target, seed=seed, epoch=0, step=0, rank=0, k_min=1, k_max=29, samples=1, state_len=length)
            rng = np.random.default_rng(seed)
            w = np.concatenate([rng.standard_normal(int(np.prod(size))) * s for size, s in zip(sizes, std)]).astype(np.float32)
            st = engine.launch_mlp_loss_grad(c, torch.from_numpy(w).to(DEV), None, torch.from_numpy(state).to(DEV), torch.from_numpy(depth).to(DEV), 1, loss, grad, ws,
                                             floats, use_half_input_grad=False, use_half_linear=False)
            assert st == 0 and engine.check()[0] == 0
            part, g = split(w), split(grad.cpu().numpy())
            a = part[1][None].copy()
            for p in range(length):
                a += part[0][p * values + int(state[0, p])]
            a = np.maximum(a, np.float32(0))
            layers = [(a, 2)]
            x = np.maximum(multiply_in_order(a, part[2]) + part[3], np.float32(0))
            for b in range(4, 4 + 4 * blocks, 4):
                r = np.maximum(multiply_in_order(x, part[b]) + part[b + 1], np.float32(0))
                layers += [(x, b), (r, b + 2)]
                x = np.maximum((multiply_in_order(r, part[b + 2]) + part[b + 3]) + x, np.float32(0))
            layers.append((x, 4 + 4 * blocks))
            for act, i in layers:
                bias = g[i + 1]
                assert np.count_nonzero(act) and np.count_nonzero(bias)
                want = act[0] * bias[0] if i == 4 + 4 * blocks else act[0][:, None] * bias
                assert np.array_equal(g[i], want), (seed, i)
    finally:
        engine.close()


# fp32 table gradient behind fp16 linears: classes without samples, one class per position, many samples per class; its sort on the
# second stream (hd1 up to 256, up to 512 with 4 096 samples) and on the caller's
@pytest.mark.parametrize("dims,n,mirror", [((72, 72, 36, 40, 1, 1), 45, True), ((54, 6, 130, 64, 2, 1), 1000, True), ((16, 1, 33, 24, 1, 2), 257, False),
                                           ((20, 12, 256, 40, 2, 1), 4100, True), ((20, 12, 512, 24, 3, 1), 300, False), ((20, 12, 260, 24, 3, 1), 4100, True), ((20, 12, 516, 24, 3, 1), 300, True)])
def test_fp32_table_gradient(oracle, dims, n, mirror):
    loss_grad_case(oracle, dims, n, flags=(False, True), mirror=mirror)


# sums over partial results: lists up to, at and beyond what one launch takes, terms around the 32 lanes and the eight loads in
# flight, items that are no whole CTA and no whole quads; bit for bit in the documented order
@pytest.mark.parametrize("planes", [False, True])
@pytest.mark.parametrize("jobs,terms,items", [(1, 1, 1), (2, 33, 9), (12, 131, 40), (13, 9, 1028), (40, 160, 263)])
def test_sums_of_partial_results(planes, jobs, terms, items):
    src = np.random.default_rng(jobs).standard_normal((jobs, terms, items)).astype(np.float32)
    dst = torch.full((jobs * items,), float("nan"), device=DEV)
    engine = mgt.Engine(0)
    try:
        assert engine.debug_sums(torch.from_numpy(src).to(DEV), terms, items, jobs, planes, dst) == 0
    finally:
        engine.close()
    want = np.zeros((jobs, items), np.float32)
    for lane in range(1 if planes else min(32, terms)):
        part = np.zeros((jobs, items), np.float32)
        for t in range(lane, terms, 1 if planes else 32):
            part += src[:, t]
        want += part
    assert np.array_equal(dst.cpu().numpy().reshape(jobs, items), want)


# output head: the widths of its tile (16, 32, 64) and the per-sample form beyond them, tiles of 64 samples
@pytest.mark.parametrize("outputs,hd2,n", [(2, 16, 64), (16, 300, 65), (17, 40, 63), (32, 272, 200), (33, 24, 130), (64, 512, 70), (65, 48, 96)])
@pytest.mark.parametrize("cross_entropy", [False, True])
def test_output_head_widths(oracle, outputs, hd2, n, cross_entropy):
    dims = (72, 72, 48, hd2, 1, outputs)
    if cross_entropy and outputs < 29:
        pytest.skip("a class per depth")
    loss_grad_case(oracle, dims, n, options=dict(cross_entropy=True) if cross_entropy else None, tol=2e-3, section_tol=5e-3)


# four threads, an engine and a stream each, whose heads are one kernel with different amounts of shared memory
def test_output_heads_in_several_threads():
    failed = []

    def steps(hd2):
        c = mgt.CudaMlpShape(8, 8, 16, hd2, 0, 29)
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            w = torch.zeros(c.param_count, device=DEV)
            states, labels = torch.zeros(64, 80, dtype=torch.uint8, device=DEV), torch.ones(64 * 29, device=DEV)
            floats = mgt.mlp_loss_grad_workspace_floats(c, 64)
            ws, loss, grad = torch.empty(floats, device=DEV), torch.zeros(1, device=DEV), torch.zeros_like(w)
            engine = mgt.Engine(0)
            for _ in range(1500):
                status = engine.launch_mlp_loss_grad(c, w, None, states, labels, 64, loss, grad, ws, floats, stream=stream)
                if status != 0:
                    failed.append((hd2, status))
                    break
            stream.synchronize()
            engine.close()
    threads = [threading.Thread(target=steps, args=(hd2,)) for hd2 in (512, 224, 512, 224)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


# outputs around the limit of shared memory that a kernel gets without asking, counting the static array beside it
@pytest.mark.parametrize("outputs", [1000, 1030, 1600])
def test_many_outputs(oracle, outputs):
    loss_grad_case(oracle, (8, 8, 16, 24, 1, outputs), 70, tol=2e-3, section_tol=5e-3)


# embedding layer by gathering rows: samples around a CTA's 32, columns around its 64 and the vectors of eight, few classes, a
# single position, batches towards the rule's border
@pytest.mark.parametrize("dims,n,mirror", [((72, 72, 64, 16, 1, 1), 31, True), ((72, 72, 65, 24, 1, 1), 33, False), ((54, 6, 136, 32, 1, 1), 129, True), ((1, 3, 40, 8, 1, 1), 65, True),
                                            ((72, 72, 200, 40, 1, 1), 2100, True), ((30, 30, 1100, 48, 1, 1), 4200, True), ((7, 64, 4096, 16, 0, 1), 9000, True)])
@pytest.mark.parametrize("bf16", [False, True])
def test_embedding_forms(oracle, dims, n, mirror, bf16):
    if n > 4000 and bf16:
        pytest.skip("the oracle takes long; the form is the same")
    loss_grad_case(oracle, dims, n, mirror=mirror, options=dict(bf16=True) if bf16 else None, tol=8e-3 if bf16 else 1e-3, section_tol=2e-2 if bf16 else 3e-3)


# one-hot GEMMs for CTA pairs: ragged rows, columns and K on both sides, tiles shared by two pairs and whole ones; 64 classes and
# more (single places set and cleared), and few classes (rows written whole)
@pytest.mark.parametrize("dims,n", [((72, 72, 1000, 16, 0, 1), 9001), ((54, 6, 4090, 16, 0, 1), 9000)])
def test_one_hot_pairs(oracle, dims, n):
    loss_grad_case(oracle, dims, n)


# both forms of the embedding layer on the same small batches, whatever the rule would pick: table gradients of 110 tiles on 74
# pairs (stretches that share tiles), of few tiles (halves) and of whole tiles, few classes and 64 or more, ragged sizes, the
# weight gradients of the blocks beside the table gradient. The gathered gradient has one launch more, the sort.
@pytest.mark.parametrize("dims,n", [((72, 72, 2560, 24, 1, 1), 130), ((72, 72, 200, 24, 2, 1), 257), ((54, 6, 1030, 24, 1, 1), 300), ((20, 12, 130, 40, 1, 2), 70), ((30, 4, 130, 40, 1, 2), 70),
                                     ((1, 64, 40, 8, 1, 1), 65), ((7, 64, 4090, 16, 1, 1), 333)])
@pytest.mark.parametrize("bf16", [False, True])
def test_embedding_forms_on_one_batch(oracle, monkeypatch, dims, n, bf16):
    launches = {}
    for form in ("gather", "onehot"):
        monkeypatch.setenv("MGT_EMBEDDING_FORM", form)
        launches[form] = loss_grad_case(oracle, dims, n, scale=0.02, options=dict(bf16=True) if bf16 else None, tol=8e-3 if bf16 else 1e-3, section_tol=2e-2 if bf16 else 3e-3)
    assert launches["gather"] == launches["onehot"] + 1


# states that start anywhere: a caller's own array of 80-byte records has no alignment to keep
@pytest.mark.parametrize("half_lin", [True, False])
@pytest.mark.parametrize("form", ["gather", "onehot"])
def test_states_at_odd_addresses(oracle, monkeypatch, form, half_lin):
    monkeypatch.setenv("MGT_EMBEDDING_FORM", form)
    n, c = 333, mgt.CudaMlpShape(72, 72, 200, 24, 1, 1)
    moves, target = random_puzzle(72, 18, 1)
    _, states, depth, _ = oracle.random_walks(moves, target, seed=1, epoch=0, step=0, rank=0, k_min=1, k_max=29, samples=n)
    w = torch.from_numpy((np.random.default_rng(1).standard_normal(c.param_count) * 0.03).astype(np.float32)).to(DEV)
    floats = mgt.mlp_loss_grad_workspace_floats(c, n, 1, half_lin, half_lin)
    ws, loss, labels = torch.empty(floats, device=DEV), torch.zeros(1, device=DEV), torch.from_numpy(depth).to(DEV)
    grads = []
    engine = mgt.Engine(0)
    try:
        for offset in (0, 1, 2):
            buffer = torch.zeros(n * 80 + 16, dtype=torch.uint8, device=DEV)
            buffer[offset:offset + n * 80] = torch.from_numpy(states).to(DEV).ravel()
            grad = torch.full((c.param_count,), float("nan"), device=DEV)
            assert engine.launch_mlp_loss_grad(c, w, None, buffer[offset:], labels, n, loss, grad, ws, floats, use_half_input_grad=half_lin, use_half_linear=half_lin) == 0
            assert engine.check()[0] == 0
            grads.append(grad.cpu().numpy())
    finally:
        engine.close()
    assert np.isfinite(grads[0]).all() and np.array_equal(grads[0], grads[1]) and np.array_equal(grads[0], grads[2])


# residual tower for pairs of CTAs (hd2 above 256): unequal halves, a second half of one chunk, whole panels, ragged tiles
@pytest.mark.parametrize("hd2,n,mirror", [(257, 130, False), (264, 128, True), (320, 129, True), (390, 300, False), (512, 257, True)])
@pytest.mark.parametrize("bf16", [False, True])
def test_wide_residual_tower(oracle, hd2, n, mirror, bf16):
    loss_grad_case(oracle, (72, 72, 48, hd2, 3, 1), n, scale=0.02, mirror=mirror, options=dict(bf16=True) if bf16 else None, tol=8e-3 if bf16 else 1e-3,
                   section_tol=2e-2 if bf16 else 3e-3)


# The hidden layer's input gradient by TMA stores (more tiles than SMs): ragged last rows and columns, one to four K chunks
@pytest.mark.parametrize("hd1,hd2,n", [(1000, 64, 10001), (300, 129, 25700)])
def test_hidden_input_gradient_stores(oracle, monkeypatch, hd1, hd2, n):
    monkeypatch.setenv("MGT_EMBEDDING_FORM", "onehot")
    loss_grad_case(oracle, (8, 8, hd1, hd2, 1, 1), n, mirror=False)


# weight gradients on the second stream beside the table gradient, by gathering (its sort on that stream too) and by the one-hot
# product; the last call of a case runs on one stream and has to give the same bits
@pytest.mark.parametrize("dims,n", [((72, 72, 896, 40, 2, 1), 96), ((72, 72, 897, 40, 2, 1), 96), ((54, 6, 1024, 64, 1, 3), 513), ((72, 72, 1032, 33, 0, 1), 257)])
@pytest.mark.parametrize("form", ["gather", "onehot"])
def test_weight_gradients_beside_the_embedding_gradient(oracle, monkeypatch, dims, n, form):
    monkeypatch.setenv("MGT_EMBEDDING_FORM", form)
    loss_grad_case(oracle, dims, n, scale=0.02, forks=True)


# ... where that begins, by the number of blocks
@pytest.mark.parametrize("blocks,hd1,n,forks", [(0, 255, 256, False), (0, 256, 256, True), (1, 127, 128, False), (1, 128, 128, True), (2, 31, 66, False), (2, 32, 64, True), (3, 8, 64, True),
                                                (3, 8, 16385, False)])
def test_steps_that_fork(oracle, blocks, hd1, n, forks):
    loss_grad_case(oracle, (12, 6, hd1, 24, blocks, 1), n, forks=forks)


# Bias sums of the backward tower with two and three tiles to a CTA (or pair), whose products follow one another into the same
# tensor memory: the same bits every time, and the layer-by-layer path's sums up to fp16 roundings that fall the other way.
@pytest.mark.parametrize("hd2,n", [(64, 37965), (160, 37965), (256, 40000), (272, 19021), (512, 19021)])
def test_tower_bias_sums_over_tiles(oracle, monkeypatch, hd2, n):
    dims = (8, 8, 32, hd2, 3, 1)
    shape = MlpShape(*dims)
    moves, target = random_puzzle(8, 18, 3)
    _, states, depth, _ = oracle.random_walks(moves, target, seed=3, epoch=0, step=0, rank=0, k_min=1, k_max=29, samples=n, state_len=8)
    w = torch.from_numpy((np.random.default_rng(3).standard_normal(shape.param_count) * 0.05).astype(np.float32)).to(DEV)
    d_states, labels = torch.from_numpy(states).to(DEV), torch.from_numpy(depth).to(DEV)
    c = mgt.CudaMlpShape(*dims)
    floats = mgt.mlp_loss_grad_workspace_floats(c, n)
    ws, loss = torch.empty(floats, device=DEV), torch.zeros(1, device=DEV)
    grads = []
    for path in ("fused", "layered"):
        monkeypatch.setenv("MGT_RESIDUAL_PATH", path)
        engine = mgt.Engine(0)
        try:
            for _ in range(4 if path == "fused" else 1):
                grad = torch.full((shape.param_count,), float("nan"), device=DEV)
                assert engine.launch_mlp_loss_grad(c, w, w.half(), d_states, labels, n, loss, grad, ws, floats) == 0
                assert engine.check()[0] == 0
                grads.append(grad.cpu().numpy())
        finally:
            engine.close()
    for other in grads[1:4]:
        assert np.array_equal(other, grads[0])
    first = 64 * 32 + 32 + 32 * hd2 + hd2
    for layer in range(6):
        lo = first + layer * (hd2 * hd2 + hd2) + hd2 * hd2
        assert rel_l2(grads[0][lo:lo + hd2], grads[4][lo:lo + hd2]) <= 1e-3, layer


class SmallStep:
    """Loss + gradient of a batch that the library spreads over two streams, with scratch of its own. Every call has to have done so,
    unless it asks for one stream."""

    def __init__(self, engine, n=96, dims=(72, 72, 256, 40, 2, 1)):
        rng = np.random.default_rng(n)
        self.engine, self.n, self.shape = engine, n, mgt.CudaMlpShape(*dims)
        self.w = torch.from_numpy((rng.standard_normal(self.shape.param_count) * 0.03).astype(np.float32)).to(DEV)
        self.states = torch.from_numpy(rng.integers(0, 72, (n, 80), dtype=np.uint8)).to(DEV)
        self.labels, self.loss, self.grad = torch.ones(n, device=DEV), torch.zeros(1, device=DEV), torch.zeros_like(self.w)
        self.floats = mgt.mlp_loss_grad_workspace_floats(self.shape, n)
        self.ws = torch.empty(self.floats, device=DEV)
        torch.cuda.synchronize()

    def __call__(self, stream=None, one_stream=False, forks=1):
        before = self.engine.fork_count
        status = self.engine.launch_mlp_loss_grad(self.shape, self.w, None, self.states, self.labels, self.n, self.loss, self.grad, self.ws, self.floats, stream=stream,
                                                  gradient_ready=(lambda *a: 0) if one_stream else None)
        assert self.engine.fork_count - before == (0 if one_stream else forks)
        return status

    def result(self):
        torch.cuda.synchronize()
        assert self.engine.check()[0] == 0
        got = self.grad.cpu().numpy()
        self.grad.fill_(float("nan"))
        torch.cuda.synchronize()
        return got


@pytest.fixture
def small_step():
    engine = mgt.Engine(0)
    yield SmallStep(engine)
    torch.cuda.synchronize()
    engine.close()


# Kernels that begin before the one ahead of them has ended: the same training steps with the device idle before every call, and
# with foreign kernels between the calls, must end in the same bits.
@pytest.mark.parametrize("half,batch_norm", [(True, False), (False, False), (True, True)])
@pytest.mark.parametrize("n", [64, 1500])
def test_steps_back_to_back(half, batch_norm, n):
    shape = mgt.CudaMlpShape(72, 72, 256, 40, 2, 1)
    total = shape.param_count + (mgt.bn_param_count(shape) if batch_norm else 0)
    first = torch.from_numpy((np.random.default_rng(n).standard_normal(total) * 0.03).astype(np.float32)).to(DEV)
    moves, target = random_puzzle(72, 18, n)
    moves, target = torch.from_numpy(moves).to(DEV), torch.from_numpy(target).to(DEV)
    floats = mgt.mlp_loss_grad_workspace_floats(shape, n, 1, half, half, batch_norm=batch_norm)
    engine = mgt.Engine(0)
    results = []
    try:
        assert engine.set_train_options(batch_norm=batch_norm) == 0
        for between in ("idle", "nothing", "kernels"):
            w, m, v, grad = first.clone(), torch.zeros_like(first), torch.zeros_like(first), torch.zeros_like(first)
            w_half, loss, depth = w.half(), torch.zeros(1, device=DEV), torch.zeros(n, device=DEV)
            states, meta = torch.zeros(n, 80, dtype=torch.uint8, device=DEV), torch.zeros(n, 16, dtype=torch.uint8, device=DEV)
            ws = torch.full((floats,), float("nan"), device=DEV)

            def pause():
                if between == "idle":
                    torch.cuda.synchronize()
                elif between == "kernels":
                    w.mul_(1.0)
                    grad.add_(0.0)
            for step in range(6):
                assert mgt.launch_random_walk_kernel(mgt.RandomWalkKernelConfig(n, 1, 20), 5, 0, step, 0, moves, target, states, depth, meta) == 0
                pause()
                assert engine.launch_mlp_loss_grad(shape, w, w_half, states, depth, n, loss, grad, ws, floats, use_half_input_grad=half, use_half_linear=half) == 0
                pause()
                assert mgt.launch_adamw_kernel_with_half_mirror(mgt.AdamWKernelConfig(total, step + 1, 1e-3), w, w_half, grad, m, v) == 0
                pause()
            assert engine.check()[0] == 0
            results.append([t.cpu().numpy() for t in (w, m, v, loss, states)])
    finally:
        engine.close()
    for other in results[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(other, results[0]))


def test_steps_on_several_streams_do_not_wait_for_each_other(small_step):
    other = SmallStep(small_step.engine, 64)
    assert small_step(one_stream=True) == 0
    want = small_step.result()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for stream in streams:
        assert other(stream) == 0 and other.result() is not None  # (modules loaded, second streams made)
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(3 << 30)  # a second and a half
    assert other(streams[0]) == 0
    late = streams[0].record_event()
    assert small_step(streams[1]) == 0
    streams[1].synchronize()
    assert not late.query()
    assert np.array_equal(small_step.result(), want)
    for stream in [torch.cuda.Stream() for _ in range(7)]:  # more streams than the engine keeps second ones for
        assert small_step(stream) == 0
    assert np.array_equal(small_step.result(), want)


def test_step_beside_a_capture(small_step):
    assert small_step(one_stream=True) == 0
    want = small_step.result()
    other = SmallStep(small_step.engine, 64)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    assert small_step(stream) == 0 and other() == 0
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        assert small_step(stream) == 0 and small_step(stream) == 0
        free = torch.cuda.Stream()
        assert other(free) == 0  # eager, on another stream, with the capture open
        free.synchronize()
    assert np.isfinite(other.result()).all()
    small_step.result()
    graph.replay()
    assert np.array_equal(small_step.result(), want)


def test_two_captures_at_once(small_step):
    other = SmallStep(small_step.engine, 64)
    assert other(one_stream=True) == 0 and small_step(one_stream=True) == 0
    want_other, want = other.result(), small_step.result()
    streams, graphs = [torch.cuda.Stream() for _ in range(2)], [torch.cuda.CUDAGraph() for _ in range(2)]
    assert small_step(streams[0]) == 0 and other(streams[1]) == 0  # (second streams made)
    assert np.array_equal(small_step.result(), want) and np.array_equal(other.result(), want_other)
    with torch.cuda.stream(streams[0]):
        graphs[0].capture_begin(capture_error_mode="relaxed")
        assert small_step(streams[0]) == 0
    with torch.cuda.stream(streams[1]):
        graphs[1].capture_begin(capture_error_mode="relaxed")
        assert other(streams[1]) == 0
    for stream, graph in zip(streams, graphs):
        with torch.cuda.stream(stream):
            graph.capture_end()
    for graph in graphs:
        graph.replay()
    assert np.array_equal(small_step.result(), want) and np.array_equal(other.result(), want_other)


# Steps as a graph: kernels that begin before the one ahead of them has ended, behind forks and joins, and behind the memsets of a one-hot
# product with shared tiles and of the layered tower of batch normalisation. Two steps in a graph, replayed three times.
@pytest.mark.parametrize("dims,n,flags,form,batch_norm", [((72, 72, 256, 40, 2, 1), 1500, (True, True), "gather", False), ((72, 72, 2560, 24, 1, 1), 130, (True, True), "onehot", False),
                                                          ((72, 72, 256, 40, 2, 3), 300, (True, True), "gather", True), ((72, 72, 256, 300, 2, 1), 300, (True, True), "onehot", True),
                                                          ((72, 72, 256, 300, 2, 29), 300, (False, True), "gather", False), ((72, 72, 256, 40, 2, 1), 1000, (False, False), "gather", False)])
def test_captured_steps(monkeypatch, dims, n, flags, form, batch_norm):
    monkeypatch.setenv("MGT_EMBEDDING_FORM", form)
    c = mgt.CudaMlpShape(*dims)
    total = c.param_count + (mgt.bn_param_count(c) if batch_norm else 0)
    rng = np.random.default_rng(n)
    first = torch.from_numpy((rng.standard_normal(total) * 0.03).astype(np.float32)).to(DEV)
    states = torch.from_numpy(rng.integers(0, 72, (n, 80), dtype=np.uint8)).to(DEV)
    labels, loss, grad = torch.ones(n * dims[5], device=DEV), torch.zeros(1, device=DEV), torch.zeros(total, device=DEV)
    floats = mgt.mlp_loss_grad_workspace_floats(c, n, 1, *flags, batch_norm=batch_norm)
    w, m, v, ws = first.clone(), torch.zeros_like(first), torch.zeros_like(first), torch.full((floats,), float("nan"), device=DEV)
    stream, graph, engine = torch.cuda.Stream(), torch.cuda.CUDAGraph(), mgt.Engine(0)
    forks = 2 if flags[1] else 0

    def two_steps():
        for _ in range(2):
            assert engine.launch_mlp_loss_grad(c, w, None, states, labels, n, loss, grad, ws, floats, use_half_input_grad=flags[0], use_half_linear=flags[1], stream=stream) == 0
            assert mgt.launch_adamw_kernel(mgt.AdamWKernelConfig(total, 1, 1e-3), w, grad, m, v, stream=stream) == 0

    def finish():
        torch.cuda.synchronize()
        assert engine.check()[0] == 0
        result = [t.cpu().numpy() for t in (w, m, v, grad, loss)]
        for t, start in ((w, first), (m, 0.0), (v, 0.0), (grad, float("nan"))):
            t.copy_(start) if isinstance(start, torch.Tensor) else t.fill_(start)
        torch.cuda.synchronize()
        return result
    try:
        assert engine.set_train_options(batch_norm=batch_norm) == 0
        torch.cuda.synchronize()
        for _ in range(3):
            two_steps()
        want = finish()
        assert np.isfinite(want[0]).all() and engine.fork_count == 3 * forks
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            two_steps()
        assert engine.fork_count == 4 * forks
        for _ in range(3):
            graph.replay()
        assert all(np.array_equal(a, b) for a, b in zip(finish(), want))
    finally:
        engine.close()


def test_first_step_of_an_engine_under_capture():
    # no idle second stream is left and none is made during a capture: everything on the caller's stream
    holders = [SmallStep(mgt.Engine(0), 64) for _ in range(6)]
    for holder in holders:
        assert holder() == 0
    step = SmallStep(mgt.Engine(0))
    assert step(one_stream=True) == 0
    want = step.result()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert step(forks=0) == 0
    graph.replay()
    assert np.array_equal(step.result(), want)
    for held in holders + [step]:
        held.engine.close()
