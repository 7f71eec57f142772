// Fused x passes of the operators with more than three inputs: the scalar
// fluxes (OpScal: u, v, w, phi -> phi u, phi v, phi w) and the Smagorinsky
// stress (OpSmag: six strain components -> six stresses).
//
// Four or six physical fields do not fit a thread's registers next to the
// transforms in flight, so the inverse transforms run two at a time and a field
// leaves the registers before the next pair starts.  Both kernels are a grid of
// resident CTAs (64 threads, four to an SM in FP64) walking the row pairs, with
// the next tile's rows brought in by cp.async while the current one is
// transformed, as k_xfused_st.  What bounds them is what bounds the velocity
// pass: shared-memory exchanges and FP64 latency at 8 warps per SM (L1 at 59-72 %
// of its rate, DRAM at 13-14 % at 128^3 and 35 % at 256^3).
//
// FP64 only: the FP32 form keeps the register-resident kernel, whose rounding its
// runs repeat (the same operations contracted otherwise differ by 2e-8 after a few
// steps).
// Against the register-resident kernel, which held every field of a tile in
// registers and spilled: scalar fluxes at 256^3 unpruned 0.79 -> 0.36 ms,
// Smagorinsky stress at 128^3 0.19 -> 0.08 ms.
#pragma once
#include "passes.cuh"
#include "xfused2.cuh"

template <int N> H3D_D void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// the rows (kx < lim, in 16-byte chunks) of NF fields from f0 on, of the TC row
// pairs at pair0: field f0 + i to dst + i * dstride as [row][rs]; rows of pairs
// beyond npairs are not copied
template <typename TS, int NF, int TC, int NT>
H3D_D void xp_issue(const FusedArgs &a, int f0, cx<TS> *dst, int dstride, int pair0, int nch)
{
    constexpr int PER = StageRow<TS>::PER;
    const int rs = nch * PER;
#pragma unroll
    for (int f = 0; f < NF; f++) {
        const cx<TS> *base = reinterpret_cast<const cx<TS> *>(a.in[f0 + f]) + (int64_t)(2 * pair0) * a.pitch;
        if constexpr (TC == 1) {
            if (pair0 < a.npairs)
#pragma unroll
                for (int r = 0; r < 2; r++)
                    for (int ch = threadIdx.x; ch < nch; ch += NT)
                        cp_async16(dst + f * dstride + r * rs + ch * PER, base + r * a.pitch + ch * PER);
        } else {
            const int total = 2 * TC * nch;
            const DivU32 dch(nch);  // q < total <= 2^16, nch <= 513
            for (int q = threadIdx.x; q < total; q += NT) {
                const int r = dch(q), ch = q - r * nch;
                if (pair0 + r / 2 < a.npairs) cp_async16(dst + f * dstride + r * rs + ch * PER, base + r * a.pitch + ch * PER);
            }
        }
    }
}

// forward transforms of NF packed fields already in registers, split and stored
// to a.out[o0 .. o0 + NF); ends with the buffers free
template <typename T, int L, int TC, int NT, int NF, typename TS>
H3D_D void xp_forward(const FusedArgs &a, int o0, cx<T> (&in)[NF][ColFFT<T, L, TC, NT, true, true, false>::NIN], cx<T> *sm,
                      const cx<T> *__restrict__ tw, int pair0, int lim)
{
    using FF = RowFFT<T, L, TC, NT, false>;
    FF::template run_multi_front<NF>(in, sm, tw);
    void *outs[NF];
#pragma unroll
    for (int f = 0; f < NF; f++) outs[f] = a.out[o0 + f];
    xf_last_split<T, L, TC, NT, NF, TS>(sm, tw, outs, a.pitch, pair0, a.npairs, lim, (T)0.5);
    __syncthreads();
}

// packed inputs of the inverse transforms from the staged rows of two fields
// (row stride rs0, rs1 and kx limit lim0, lim1 of each)
template <typename T, int L, int TC, int NT, typename TS>
H3D_D void xp_load2(const FusedArgs &a, const cx<TS> *s0, const cx<TS> *s1, int rs0, int rs1, int pair0, int lim0, int lim1,
                    cx<T> (&in)[2][ColFFT<T, L, TC, NT, true, false, true>::NIN])
{
    using FI = RowFFT<T, L, TC, NT, true>;
#pragma unroll
    for (int f = 0; f < 2; f++)
#pragma unroll
        for (int i = 0; i < FI::NB0; i++)
#pragma unroll
            for (int m = 0; m < FI::R0; m++) {
                int c, p;
                if (FI::in_slot(i, m, c, p) && pair0 + c < a.npairs) {
                    const int rs = f == 0 ? rs0 : rs1;
                    const cx<TS> *A = (f == 0 ? s0 : s1) + 2 * c * rs;
                    in[f][i * FI::R0 + m] = load_packed<T, L, TS>(A, A + rs, p, f == 0 ? lim0 : lim1);
                } else in[f][i * FI::R0 + m] = mk<T>(0, 0);
            }
}

// the same of NF fields staged E elements apart
template <typename T, int L, int TC, int NT, int NF, typename TS>
H3D_D void xp_load(const FusedArgs &a, const cx<TS> *s, int E, int rs, int pair0, int lim,
                   cx<T> (&in)[NF][ColFFT<T, L, TC, NT, true, false, true>::NIN])
{
    using FI = RowFFT<T, L, TC, NT, true>;
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
        for (int i = 0; i < FI::NB0; i++)
#pragma unroll
            for (int m = 0; m < FI::R0; m++) {
                int c, p;
                if (FI::in_slot(i, m, c, p) && pair0 + c < a.npairs) {
                    const cx<TS> *A = s + f * E + 2 * c * rs;
                    in[f][i * FI::R0 + m] = load_packed<T, L, TS>(A, A + rs, p, lim);
                } else in[f][i * FI::R0 + m] = mk<T>(0, 0);
            }
}

// Scalar fluxes.  Inputs u, v, w, phi (a.in[0..4)), outputs phi u, phi v, phi w.
// phi and u are inverse-transformed together, then v and w with phi and phi u
// waiting in registers; the three products go forward in lockstep.  Five buffers,
// 46 KB at 512 elements in FP64: the rows of phi and u arrive in buffers 3 and 4
// (their exchange buffers) while the previous tile's products go forward in 0, 1
// and 2, those of v and w in 1 and 2 while phi and u are transformed, so that
// every copy overlaps a transform and four CTAs share an SM.  (With a stage of
// its own for all four fields an unpruned tile left room for three CTAs.)
template <typename T, int L, int TC, int NT, typename TS, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_xscal(const FusedArgs a, const cx<T> *__restrict__ tw)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    using FI = RowFFT<T, L, TC, NT, true>;
    using FF = RowFFT<T, L, TC, NT, false>;
    static_assert(FI::NOUT == FF::NIN && sizeof(T) == sizeof(TS), "slot hand-off mismatch");
    constexpr int NP = FI::NOUT, E = Lay<L, TC, true>::elems;
    // the staged rows of a pair fit its transform's padded buffer
    static_assert(2 * StageRow<TS>::chunks(L / 2 + 1) * StageRow<TS>::PER <= L + L / 8 && E * sizeof(cx<T>) % 16 == 0, "stage");
    cx<T> *sm = reinterpret_cast<cx<T> *>(smraw);
    cx<T> *bp = sm + 3 * E, *bv = sm + E;  // phi and u; v and w
    const T norm = (T)a.norm;
    const int lim = a.kx_lim > 0 ? a.kx_lim : L / 2 + 1;
    const int nch = StageRow<TS>::chunks(lim), rs = nch * StageRow<TS>::PER;
    const int limp = a.full_phi ? L / 2 + 1 : lim, nchp = StageRow<TS>::chunks(limp), rsp = nchp * StageRow<TS>::PER;  // phi
    const int ntiles = (a.npairs + TC - 1) / TC;
    auto issue_phi_u = [&](int tile) {
        if (tile < ntiles) {
            xp_issue<TS, 1, TC, NT>(a, 3, bp, E, tile * TC, nchp);
            xp_issue<TS, 1, TC, NT>(a, 0, bp + E, E, tile * TC, nch);
        }
        cp_async_commit();
    };
    auto issue_v_w = [&](int tile) {
        if (tile < ntiles) xp_issue<TS, 2, TC, NT>(a, 1, bv, E, tile * TC, nch);
        cp_async_commit();
    };
    issue_phi_u(blockIdx.x);
    issue_v_w(blockIdx.x);
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int pair0 = tile * TC;
        cx<T> phi[NP], prod[3][NP];
        cp_async_wait_group<1>();
        __syncthreads();
        {
            cx<T> in[2][FI::NIN], out[2][NP];
            xp_load2<T, L, TC, NT, TS>(a, bp, bp + E, rsp, rs, pair0, limp, lim, in);
#pragma unroll
            for (int q = 0; q < NP; q++) out[0][q] = out[1][q] = mk<T>(0, 0);  // slots of idle butterflies
            __syncthreads();  // the staged rows are read: the buffers turn into exchange buffers
            FI::template run_multi<2>(in, bp, out, tw);
#pragma unroll
            for (int q = 0; q < NP; q++) {
                phi[q] = mk<T>(out[0][q].x * norm, out[0][q].y * norm);
                prod[0][q] = mk<T>(phi[q].x * (out[1][q].x * norm), phi[q].y * (out[1][q].y * norm));
            }
        }
        cp_async_wait_group<0>();
        __syncthreads();  // v and w have arrived, the exchange buffers of phi and u are read
        {
            cx<T> in[2][FI::NIN], out[2][NP];
            xp_load2<T, L, TC, NT, TS>(a, bv, bv + E, rs, rs, pair0, lim, lim, in);
#pragma unroll
            for (int q = 0; q < NP; q++) out[0][q] = out[1][q] = mk<T>(0, 0);
            __syncthreads();
            issue_phi_u(tile + (int)gridDim.x);
            FI::template run_multi<2>(in, bv, out, tw);
#pragma unroll
            for (int q = 0; q < NP; q++) {
                prod[1][q] = mk<T>(phi[q].x * (out[0][q].x * norm), phi[q].y * (out[0][q].y * norm));
                prod[2][q] = mk<T>(phi[q].x * (out[1][q].x * norm), phi[q].y * (out[1][q].y * norm));
            }
        }
        __syncthreads();  // the exchange buffers are read
        xp_forward<T, L, TC, NT, 3, TS>(a, 0, prod, sm, tw, pair0, lim);
        issue_v_w(tile + (int)gridDim.x);
    }
    cp_async_wait_all();
}

// Scalar fluxes of two scalars.  Inputs u, v, w, phi, psi (a.in[0..5)), outputs
// phi u, psi u, phi v, psi v, phi w, psi w.  The velocity's three inverse transforms
// serve both scalars (11 transforms in five steps, where two passes of k_xscal take
// 14 in six).  phi, psi and u go back together, phi and psi stay in registers, the
// products leave two at a time.  Five buffers as k_xscal's: phi, psi and u in 0, 1
// and 2 while the rows of v and w wait in 3 and 4, and the other way round.
// Velocity and two scalars' x passes of a step, FP64 pruned: 128^3 0.173 -> 0.158 ms,
// 256^3 1.26 -> 1.08 ms.
template <typename T, int L, int TC, int NT, typename TS, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_xscal2(const FusedArgs a, const cx<T> *__restrict__ tw)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    using FI = RowFFT<T, L, TC, NT, true>;
    using FF = RowFFT<T, L, TC, NT, false>;
    static_assert(FI::NOUT == FF::NIN && sizeof(T) == sizeof(TS), "slot hand-off mismatch");
    constexpr int NP = FI::NOUT, E = Lay<L, TC, true>::elems;
    static_assert(2 * StageRow<TS>::chunks(L / 2 + 1) * StageRow<TS>::PER <= L + L / 8 && E * sizeof(cx<T>) % 16 == 0, "stage");
    cx<T> *sm = reinterpret_cast<cx<T> *>(smraw);
    cx<T> *bv = sm + 3 * E;  // v and w
    const T norm = (T)a.norm;
    const int lim = a.kx_lim > 0 ? a.kx_lim : L / 2 + 1;
    const int nch = StageRow<TS>::chunks(lim), rs = nch * StageRow<TS>::PER;
    const int ntiles = (a.npairs + TC - 1) / TC;
    auto issue_scal_u = [&](int tile) {
        if (tile < ntiles) {
            xp_issue<TS, 2, TC, NT>(a, 3, sm, E, tile * TC, nch);
            xp_issue<TS, 1, TC, NT>(a, 0, sm + 2 * E, E, tile * TC, nch);
        }
        cp_async_commit();
    };
    auto issue_v_w = [&](int tile) {
        if (tile < ntiles) xp_issue<TS, 2, TC, NT>(a, 1, bv, E, tile * TC, nch);
        cp_async_commit();
    };
    issue_scal_u(blockIdx.x);
    issue_v_w(blockIdx.x);
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int pair0 = tile * TC;
        cx<T> phi[NP], psi[NP];
        cp_async_wait_group<1>();
        __syncthreads();
        {
            cx<T> prod[2][NP];
            {
                cx<T> in[3][FI::NIN], out[3][NP];
                xp_load<T, L, TC, NT, 3, TS>(a, sm, E, rs, pair0, lim, in);
#pragma unroll
                for (int q = 0; q < NP; q++) out[0][q] = out[1][q] = out[2][q] = mk<T>(0, 0);  // slots of idle butterflies
                __syncthreads();  // the staged rows are read: the buffers turn into exchange buffers
                FI::template run_multi<3>(in, sm, out, tw);
#pragma unroll
                for (int q = 0; q < NP; q++) {
                    const cx<T> u = mk<T>(out[2][q].x * norm, out[2][q].y * norm);
                    phi[q] = mk<T>(out[0][q].x * norm, out[0][q].y * norm);
                    psi[q] = mk<T>(out[1][q].x * norm, out[1][q].y * norm);
                    prod[0][q] = mk<T>(phi[q].x * u.x, phi[q].y * u.y);
                    prod[1][q] = mk<T>(psi[q].x * u.x, psi[q].y * u.y);
                }
            }
            __syncthreads();  // the exchange buffers are read
            xp_forward<T, L, TC, NT, 2, TS>(a, 0, prod, sm, tw, pair0, lim);
        }
        cp_async_wait_group<0>();
        __syncthreads();  // v and w have arrived
        {
            cx<T> pv[2][NP], pw[2][NP];
            {
                cx<T> in[2][FI::NIN], out[2][NP];
                xp_load<T, L, TC, NT, 2, TS>(a, bv, E, rs, pair0, lim, in);
#pragma unroll
                for (int q = 0; q < NP; q++) out[0][q] = out[1][q] = mk<T>(0, 0);
                __syncthreads();
                issue_scal_u(tile + (int)gridDim.x);
                FI::template run_multi<2>(in, bv, out, tw);
#pragma unroll
                for (int q = 0; q < NP; q++) {
                    const cx<T> v = mk<T>(out[0][q].x * norm, out[0][q].y * norm);
                    const cx<T> w = mk<T>(out[1][q].x * norm, out[1][q].y * norm);
                    pv[0][q] = mk<T>(phi[q].x * v.x, phi[q].y * v.y);
                    pv[1][q] = mk<T>(psi[q].x * v.x, psi[q].y * v.y);
                    pw[0][q] = mk<T>(phi[q].x * w.x, phi[q].y * w.y);
                    pw[1][q] = mk<T>(psi[q].x * w.x, psi[q].y * w.y);
                }
            }
            __syncthreads();
            xp_forward<T, L, TC, NT, 2, TS>(a, 2, pv, bv, tw, pair0, lim);
            xp_forward<T, L, TC, NT, 2, TS>(a, 4, pw, bv, tw, pair0, lim);
        }
        issue_v_w(tile + (int)gridDim.x);
    }
    cp_async_wait_all();
}

// Smagorinsky stress (OpSmag's arithmetic: nu_t = p0 sqrt(2 S:S), tau = -2 nu_t S).
// Buffer f holds field f throughout: its staged input rows, the exchanges of its
// inverse transform, its physical values (each thread at its own slots) and the
// exchanges of its forward transform; as a pair of fields leaves for HBM the
// next tile's rows of that pair are copied in.  Six buffers: 55 KB at 512
// elements in FP64, four CTAs per SM.
template <typename T, int L, int TC, int NT, typename TS, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_xsmag(const FusedArgs a, const cx<T> *__restrict__ tw)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    using FI = RowFFT<T, L, TC, NT, true>;
    using FF = RowFFT<T, L, TC, NT, false>;
    static_assert(FI::NOUT == FF::NIN && sizeof(T) == sizeof(TS), "slot hand-off mismatch");
    constexpr int NP = FI::NOUT, E = Lay<L, TC, true>::elems;
    // the staged rows of a pair fit its transform's padded buffer
    static_assert(2 * StageRow<TS>::chunks(L / 2 + 1) * StageRow<TS>::PER <= L + L / 8 && E * sizeof(cx<T>) % 16 == 0, "stage");
    using LY = Lay<L, TC, true>;
    cx<T> *sm = reinterpret_cast<cx<T> *>(smraw);
    const T norm = (T)a.norm, p0 = (T)a.p0;
    const int lim = a.kx_lim > 0 ? a.kx_lim : L / 2 + 1;
    const int nch = StageRow<TS>::chunks(lim), rs = nch * StageRow<TS>::PER;
    const int ntiles = (a.npairs + TC - 1) / TC;
#pragma unroll
    for (int g = 0; g < 3; g++) {
        if ((int)blockIdx.x < ntiles) xp_issue<TS, 2, TC, NT>(a, 2 * g, sm + 2 * g * E, E, blockIdx.x * TC, nch);
        cp_async_commit();
    }
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int pair0 = tile * TC;
        cx<T> ss[NP];
#pragma unroll
        for (int g = 0; g < 3; g++) {
            cx<T> *b = sm + 2 * g * E;
            cx<T> in[2][FI::NIN], out[2][NP];
            if (g == 0) cp_async_wait_group<2>();
            else if (g == 1) cp_async_wait_group<1>();
            else cp_async_wait_group<0>();
            __syncthreads();
            xp_load2<T, L, TC, NT, TS>(a, b, b + E, rs, rs, pair0, lim, lim, in);
#pragma unroll
            for (int q = 0; q < NP; q++) out[0][q] = out[1][q] = mk<T>(0, 0);
            __syncthreads();  // the staged rows are read: the buffers turn into exchange buffers
            FI::template run_multi<2>(in, b, out, tw);
            __syncthreads();  // and into the physical fields
#pragma unroll
            for (int i = 0; i < FI::NBL; i++)
#pragma unroll
                for (int m = 0; m < FI::RL; m++) {
                    const int q = i * FI::RL + m;
                    const cx<T> s0 = mk<T>(out[0][q].x * norm, out[0][q].y * norm), s1 = mk<T>(out[1][q].x * norm, out[1][q].y * norm);
                    // S11 S12 | S13 S22 | S23 S33, the off-diagonal ones twice
                    if (g == 0) {
                        ss[q] = mk<T>(s0.x * s0.x, s0.y * s0.y);
                        ss[q] = mk<T>(ss[q].x + (T)2 * (s1.x * s1.x), ss[q].y + (T)2 * (s1.y * s1.y));
                    } else {
                        ss[q] = mk<T>(ss[q].x + (T)2 * (s0.x * s0.x), ss[q].y + (T)2 * (s0.y * s0.y));
                        ss[q] = mk<T>(ss[q].x + s1.x * s1.x, ss[q].y + s1.y * s1.y);
                    }
                    int c, p;
                    if (FI::out_slot(i, m, c, p)) {
                        b[LY::idx(c, p)] = s0;
                        b[E + LY::idx(c, p)] = s1;
                    }
                }
        }
#pragma unroll
        for (int q = 0; q < NP; q++) ss[q] = mk<T>((T)-2 * (sqrt((T)2 * ss[q].x) * p0), (T)-2 * (sqrt((T)2 * ss[q].y) * p0));
#pragma unroll
        for (int g = 0; g < 3; g++) {
            cx<T> *b = sm + 2 * g * E;
            cx<T> in[2][FF::NIN];
#pragma unroll
            for (int i = 0; i < FF::NB0; i++)
#pragma unroll
                for (int m = 0; m < FF::R0; m++) {
                    const int q = i * FF::R0 + m;
                    int c, p;
                    in[0][q] = in[1][q] = mk<T>(0, 0);
                    if (FF::in_slot(i, m, c, p)) {  // the slots the inverse left this thread
                        const cx<T> s0 = b[LY::idx(c, p)], s1 = b[E + LY::idx(c, p)];
                        in[0][q] = mk<T>(ss[q].x * s0.x, ss[q].y * s0.y);
                        in[1][q] = mk<T>(ss[q].x * s1.x, ss[q].y * s1.y);
                    }
                }
            __syncthreads();
            xp_forward<T, L, TC, NT, 2, TS>(a, 2 * g, in, b, tw, pair0, lim);
            if (tile + (int)gridDim.x < ntiles) xp_issue<TS, 2, TC, NT>(a, 2 * g, b, E, (tile + gridDim.x) * TC, nch);
            cp_async_commit();
        }
    }
    cp_async_wait_all();
}
