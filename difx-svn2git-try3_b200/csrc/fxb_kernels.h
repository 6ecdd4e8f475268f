// Kernel launchers (host-callable) of the sm_100a FX path.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "fxb_internal.h"

namespace fxb {

// Per-frequency XMAC plan on the device.
struct DevFreqPlan {
	int32_t nrow, nchan;              // rows, channels
	int32_t tcb;                      // tensor-core form: channels per spectra block (0: spectra [t][row][chan])
	int32_t tnblk;                    // tensor-core form: blocks per time, spectra [t][block][trow][tcb]
	int32_t trow;                     // tensor-core form: rows of a block (nrow and, in the FP16 / BF16 form, zero rows)
	int32_t pbits;                    // tensor-core form: log2(nchan / 4), see chan_pos
	int32_t acc_cstride;              // accumulator stride between channels (1: [out][chan], nout: [chan][out])
	int32_t acc_ostride;              // accumulator stride between outputs
	int64_t spec_off;                 // complex offset of this frequency's spectra
	int64_t acc_off;                  // complex offset of accumulators [nout][nchan]
	const int32_t *destA;             // [nrow*nrow]
	const int32_t *destB;             // [nrow*nrow]
	const int32_t *outsrc;            // [nout] source of each output: a | b << 8 | conj << 16 (a <= b), or -1
	int64_t spec8_off;                // FP8 form: offset (16-bit words) of this frequency's e4m3 spectra
	float *iscale;                    // FP8 form: [nchan][nrow] 1 / quantisation scale of the subint
	uint32_t magic;                   // tensor-core form: p / tcb = umulhi(p, magic) for p < 2^16
};

struct DevOutMap {
	int64_t acc, core;
	int32_t nchan, avg;
	int32_t cstride, pad;
};

// Tensor-core form: channel c sits at position p of its plan's blocks (block p /
// tcb, p % tcb), the four channels nchan / 4 apart side by side: they are the
// outputs of one thread of the F stage's last pass, which stores them at once
// (the XMAC takes the channels of a block in any order).
#if defined(__CUDACC__)
__host__ __device__ __forceinline__ int chan_pos(int pbits, int c)
{
	return ((c & ((1 << pbits) - 1)) << 2) | (c >> pbits);
}
__host__ __device__ __forceinline__ int pos_chan(int pbits, int p) { return ((p & 3) << pbits) | (p >> 2); }
// Tensor-core form: the four channels of positions p0 .. p0 + 3 (a multiple of 4)
// of one row of a time's blocks [block][trow][tcb], o its first.  tcb is even;
// bextra = (trow - 1) tcb lies between the end of a block's run of the row and the
// next block's, and p / tcb = umulhi(p, magic) for p < 2^16.
__device__ __forceinline__ void store_quad(uint32_t *o, uint32_t p0, uint32_t tcb, uint32_t magic, uint32_t bextra,
                                           uint4 h)
{
	uint32_t *q = o + p0 + __umulhi(p0, magic) * bextra;
	if(tcb & 2u)
	{
		*(uint2 *)q = make_uint2(h.x, h.y);
		*(uint2 *)(o + p0 + 2u + __umulhi(p0 + 2u, magic) * bextra) = make_uint2(h.z, h.w);
	}
	else
		*(uint4 *)q = h;
}
#endif

// A weight sum: stations and, of INTERLACEDVDIF stations, recorded bands (-1:
// the station's own weight); s2 = -1: the weights of s1 alone.
struct DevWeightSum {
	int32_t s1, s2, b1, b2;
};

// A weight slot of the core result (float index) and the sum it shows.  The
// products of one baseline share a sum, so do a station's autocorrelations.
struct DevWeightOut {
	int64_t dst;
	int32_t sum, pad;
};

// One zoom-band row: spectra channels [choff, choff + nchan) of row src_row
// of plan src_plan, copied to row dst_row of plan dst_plan.
struct DevZoomCopy {
	int32_t src_plan, src_row, dst_plan, dst_row, choff, nchan;
};
// consecutive rows of one zoom frequency
struct DevZoomGroup {
	int32_t first, count;
};

// raw INTERLACEDVDIF reads (DevStation::muxraw): frame slots, muxed headers
// and the muxed stream's length and start, before the frame validity
// (fxb_mux.cu); maxslots / maxproc bound every raw station's slots / frames
void launch_mux_raw(const DevStation *st, DevSubintStation *sub, int S, int maxslots, int maxproc,
                    cudaStream_t stream);
// bandok (may be null): per frame, the bands that keep their samples
// fillok (may be null): per frame, no fill pattern (the only check that the
// first frame of a complex unpack window gets)
void launch_frame_valid(const DevStation *st, const DevSubintStation *sub, uint8_t *valid, uint32_t *bandok,
                        int64_t valid_stride, int S, cudaStream_t stream, uint8_t *fillok = nullptr);
// the subint time is read from sub[s].subsec / subns
void launch_interpolators(const DevStation *st, DevSubintStation *sub, int S, int blockspersend, cudaStream_t stream);
// launch_interpolators and launch_frame_valid as one launch (stations without
// raw INTERLACEDVDIF reads, whose frame check needs the placement first)
void launch_prep(const DevStation *st, DevSubintStation *sub, int S, int blockspersend, uint8_t *valid,
                 uint32_t *bandok, int64_t valid_stride, cudaStream_t stream, uint8_t *fillok);
void launch_fft_params(const DevStation *st, const DevSubintStation *sub, const int32_t *validflags, int nflagint,
                       const uint8_t *valid, const uint32_t *bandok, int64_t valid_stride, int S, int T, int order,
                       FftParam *out, float *pbw, int nbm, cudaStream_t stream, const uint8_t *fillok = nullptr,
                       float *wts = nullptr);

// Fused unpack -> fringe rotation -> FFT -> fractional-sample correction.
// One CTA per (station, FFT); writes FP32 spectra into spec.  Returns the
// launch's error (including that of raising the shared-memory limit).
cudaError_t launch_fstage(const DevStation *st, const DevSubintStation *sub, const DevBand *bands, int maxband,
                   const DevFreqPlan *plans, const uint8_t *valid, int64_t valid_stride, const FftParam *params,
                   const float2 *twiddle, int maxN, int S, int T, int order, bool fractionallofreq, int maxfft,
                   float2 *spec, cudaStream_t stream);

// F stage (csrc/fxb_fstage.cu).  A work item is one subband of one station
// with the one or two bands recording it; items of the same kind (FFT length,
// band packing) share a launch.
struct FGroup {
	int32_t station, freq;
	int32_t band[2];
	int32_t row[2];          // rows within the frequency's spectra (-1: band not output)
	int32_t nb;
	int32_t lsb;
	double lofreq;
	// corrections of the subband's recorded frequency (mode.cpp:870-1145,
	// 1296-1347): per band the clock term of the fractional-sample rotation,
	// fse - clk[j] (us; offset -/+ delta/2 by polarisation), and the
	// phase-offset rotation (turns); the LO offset (Hz) of the fringe rotation
	double clk[2];
	double looff;
	float phase[2];
	int32_t corr;            // any correction nonzero
	// two bands of different subbands (equal sideband and spectra shape, no
	// corrections): the second band's subband; else freq and lofreq again
	int32_t freq1;
	double lofreq1;
};

#if defined(__CUDACC__)
// D (turns per channel) as hi + lo with hi holding 10 significant bits, so
// that c * hi is exact in FP32 for |c| <= 8192 and the channel phase
// c * D = (c * hi mod 1) + c * lo keeps FP32 accuracy however many turns
// c * D spans (large clock offsets)
__device__ __forceinline__ void split_turns(double D, float &hi, float &lo)
{
	int e;
	frexp(D, &e);
	const double h = D == 0.0 ? 0.0 : ldexp(rint(ldexp(D, 9 - e)), e - 9);
	hi = (float)h;
	lo = (float)(D - h);
}

// LO-offset fringe phase (turns) at wall-clock time w (seconds since the job
// start) except the per-sample term: -looff (w - int w) - frac(looff) int w,
// the integer seconds entering only through the offset's fractional part
// (mode.cpp:873-882, 932-951)
__device__ __forceinline__ double looff_wall_turns(double looff, double w)
{
	if(looff == 0.0)
		return 0.0;
	const int iw = (int)w;
	double fl = fabs(looff) - (int)fabs(looff);
	if(looff < 0)
		fl = -fl;
	return -looff * (w - iw) - (fabs(fl) > (double)1e-9f ? fl * iw : 0.0);
}
#endif

struct FKind {
	int32_t first, count;    // range of work items in the item table
	int32_t N, nb;           // FFT length, bands per item
	int32_t kb, fpc;         // radix-8 butterflies per thread and pass, FFTs side by side per CTA
	int32_t threads, tq;     // CTA size, FFT iterations per CTA
	int32_t pp, out;         // two exchange buffers (else one), output form (0 FP32 spectra, 1 tensor-core spectra)
	int32_t items_fast;      // grid order: work items fastest (else time chunks); scheduling only
	int32_t twn, tcfft;      // twiddle entries of length N; 1: tensor-core FFT kernel (fxb_fstage_tc.cu)
	size_t smem;
	const void *tw;          // twiddle table of length N (make_fstage_twiddles layout)
	const void *tctab;       // constant tables of the tensor-core FFT kernel
	const int32_t *tcpairs;  // tensor-core FFT: [tcnpairs][2] FGroup indices of each work unit's two subbands
	int64_t tcrec0;          // tensor-core FFT: first byte of its units' records (launch_tc_units) in FsArgs::tcrec
	int32_t tcnpairs;
	int32_t tcbpt;           // tensor-core FFT: bits per time of the stations' VDIF words
	int32_t muxraw;          // 1: the items' stations hand over raw INTERLACEDVDIF reads
	int32_t cplx;            // 1: the items' stations sample complex (N = nchan points)
	int32_t pair0, two;      // two-band kinds: first PairItem; the bands are of different subbands
	int32_t persist;         // 1: run by the persistent launches (launch_fstage_multi), not launch_fstage_kind
};

// Spectra of the tensor-core forms hold X 2^-kTcSpecExp (FP16 or BF16), so
// that the largest value of any supported FFT (16384 points of 8-bit levels,
// |X| <= 16384 x 38.8) stays inside the FP16 range; the XMAC epilogue scales
// the products back by 2^(2 kTcSpecExp), exactly.
constexpr int kTcSpecExp = 5;

// Two-band items (csrc/fxb_fstage_pair.cuh).  Constants of one FFT of one item,
// computed by k_pair_consts with the subint's FFT parameters.
// In this order without gaps: with gaps they took 128 (twists 48) bytes, written and
// read once per item and FFT (20 stations x 4 subbands x 4096 FFTs of 256 points: the
// preparation kernels 41.7 us, 38.8 without).
struct alignas(16) PairConst {
	float P0, alpha, beta, gamma;        // fringe phase (turns): start and per-sample terms
	float eps;
	int32_t flags;
	float2 st;                           // order 1: rotator step over N/8 samples, exp(-2 pi i alpha N/8)
	float dhi[2], dlo[2];                // fractional-sample turns per channel of each band (split_turns)
	float2 os[2];                        // rotator step over N/8 channels of each band
	float post[2];                       // order-0 post-F turns and the band's phase offset
	const uint8_t *wp;                   // first payload byte of the window's first frame (raw reads: the buffer)
	uint32_t fa, so;                     // first frame of the window, window start within it
	uint32_t fmask;                      // validity of the window's frames (bit k: frame fa + k)
	int32_t stuck;                       // samples [stuck, N) read as zero
	int32_t mi00, mi01, mi10, mi11;      // raw reads: thread frames of the window's first and second frame, per band
};
// kPTwo: the second band's fringe rotation, in an array of its own
struct alignas(16) PairTwist {
	float2 st;
	float P0, alpha, beta, gamma;
	float eps;
	int32_t pad_;
};
static_assert(sizeof(PairConst) == 112 && sizeof(PairTwist) == 32, "no gaps");
// What does not change from subint to subint: the samples' place in the frames
// and the spectra's place.  FP32 form [t][row][chan]; tensor-core form blocked
// [t][block][trow][tcb] in the order of chan_pos.
struct alignas(16) PairItem {
	int64_t first, tstride;              // the first band's value of time 0, channel (position) 0; a time
	int64_t rowd;                        // from the first band's values to the second's
	uint32_t tcb, magic, bextra;         // channels of a block; p / tcb = umulhi(p, magic) for p < 2^16;
	                                     // position p sits at p + p / tcb x bextra
	int32_t shift, oflags;               // shift: log2 tcb (kOWide)
	uint32_t fs, bpt, boff0, boff1;      // samples per frame, bits per time, first bit of each band
	uint32_t hbits;                      // header bits
	int32_t nbits, header, framebytes, minfb, mnthr;
	int32_t station, band0, band1, lsb, asl, adj;   // adj: both bands side by side in one aligned field
	int32_t group, two;                  // two: the bands' LOs differ
};
enum : int32_t {
	kORow0 = 1,       // the band has a row
	kORow1 = 2,
	kOH16 = 4,        // FP16 (else BF16)
	kOBoth = 8,       // blocks of two channels, the bands' rows an aligned pair
	kOWide = 16       // blocks of a power of two channels, at least 4
};
enum : int32_t {
	kPActive = 1,     // valid FFT
	kPNarrow = 2,     // fmask covers the window
	kPBlank = 4,      // a valid frame of the window blanks one of the item's bands
	kPSame = 8,       // the two bands take the same output rotation
	kPTwo = 32,       // the bands take different fringe rotations
	kPFast = 16,      // every sample of the window counts, frames of at least N/8 samples, bands side by
	                  // side; raw reads: at most two frames
	kPApart = 64      // the same with the bands apart
};

struct FsArgs {
	const DevStation *st;
	const DevSubintStation *sub;
	const FGroup *groups;
	const DevFreqPlan *plans;
	const uint8_t *valid;
	const uint32_t *bandok;       // per frame: bands that keep their samples (null: all)
	const uint8_t *fillok;        // per frame: no fill pattern (complex data: the window's first frame)
	int64_t valid_stride;
	const FftParam *params;
	const void *tw;          // set from FKind::tw by launch_fstage_kind
	int32_t maxN, T, tq, order;
	int32_t fraclo, pp, first, items_fast;
	void *spec;              // [t][row][chan]: float2 (out 0), or half2 / bf16x2 (out 1) scaled by 2^-kTcSpecExp
	int32_t *err;            // device error flag (bounded waits of the tensor-core FFT kernel)
	int32_t h16;             // out 1: spectra as FP16 (else BF16)
	int32_t pair0;           // set from FKind::pair0 by launch_fstage_kind
	const PairItem *pitems;  // two-band items, and the constants of their FFTs [item][T]
	PairConst *pconst;
	PairTwist *ptwist;       // of the two-band items from ptwist0 on, [item - ptwist0][T]
	unsigned char *tcrec;    // unit records of the tensor-core FFT kinds
	int32_t ptwist0, two;    // two: the launch's items have twists (set by launch_fstage_kind)
};
// constants of the subint's FFTs of a two-band kind's items
void launch_pair_consts(const FKind &k, const FsArgs &a, cudaStream_t stream);

bool fstage_plan(int N, int nb, int out, FKind *k);
// the kernels of one-band and two-band items by output form, and the
// persistent launch of a class (fxb_fs_*.cu)
struct FsMultiArgs;
void launch_fs_one_f32(const FKind &k, const FsArgs &a, cudaStream_t stream);
void launch_fs_pair_f32(const FKind &k, const FsArgs &a, cudaStream_t stream);
void launch_fs_one_tc(const FKind &k, const FsArgs &a, cudaStream_t stream);
void launch_fs_pair_tc(const FKind &k, const FsArgs &a, cudaStream_t stream);
void launch_fs_one_multi(const FsMultiArgs &m, int cls, int nsm, cudaStream_t st);
void launch_fs_pair_multi(const FsMultiArgs &m, int cls, int nsm, cudaStream_t st);
void launch_fstage_kind(const FKind &k, FsArgs a, cudaStream_t stream);

// The persistent F-stage launches over the CUDA-core kinds of tensor-core-
// form contexts (VDIF stations, plain or raw INTERLACEDVDIF reads) of one
// context or several: CTAs take
// work units from a list in order, each run as one CTA of launch_fstage_kind
// would run it (tq x fpc FFT times of one work item), one launch per class of
// units.  Every tensor-core-form context runs these kinds this way, alone or in
// a batch, so results do not depend on it.
constexpr int kFsMultiMembers = 16;
constexpr int kFsMultiFc = 64;           // FFT constants of one unit at most (tq x fpc)
// classes of units: by length and bands, plain VDIF's (fstage_multi_class), then
// those of raw reads
constexpr int kFsMultiPer = 18, kFsMultiClasses = 2 * kFsMultiPer;
struct FsMultiKind {
	const void *tw;                      // twiddles of length N
	int32_t member, code;                // context; 128 x raw INTERLACEDVDIF reads + 32 x bands per item + log2 N
	int32_t first, tq;                   // first FGroup of the kind, FFT iterations per unit
};
struct alignas(16) FsMultiUnit {
	int32_t kind, item, tchunk;
	int32_t t0, nfc, pad_;               // two-band units: first FFT, FFTs
	const PairItem *pitem;
	const PairConst *consts;             // of FFT t0
	const PairTwist *twists;             // of FFT t0, or null
};
struct FsMultiArgs {
	FsArgs m[kFsMultiMembers];           // per context, with its subint's staging
	const FsMultiKind *kinds;
	const FsMultiUnit *units;            // by class
	int32_t unit0[kFsMultiClasses], nunit[kFsMultiClasses];   // each class's first unit and units
	int32_t *ctr;                        // one counter per class, zero before the launch
};
// class of a kind (FFT length N = 8192 .. 32, bands per item nb) in the persistent
// launches: 2 log2(8192 / N), one more for one band; -1: not run there.  And the FFT
// iterations per unit for a kind's tq
int fstage_multi_class(int N, int nb);
int fstage_multi_tq(int N, int nb, int tq);
cudaError_t launch_fstage_multi(const FsMultiArgs &m, int nsm, cudaStream_t stream);
// the same with the class kernels spread over streams (each kernel on the
// next stream of the set), for callers that run them as parallel branches
cudaError_t launch_fstage_multi_on(const FsMultiArgs &m, int nsm, const cudaStream_t *streams, int nstream);
// F stage of the tensor-core form with the FFT on the tensor cores (N = 2048;
// csrc/fxb_fstage_tc.cu).  Eligible: 2048-point FFTs, fringe rotation order
// 1 (or 0 with upper sidebands only), 2-bit stations of 2..32 bands (all
// stations of the kind alike), each subband's two bands in one 4-bit field,
// 16-byte aligned frames of at least 128 samples; a work unit is two
// subbands of one station with equal sideband at one FFT time.
size_t fstage_tc_tables_bytes();
void make_fstage_tc_tables(void *out);
bool fstage_tc_eligible(int N, int order, bool any_lsb);
size_t fstage_tc_rec_bytes(int npairs, int T);
// the subint's unit records, before launch_fstage_tc
void launch_tc_units(const FKind &k, const FsArgs &a, cudaStream_t stream);
// returns the launch's error
cudaError_t launch_fstage_tc(const FKind &k, FsArgs a, int nsm, cudaStream_t stream);

// twiddles of FFT length N, FKind::twn entries
void make_fstage_twiddles(int N, float2 *out32);

// FP32 cross-multiply-accumulate into acc over a set of frequencies with
// equal (rows, channels): plan_idx[0..nf) index dplans.
void launch_xmac_fp32(const DevFreqPlan &plan0, const DevFreqPlan *dplans, const int32_t *plan_idx, int nf, int T,
                      int nsm, const float2 *spec, float2 *acc, cudaStream_t stream);

// Tensor-core XMAC (csrc/fxb_xmac_h.cu; FP8 form: csrc/fxb_xmac_f8.cu) over one
// group of equally shaped subbands whose bf16x2 spectra lie in one block
// [subband][Tpad][block][trow][CB].
struct TcShape {
	int32_t f8;                       // FP8 form: e4m3 pairs, K tiles of 64 times
	int32_t h16;                      // operands (or the FP8 form's source spectra) FP16, else BF16
	int32_t nrow, nchan, T;
	int32_t CB, trow, Tpad;           // channels and rows of a block, times padded to whole K tiles
	int32_t nkt, nslice;              // K tiles; slices of a unit's times summed apart
	int32_t split;                    // 1: the two operand tiles of a block are units of their own
	int32_t nrs, nas;                 // ring stages (FP8 form: raw and operand stages)
	int32_t nb;                       // 2: one CTA per SM, 1: two
	// FP8 form
	int32_t w8;                       // values per time of a block, nrow * CB padded to 8
	int32_t r2p, G;                   // real rows per channel (padded to 8), channels per tile
	int32_t raw_bytes, raw_stride;    // bytes of one TMA box, stride of the raw stages
	int32_t dstride, dump_off;        // accumulator copy: floats per row, byte offset
	size_t smem;
};
bool tc_shape(int nrow, int nchan, int nf, int T, int nsm, bool f8, bool h16, TcShape *s);
// set the ring depths and CTAs per SM of a shape (and its shared-memory plan);
// false if they do not fit (227 KB for one CTA per SM, 112 KB each for two)
bool tc_stages(TcShape *s, int nrs, int nas, int nb);
bool tc_make_tensormap(void *map_out, const void *spec, const TcShape &s, int nf);
size_t tc_tensormap_size();
// complex values of workspace a group needs for its slices' sums (maxout: the
// most outputs of its subbands)
int64_t tc_workspace(const TcShape &s, int nf, int maxout);
void launch_xmac_tc(const void *tmap, const TcShape &s, const DevFreqPlan *dplans, const int32_t *plan_idx, int nf,
                    float2 *ws, int maxout, int nsm, int32_t *err, float2 *acc, cudaStream_t stream);
// One launch over several groups (of one context or several) whose shapes
// share rows and form: the CTAs stride over the groups' work
// units in turn.  Each product is added to its accumulator once per subint
// whatever the schedule, so results equal those of a launch per group.
constexpr int kXMultiGroups = 16;
struct alignas(64) TmapBytes {
	unsigned char b[128];
};
struct XGroupRec {
	const DevFreqPlan *plans;
	const int32_t *plan_idx;             // [subbands of the group] plan of each
	float2 *acc;                         // the context's accumulators
	float2 *ws;                          // sums of each slice [slice][subband][channel][ws_nout]
	int64_t ws_slice;
	int32_t ws_nout, nf;
	int32_t nchan, nkt, nblk, unit0;     // channels, K tiles, channel blocks per subband, first unit
	int32_t nslice, split;               // 1: an operand tile per unit
};
struct XMultiArgs {
	TmapBytes map[kXMultiGroups];        // CUtensorMap of each group's spectra block
	XGroupRec g[kXMultiGroups];
	int32_t ngroups, nunits;
};
// appends a group (false when the launch is full)
bool xmac_multi_add(XMultiArgs *xm, const void *tmap, const TcShape &s, const DevFreqPlan *dplans,
                    const int32_t *plan_idx, int nf, float2 *ws, int maxout, float2 *acc);
void launch_xmac_tc_multi(const XMultiArgs &xm, const TcShape &s, int nsm, int32_t *err, cudaStream_t stream);
// FP8 form (fxb_xmac_f8.cu)
bool f8_shape(TcShape *s);
bool f8_stages(TcShape *s, int nrs, int nas, int nb);
bool f8_tensormap(void *map_out, const void *spec, const TcShape &s, int nf);
void f8_launch(const XMultiArgs &xm, const TcShape &s, int nsm, int32_t *err, cudaStream_t stream);
// FP8 form: per subband of the group (plan_idx[nf]), the bf16x2 spectra
// [Tpad][nblk][nrow][CB] at spec_off -> e4m3x2 [Tpad][nblk][w8] at spec8_off,
// scaled per (channel, input) so that the input's largest component over the
// subint's T times maps to 240; writes 1 / scale to iscale[channel][input]
void launch_quant_fp8(const TcShape &s, const DevFreqPlan *dplans, const int32_t *plan_idx, int nf, int T,
                      const uint32_t *spec16, uint16_t *spec8, cudaStream_t stream);

// Phase cal (csrc/fxb_pcal.cu).  A group is up to kPcalGroupBands recorded
// bands of one station with the same bin count; a band is one band's tones.
constexpr int kPcalGroupBands = 16;
struct DevPcalGroup {
	int32_t station, nb, nbins, shift;  // shift: the shifting extractor's offset (Hz), complex bins; else 0
	int64_t fs;                         // samples per second
	int32_t band[kPcalGroupBands];
	int64_t bin_off[kPcalGroupBands];   // first bin (double) of each band in the bin accumulator
};
struct DevPcalBand {
	int32_t ntones, nbins, first, step;
	int32_t shift, pad;                 // complex bins when shift != 0
	int64_t bin_off, core;
};
// shared memory of a group's lane sums (bin counts below the CTA width) and
// of one launch with tpc windows per chunk
size_t pcal_group_smem(const DevPcalGroup &g);
size_t pcal_smem(size_t group_smem, int tpc);
constexpr size_t kPcalSmemMax = 96 * 1024;    // lane sums of one group at most
constexpr size_t kPcalSmemLaunchMax = 200 * 1024;   // a launch's window table and lane sums at most
// split: windows per FFT; tpc: windows per chunk; chunks: slices of the bins
struct PcalPlan { int split, tpc, chunks; };
// nbins: bins (doubles) of a slice; minfft: the groups' shortest FFT
PcalPlan pcal_plan(const DevPcalGroup *groups, int ngroups, int64_t nbins, int T, int minfft);
// allows the binning kernels smem bytes of dynamic shared memory (once per context)
cudaError_t pcal_init(size_t smem);
// folds the subint's samples into the FP64 bins: chunk c of the plan adds to
// bins + c * chunk_stride.  Every group of one
// launch belongs to stations of nbits-bit samples with bpt bits per time and
// to one extractor (shift: the shifting extractor's complex bins); maxbins is
// the launch's largest bin count, smem its pcal_smem.
void launch_pcal_bin(const DevPcalGroup *groups, int ngroups, int maxbins, const PcalPlan &plan, int nbits, int bpt, bool shift,
                     size_t smem, const DevStation *st, const DevSubintStation *sub, const FftParam *params,
                     const uint8_t *valid, int64_t valid_stride, int T, int64_t chunk_stride, double *bins,
                     cudaStream_t stream);
// writes the tones of every band into the core result
void launch_pcal_final(const DevPcalBand *bands, int nbands, int nchunk, int64_t chunk_stride, const double *bins,
                       float2 *core, cudaStream_t stream);

// Zoom-band spectra from their parents' (after the F stage, before the
// XMAC): tc selects the tensor-core form's bf16x2 spectra.
void launch_zoom_gather(const DevZoomCopy *zc, int nzc, const DevZoomGroup *groups, int ngroups, int maxquads,
                        const DevFreqPlan *plans, int T, bool tc, void *spec, cudaStream_t stream);

// adds the subint's weight sums to acc[nsum].  wts: data weights [station][FFT];
// pbw: per-band data weights [station][FFT][nbm] of INTERLACEDVDIF stations (null: none)
void launch_weights(const DevWeightSum *sums, int nsum, const float *wts, const float *pbw, int nbm, int T, float *acc,
                    cudaStream_t stream);

void launch_finalise(const DevOutMap *om, int nom, const float2 *acc, const DevWeightOut *wout, int nwout,
                     const float *wacc, float2 *core, int64_t corelen, cudaStream_t stream);

void launch_vdif_unpack(const uint8_t *data, int64_t nbytes, int payload, int header, int nchan, int nbits,
                        int64_t offsetsamples, int nsamp, float *out, int *good, cudaStream_t stream);

}  // namespace fxb
