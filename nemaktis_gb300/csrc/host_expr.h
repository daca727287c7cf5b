// Arithmetic-expression compiler/evaluator for refractive-index and mask formulas.
//
// The reference hands these strings to muParser (PhysicsCoefficients.cpp:27-103 with the
// variable "lambda" in µm; VectorField.cpp:72-76 with "x", "y", "z"). muParser is an
// external dependency; this file implements the subset of its documented grammar that the
// Nemaktis front end emits, compiled once to a postfix program and evaluated in FP64:
//   ternary  := or ('?' ternary ':' ternary)?
//   or/and   := '||' / '&&'        cmp := '<' '>' '<=' '>=' '==' '!='
//   add      := mul (('+'|'-') mul)*      mul := unary (('*'|'/') unary)*
//   unary    := ('-'|'+') unary | power   power := primary ('^' unary)?   (right assoc.)
//   primary  := number | variable | _pi | _e | func '(' args ')' | '(' ternary ')'
// Functions: sin cos tan asin acos atan sinh cosh tanh asinh acosh atanh log2 log10 log ln
// exp sqrt sign rint abs (one argument) and min max sum avg (one or more arguments).
#pragma once

#include <cctype>
#include <cmath>
#include <stdexcept>
#include <string>
#include <vector>

namespace nbpm {

struct ExprError : std::runtime_error {
	using std::runtime_error::runtime_error;
};

class Expr {
	enum Code { C_NUM, C_VAR, C_NEG, C_ADD, C_SUB, C_MUL, C_DIV, C_POW, C_LT, C_GT, C_LE, C_GE,
		C_EQ, C_NE, C_AND, C_OR, C_SEL, C_F1, C_FN, C_TAB };
	struct Op { Code code; int arg; double val; };
	// One operation on the stack st of sp values.
	static inline void step(const Op& o, double* st, int& sp, const double* v) {
		switch(o.code) {
			case C_NUM: st[sp++] = o.val; break;
			case C_VAR: st[sp++] = v[o.arg]; break;
			case C_NEG: st[sp - 1] = -st[sp - 1]; break;
			case C_ADD: sp--; st[sp - 1] += st[sp]; break;
			case C_SUB: sp--; st[sp - 1] -= st[sp]; break;
			case C_MUL: sp--; st[sp - 1] *= st[sp]; break;
			case C_DIV: sp--; st[sp - 1] /= st[sp]; break;
			case C_POW: sp--; st[sp - 1] = std::pow(st[sp - 1], st[sp]); break;
			case C_LT: sp--; st[sp - 1] = st[sp - 1] < st[sp]; break;
			case C_GT: sp--; st[sp - 1] = st[sp - 1] > st[sp]; break;
			case C_LE: sp--; st[sp - 1] = st[sp - 1] <= st[sp]; break;
			case C_GE: sp--; st[sp - 1] = st[sp - 1] >= st[sp]; break;
			case C_EQ: sp--; st[sp - 1] = st[sp - 1] == st[sp]; break;
			case C_NE: sp--; st[sp - 1] = st[sp - 1] != st[sp]; break;
			case C_AND: sp--; st[sp - 1] = (st[sp - 1] != 0) && (st[sp] != 0); break;
			case C_OR: sp--; st[sp - 1] = (st[sp - 1] != 0) || (st[sp] != 0); break;
			case C_SEL: sp -= 2; st[sp - 1] = (st[sp - 1] != 0) ? st[sp] : st[sp + 1]; break;
			case C_F1: st[sp - 1] = fn1(o.arg, st[sp - 1]); break;
			case C_FN: {
				int n = (int)o.val;
				sp -= n;
				double r = st[sp];
				for(int k = 1; k < n; k++) {
					double x = st[sp + k];
					if(o.arg == 0) r = std::fmin(r, x);
					else if(o.arg == 1) r = std::fmax(r, x);
					else r += x;
				}
				if(o.arg == 3) r /= n;
				st[sp++] = r;
				break;
			}
			case C_TAB: break;  // Grid only
		}
	}
public:
	Expr() = default;
	Expr(const std::string& src, const std::vector<std::string>& vars) : vars_(vars) {
		s_ = src;
		pos_ = 0;
		next();
		ternary();
		if(tok_ != T_END) throw ExprError("unexpected token in expression \"" + src + "\"");
	}

	double eval(const double* v) const {
		double st[64];
		int sp = 0;
		for(const Op& o : prog_) step(o, st, sp, v);
		return st[0];
	}
	double eval1(double a) const { return eval(&a); }

	// The expression on a grid of points (v0[i], v1[j], v2[k]) of three variables. A voxel's evaluation is bound
	// by pow and by the branch per operation, and most of a mask formula's operations see one coordinate: a
	// 64x64x64 sphere's weights took 3.2 ms on 16 cores point by point, 0.9 ms from tables with lines of
	// values per operation. Subexpressions of one
	// variable are evaluated once per grid value, with the same operations in the same order, so that the
	// results are those of eval() bit for bit. `hoist`: bit mask of the variables taken from tables; the
	// others are given to line() or point() by value.
	class Grid {
	public:
		Grid(const Expr& e, const std::vector<double> v[3], unsigned hoist) : e_(&e), hoist_(hoist) {
			std::vector<Node> st;
			for(const Op& o : e.prog_) {
				size_t n = 0;
				switch(o.code) {
					case C_NUM: case C_VAR: break;
					case C_NEG: case C_F1: n = 1; break;
					case C_SEL: n = 3; break;
					case C_FN: n = (size_t)o.val; break;
					default: n = 2;
				}
				Node r;
				r.vars = o.code == C_VAR ? 1u << o.arg : 0u;
				const size_t first = st.size() - n;
				for(size_t k = first; k < st.size(); k++) r.vars |= st[k].vars;
				const bool split = !one(r.vars);
				for(size_t k = first; k < st.size(); k++) {
					if(split) table(st[k], v);
					r.ops.insert(r.ops.end(), st[k].ops.begin(), st[k].ops.end());
				}
				r.ops.push_back(o);
				st.resize(first);
				st.push_back(r);
			}
			table(st[0], v);
			prog_ = st[0].ops;
		}
		// values at (i, j, 0 .. n - 1), every variable from the tables; st: depth() * n scratch
		void line(size_t i, size_t j, size_t n, double* out, double* st) const {
			const size_t idx[2] = {i, j};
			size_t sp = 0;
			auto S = [&](size_t k) { return st + k * n; };
			for(const Op& o : prog_) {
				if(o.code == C_TAB) {
					const Table& t = tab_[(size_t)o.arg];
					double* d = S(sp++);
					if(t.var == 2) for(size_t k = 0; k < n; k++) d[k] = t.val[k];
					else { const double c = t.val[t.var < 0 ? 0 : idx[t.var]]; for(size_t k = 0; k < n; k++) d[k] = c; }
				}
				else if(o.code == C_ADD || o.code == C_SUB || o.code == C_MUL || o.code == C_DIV) {
					sp--;
					double* a = S(sp - 1);
					const double* b = S(sp);
					if(o.code == C_ADD) for(size_t k = 0; k < n; k++) a[k] += b[k];
					else if(o.code == C_SUB) for(size_t k = 0; k < n; k++) a[k] -= b[k];
					else if(o.code == C_MUL) for(size_t k = 0; k < n; k++) a[k] *= b[k];
					else for(size_t k = 0; k < n; k++) a[k] /= b[k];
				}
				else {
					// the rest one value at a time through the scalar step
					size_t args = o.code == C_NEG || o.code == C_F1 ? 1 : o.code == C_SEL ? 3 : o.code == C_FN ? (size_t)o.val : 2;
					sp -= args;
					for(size_t k = 0; k < n; k++) {
						double t[64];
						for(size_t q = 0; q < args; q++) t[q] = S(sp + q)[k];
						int tp = (int)args;
						step(o, t, tp, nullptr);
						S(sp)[k] = t[0];
					}
					sp++;
				}
			}
			for(size_t k = 0; k < n; k++) out[k] = st[k];
		}
		// value at (i, j, z): variable 2 by value
		double point(size_t i, size_t j, double z) const {
			const double v[3] = {0, 0, z};
			double st[64];
			int sp = 0;
			for(const Op& o : prog_) {
				if(o.code == C_TAB) {
					const Table& t = tab_[(size_t)o.arg];
					st[sp++] = t.val[t.var < 0 ? 0 : t.var == 0 ? i : j];
				}
				else step(o, st, sp, v);
			}
			return st[0];
		}
		size_t depth() const { return (size_t)e_->maxdepth_ + 1; }

	private:
		struct Node { std::vector<Op> ops; unsigned vars = 0; };
		struct Table { int var; std::vector<double> val; };
		const Expr* e_;
		unsigned hoist_;
		std::vector<Op> prog_;
		std::vector<Table> tab_;
		static bool one(unsigned m) { return (m & (m - 1)) == 0; }
		// replaces a subexpression of at most one, tabulated variable by its table
		void table(Node& nd, const std::vector<double> v[3]) {
			if(!one(nd.vars) || (nd.vars & ~hoist_) || (nd.ops.size() == 1 && nd.ops[0].code == C_TAB)) return;
			Table t;
			t.var = nd.vars == 1 ? 0 : nd.vars == 2 ? 1 : nd.vars == 4 ? 2 : -1;
			const size_t n = t.var < 0 ? 1 : v[t.var].size();
			for(size_t k = 0; k < n; k++) {
				double x[3] = {0, 0, 0}, st[64];
				if(t.var >= 0) x[t.var] = v[t.var][k];
				int sp = 0;
				for(const Op& o : nd.ops) step(o, st, sp, x);
				t.val.push_back(st[0]);
			}
			nd.ops.assign(1, Op{C_TAB, (int)tab_.size(), 0});
			tab_.push_back(t);
		}
	};

private:
	enum Tok { T_END, T_NUM, T_NAME, T_OP };

	std::vector<std::string> vars_;
	std::vector<Op> prog_;
	std::string s_;
	size_t pos_ = 0;
	Tok tok_ = T_END;
	std::string tv_;
	double tnum_ = 0;
	int depth_ = 0, maxdepth_ = 0;

	static double fn1(int id, double x) {
		switch(id) {
			case 0: return std::sin(x); case 1: return std::cos(x); case 2: return std::tan(x);
			case 3: return std::asin(x); case 4: return std::acos(x); case 5: return std::atan(x);
			case 6: return std::sinh(x); case 7: return std::cosh(x); case 8: return std::tanh(x);
			case 9: return std::asinh(x); case 10: return std::acosh(x); case 11: return std::atanh(x);
			case 12: return std::log2(x); case 13: return std::log10(x); case 14: return std::log(x);
			case 15: return std::log(x); case 16: return std::exp(x); case 17: return std::sqrt(x);
			case 18: return (x > 0) - (x < 0); case 19: return std::rint(x); case 20: return std::fabs(x);
		}
		return NAN;
	}
	static int fn1_id(const std::string& n) {
		static const char* names[] = {"sin", "cos", "tan", "asin", "acos", "atan", "sinh", "cosh",
			"tanh", "asinh", "acosh", "atanh", "log2", "log10", "log", "ln", "exp", "sqrt", "sign",
			"rint", "abs"};
		for(int k = 0; k < 21; k++) if(n == names[k]) return k;
		return -1;
	}
	void emit(Code c, int arg = 0, double val = 0) {
		prog_.push_back({c, arg, val});
		int d = 0;
		switch(c) {
			case C_NUM: case C_VAR: d = 1; break;
			case C_NEG: case C_F1: d = 0; break;
			case C_SEL: d = -2; break;
			case C_FN: d = 1 - (int)val; break;
			default: d = -1;
		}
		depth_ += d;
		if(depth_ > maxdepth_) maxdepth_ = depth_;
		if(maxdepth_ > 60) throw ExprError("expression too deep: \"" + s_ + "\"");
	}
	[[noreturn]] void fail(const std::string& w) {
		throw ExprError(w + " in expression \"" + s_ + "\"");
	}
	void next() {
		while(pos_ < s_.size() && std::isspace((unsigned char)s_[pos_])) pos_++;
		if(pos_ >= s_.size()) { tok_ = T_END; return; }
		char c = s_[pos_];
		if(std::isdigit((unsigned char)c) || (c == '.' && pos_ + 1 < s_.size() && std::isdigit((unsigned char)s_[pos_ + 1]))) {
			size_t st = pos_;
			while(pos_ < s_.size() && (std::isdigit((unsigned char)s_[pos_]) || s_[pos_] == '.')) pos_++;
			if(pos_ < s_.size() && (s_[pos_] == 'e' || s_[pos_] == 'E')) {
				size_t save = pos_;
				pos_++;
				if(pos_ < s_.size() && (s_[pos_] == '+' || s_[pos_] == '-')) pos_++;
				if(pos_ < s_.size() && std::isdigit((unsigned char)s_[pos_])) {
					while(pos_ < s_.size() && std::isdigit((unsigned char)s_[pos_])) pos_++;
				}
				else pos_ = save;
			}
			tok_ = T_NUM;
			std::string t = s_.substr(st, pos_ - st);
			char* end = nullptr;
			tnum_ = std::strtod(t.c_str(), &end);
			if(!end || *end) fail("bad number \"" + t + "\"");
			return;
		}
		if(std::isalpha((unsigned char)c) || c == '_') {
			size_t st = pos_;
			while(pos_ < s_.size() && (std::isalnum((unsigned char)s_[pos_]) || s_[pos_] == '_')) pos_++;
			tok_ = T_NAME;
			tv_ = s_.substr(st, pos_ - st);
			return;
		}
		static const char* two[] = {"||", "&&", "<=", ">=", "==", "!="};
		for(auto t : two)
			if(s_.compare(pos_, 2, t) == 0) { tok_ = T_OP; tv_ = t; pos_ += 2; return; }
		if(std::string("+-*/^(),<>?:").find(c) != std::string::npos) {
			tok_ = T_OP; tv_ = std::string(1, c); pos_++; return;
		}
		fail(std::string("unexpected character '") + c + "'");
	}
	bool is_op(const char* o) const { return tok_ == T_OP && tv_ == o; }
	void expect(const char* o) {
		if(!is_op(o)) fail(std::string("expected '") + o + "'");
		next();
	}
	void ternary() {
		lor();
		if(is_op("?")) {
			next();
			ternary();
			expect(":");
			ternary();
			emit(C_SEL);
		}
	}
	void lor() { land(); while(is_op("||")) { next(); land(); emit(C_OR); } }
	void land() { cmp(); while(is_op("&&")) { next(); cmp(); emit(C_AND); } }
	void cmp() {
		add();
		while(true) {
			Code c;
			if(is_op("<")) c = C_LT; else if(is_op(">")) c = C_GT; else if(is_op("<=")) c = C_LE;
			else if(is_op(">=")) c = C_GE; else if(is_op("==")) c = C_EQ; else if(is_op("!=")) c = C_NE;
			else return;
			next(); add(); emit(c);
		}
	}
	void add() {
		mul();
		while(is_op("+") || is_op("-")) {
			Code c = is_op("+") ? C_ADD : C_SUB;
			next(); mul(); emit(c);
		}
	}
	void mul() {
		unary();
		while(is_op("*") || is_op("/")) {
			Code c = is_op("*") ? C_MUL : C_DIV;
			next(); unary(); emit(c);
		}
	}
	void unary() {
		if(is_op("-")) { next(); unary(); emit(C_NEG); return; }
		if(is_op("+")) { next(); unary(); return; }
		power();
	}
	void power() {
		primary();
		if(is_op("^")) { next(); unary(); emit(C_POW); }
	}
	void primary() {
		if(tok_ == T_NUM) { emit(C_NUM, 0, tnum_); next(); return; }
		if(is_op("(")) { next(); ternary(); expect(")"); return; }
		if(tok_ == T_NAME) {
			std::string name = tv_;
			next();
			if(is_op("(")) {
				next();
				int nargs = 1;
				ternary();
				while(is_op(",")) { next(); ternary(); nargs++; }
				expect(")");
				int id = fn1_id(name);
				if(id >= 0) {
					if(nargs != 1) fail("function " + name + " takes one argument");
					emit(C_F1, id);
					return;
				}
				int vid = name == "min" ? 0 : name == "max" ? 1 : name == "sum" ? 2 : name == "avg" ? 3 : -1;
				if(vid < 0) fail("unknown function \"" + name + "\"");
				emit(C_FN, vid, nargs);
				return;
			}
			for(size_t k = 0; k < vars_.size(); k++)
				if(vars_[k] == name) { emit(C_VAR, (int)k); return; }
			if(name == "_pi") { emit(C_NUM, 0, 3.141592653589793238462643); return; }
			if(name == "_e") { emit(C_NUM, 0, 2.718281828459045235360287); return; }
			fail("unknown variable \"" + name + "\"");
		}
		if(tok_ == T_END) fail("unexpected end");
		fail("unexpected token \"" + tv_ + "\"");
	}
};

}  // namespace nbpm
